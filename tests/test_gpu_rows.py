"""Products of a few rows (csrc/gemm_rows.cu) through ternary_gemm_packed: edges of the 16-row blocks, the
64-feature tiles, the groups and their split over clusters, against the oracle in 64 bits; matrices packed back to
back, here and in the tcgen05 GEMM, through the decoder."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import layer_oracle, oracle
from ternary_llm_b200 import tllm_format as tf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4, 5, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("n,k", [(1, 128), (15, 384), (64, 512), (65, 1152), (333, 2048), (130, 4352), (20000, 256)])
def test_rows(m, n, k):
    nz, sg, sc, x = oracle.make_case(n, k, seed=m * 1000 + n + k, batch=m)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")     # one row more than is asked for
    tl.ternary_gemm_packed(dev[3], w, y, m)
    tl.check_device_errors()
    got = y.cpu().numpy().astype(np.float64)
    assert (got[m] == 7.0).all()
    y64 = oracle.ternary_matvec(nz, sg, sc, x, 128, np.float64)
    # products are exact; K sums in FP32, each rounded once: K * 2^-24 of the sum of magnitudes, then FP16
    bound = k * 2.0 ** -24 * oracle.tolerance_bound(nz, sg, sc, x) / 2e-3 + 2.0 ** -11 * np.abs(y64) + 2.0 ** -25
    assert (np.abs(got[:m] - y64) <= bound).all(), np.max(np.abs(got[:m] - y64) / bound)


@pytest.mark.parametrize("k", [7168, 6784])
@pytest.mark.parametrize("n", [500, 2113, 2700, 3300, 4544, 5800, 9472])
def test_clusters_of_all_sizes(n, k):
    """Eight to one CTAs that share 56 or 53 groups of a tile, whose shares of the groups and of the 64 features are uneven."""
    nz, sg, sc, x = oracle.make_case(n, k, seed=n + k, batch=32)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    wd = torch.from_numpy(oracle.unpack_bitmasks(nz, sg).astype(np.float32) * np.repeat(sc.astype(np.float32), 128, axis=1)).cuda().double()
    want, size = dev[3].double() @ wd.T, dev[3].double().abs() @ wd.T.abs()
    for m in (4, 7, 13, 24, 32):
        y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")
        tl.ternary_gemm_packed(dev[3], w, y, m)
        assert (y[m] == 7.0).all()
        bound = k * 2.0 ** -24 * size[:m] + 2.0 ** -11 * want[:m].abs() + 2.0 ** -25      # as above
        assert ((y[:m].double() - want[:m]).abs() <= bound).all(), m
    tl.check_device_errors()


@pytest.mark.parametrize("n", [2368, 2369, 4736, 4737, 9472, 9473])
def test_both_sides_of_the_lines(n):
    """Where a tile's CTAs go from eight to four, two and one, and with them the kernel of a number of vectors."""
    k, ms = 4096, (3, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33)
    nz, sg, sc, x = oracle.make_case(n, k, seed=n, batch=max(ms))
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    wd = torch.from_numpy(oracle.unpack_bitmasks(nz, sg).astype(np.float32) * np.repeat(sc.astype(np.float32), 128, axis=1)).cuda().double()
    want, size = dev[3].double() @ wd.T, dev[3].double().abs() @ wd.T.abs()
    for m in ms:
        y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")
        tl.ternary_gemm_packed(dev[3][:m].contiguous(), w, y, m)
        assert (y[m] == 7.0).all()
        # products are exact; K sums cut or rounded to FP32, then FP16
        bound = k * 2.0 ** -23 * size[:m] + 2.0 ** -11 * want[:m].abs() + 2.0 ** -25
        if m <= 8:       # the GEMV holds 3 and 4 vectors in steps of 2^-14 of a group's largest magnitude or less, each off by half a step
            bound = bound + 2.0 ** -15 * dev[3][:m].double().abs().amax(1, keepdim=True) * wd.abs().sum(1)
        assert ((y[:m].double() - want[:m]).abs() <= bound).all(), m
    tl.check_device_errors()


@pytest.mark.parametrize("n,k,ms", [
    (832, 10240, (25, 32)), (833, 10240, (25, 32)), (2176, 2816, (25, 32)), (2177, 2816, (25, 32)), (3840, 1024, (17, 24)), (3841, 1024, (17, 24)),
    (600, 640, (17, 24)), (600, 768, (17, 24)), (4736, 640, (13, 16)), (4737, 640, (13, 16)), (9472, 640, (9, 13, 16)), (9473, 640, (9, 13, 16)),
    (18944, 640, (9, 12, 13)), (18945, 640, (9, 12, 13))])
def test_both_sides_of_the_lines_of_tiles(n, k, ms):
    """Where the number of tiles or of a stage's groups decides on the kernel."""
    nz, sg, sc, x = oracle.make_case(n, k, seed=n, batch=max(ms))
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    wd = torch.from_numpy(oracle.unpack_bitmasks(nz, sg).astype(np.float32) * np.repeat(sc.astype(np.float32), 128, axis=1)).cuda().double()
    want, size = dev[3].double() @ wd.T, dev[3].double().abs() @ wd.T.abs()
    for m in ms:
        y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")
        tl.ternary_gemm_packed(dev[3][:m].contiguous(), w, y, m)
        assert (y[m] == 7.0).all()
        bound = k * 2.0 ** -23 * size[:m] + 2.0 ** -11 * want[:m].abs() + 2.0 ** -25      # as above
        assert ((y[:m].double() - want[:m]).abs() <= bound).all(), m
    tl.check_device_errors()


@pytest.mark.parametrize("n", [4, 5, 8, 9, 16, 17, 32, 33, 65])
def test_matrices_packed_back_to_back(n):
    """q|k|v and gate|up of a prompt in one launch each, k and v of 48 rows, whose borders fall inside the tiles of 64
    and 128 features: the logits show every row of every output, through the attention and the gate."""
    cfg = tf.TllmConfig(vocab_size=512, hidden_dim=384, intermediate_dim=640, n_layers=1, n_heads=24, n_kv_heads=3, head_dim=16,
                        max_seq_len=80, rope_theta=10000.0, rms_norm_eps=1e-5)
    model = tf.random_model(cfg, seed=n)
    dec = tl.Decoder(model, int8_decode=False)
    t = np.random.default_rng(n).integers(0, cfg.vocab_size, n).astype(np.int32)
    got = dec.forward(torch.from_numpy(t).cuda(), 0).double().cpu().numpy()
    want = layer_oracle.Transformer(model, int8_decode=False).forward(list(t), 0).astype(np.float64)
    tl.check_device_errors()
    # one layer in FP16: two roundings per operator, on kernels that sum in another order
    assert np.linalg.norm(got - want) <= 1e-2 * np.linalg.norm(want)
    dec.close()


@pytest.mark.parametrize("hidden,inter,heads,kv_heads", [(128, 128, 2, 1), (1152, 3200, 18, 9), (2304, 6784, 36, 12), (4096, 11008, 64, 8)])
def test_step_of_one_vector(hidden, inter, heads, kv_heads):
    """FP16 steps, whose products make their vector (norm with and without a residual, SwiGLU) inside the launch: one and uneven
    numbers of groups, one to eight CTAs a tile, matrices that stay with the GEMV; against the oracle, with the limits of the
    decoder's tests, and against the same token in lock step, which takes the other kernels."""
    cfg = tf.TllmConfig(vocab_size=777, hidden_dim=hidden, intermediate_dim=inter, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=64,
                        max_seq_len=16, rope_theta=10000.0, rms_norm_eps=1e-5)
    model = tf.random_model(cfg, seed=hidden)
    dec, ora = tl.Decoder(model, int8_decode=False, max_batch=5), layer_oracle.Transformer(model, int8_decode=False)
    tokens = np.random.default_rng(hidden).integers(0, cfg.vocab_size, 3).astype(np.int32)
    for i, token in enumerate(tokens):
        ids = torch.from_numpy(np.repeat(token, 5).astype(np.int32)).cuda()
        both = dec.forward_batch(ids, i).clone()
        got = dec.forward(ids[:1], i).float()
        want = torch.from_numpy(np.asarray(ora.forward([int(token)], i), np.float32)).cuda()
        scale = max(1.0, want.abs().max().item())
        assert (got - want).abs().max().item() <= 2e-2 * scale, f"step {i}"
        assert (got - both[0].float()).abs().max().item() <= 2e-2 * scale, f"step {i}, lock step"
    tl.check_device_errors()
    dec.close()


@pytest.mark.parametrize("m", [5, 8, 9])
def test_more_tiles_than_a_grid_is_high(m):
    """65537 tiles of 64 features and a ragged one: more than the second or third dimension of a grid holds."""
    n, k = 65536 * 64 + 69, 128
    gen = torch.Generator(device="cuda").manual_seed(m)
    words = lambda: torch.randint(-2 ** 31, 2 ** 31, (n, k // 32), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    nz = words()
    sg, sc = words() & nz, (torch.rand(n, 1, generator=gen, device="cuda") + 0.5).half()
    w = tl.PreparedWeight(nz, sg, sc, n, k, register=False, keep_source=False)
    x = torch.randn(m, k, generator=gen, device="cuda").half()
    y = torch.full((m, n), 9.0, device="cuda", dtype=torch.float16)
    tl.ternary_gemv_packed(w, x, y, batch=m)
    shift = torch.arange(32, device="cuda", dtype=torch.int32)
    for rows in (slice(0, 130), slice(n // 2, n // 2 + 130), slice(n - 200, n)):
        t = (((nz[rows, :, None] >> shift) & 1) * (2 * ((sg[rows, :, None] >> shift) & 1) - 1)).reshape(-1, k).double()
        want = (x.double() @ t.T) * sc[rows, 0].double()
        # 128 exact products, their sums in FP32, each cut or rounded once, and one rounding to FP16
        size = (x.double().abs() @ t.abs().T) * sc[rows, 0].double()
        assert ((y[:, rows].double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -16 * size + 1e-7).all()
    tl.check_device_errors()
