"""The dense FP16 head on the tensor cores (csrc/fp16_rows.cu) and, up to 8192 rows of one vector, on the CUDA
cores: edges of the 16-row blocks, odd and even numbers of 128-column windows, one vector and batches that fill one, two and more column blocks of the MMA
or need a second pass, against 64 bits."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import layer_ops as ops
from ternary_llm_b200 import tllm_format as tf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 15, 17, 2400, 8192, 8193, 40001])
@pytest.mark.parametrize("cols", [128, 384, 2048, 14336])
def test_one_vector(rows, cols):
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    w = (0.02 * torch.randn(rows, cols, generator=gen, device="cuda")).half()
    x = torch.randn(cols, generator=gen, device="cuda").half()
    y = torch.full((rows + 16,), 7.0, dtype=torch.float16, device="cuda")
    ops.fp16_gemv(w, x, y[:rows], rows, cols)
    torch.cuda.synchronize()
    assert (y[rows:] == 7.0).all()
    want = w.double() @ x.double()
    # cols FP32 roundings of at most the sum of magnitudes, then one to FP16
    bound = cols * 2.0 ** -24 * (w.double().abs() @ x.double().abs()) + 2.0 ** -11 * want.abs() + 2.0 ** -25
    assert ((y[:rows].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("batch", [2, 8, 9, 17, 25, 40])
def test_batch_equals_single_sequences(batch):
    """No layer's sums depend on the vectors beside them: with the layers' products on the same kernel (up to 32
    rows), a sequence's logits in a batch are those of the same sequence in another place of it."""
    cfg = tf.TllmConfig(vocab_size=1003, hidden_dim=256, intermediate_dim=512, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64,
                        max_seq_len=16, rope_theta=10000.0, rms_norm_eps=1e-5)
    model = tf.random_model(cfg, seed=5)
    dec = tl.Decoder(model, int8_decode=False, max_batch=batch)
    tokens = torch.from_numpy(np.random.default_rng(batch).integers(0, cfg.vocab_size, batch).astype(np.int32)).cuda()
    got = dec.forward_batch(tokens, 0).clone()
    turned = dec.forward_batch(tokens.flip(0).contiguous(), 0).clone()
    assert torch.equal(got, turned.flip(0))
    for b in {0, batch // 2, batch - 1}:
        one = dec.forward_seq(0, tokens[b:b + 1], 0).double()
        # two FP16 roundings per operator of one layer, on different kernels
        assert (got[b].double() - one).norm() <= 1e-2 * one.norm()
    tl.check_device_errors()
    dec.close()


@pytest.mark.parametrize("cols", [2048, 12288])
def test_products_of_one_sign(cols):
    """The tensor cores cut their sums; the rounding of the result to FP16 is all that is left of the error even where every
    product has the same sign and the cuts add up."""
    rows = 12304
    gen = torch.Generator(device="cuda").manual_seed(cols)
    w = (0.02 * torch.rand(rows, cols, generator=gen, device="cuda")).half()
    x = torch.rand(cols, generator=gen, device="cuda").half()
    y = torch.empty(rows, dtype=torch.float16, device="cuda")
    ops.fp16_gemv(w, x, y, rows, cols)
    want = w.double() @ x.double()
    # sums eight cuts of 2^-23 long and FP32 rounding of 96 of them move a result by less than 2^-20 of itself: the rounding to
    # FP16, 2^-11 at most and 2^-12.8 in the mean square, grows by less than a hundredth
    assert (y.double() - want).norm() <= 1.01 * (want.half().double() - want).norm()


@pytest.mark.parametrize("producer", ["gemm", "embedding"])
def test_matrix_made_by_the_launch_before(producer):
    """W is a tensor like any other: the operators that can make it let the next launch start early, and
    that launch reads none of it before they have ended."""
    rows, cols, k = 12304, 2048, 1024
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(cols, generator=gen, device="cuda").half()
    a = (0.05 * torch.randn(2, rows, k, generator=gen, device="cuda")).half()
    b = torch.randn(cols, k, generator=gen, device="cuda").half()
    table = torch.randn(2 * rows, cols, generator=gen, device="cuda").half()
    ids = torch.randperm(2 * rows, generator=gen, device="cuda").to(torch.int32).view(2, rows)
    w, y = torch.zeros(rows, cols, dtype=torch.float16, device="cuda"), torch.empty(2, rows, dtype=torch.float16, device="cuda")
    for i in range(8):
        if producer == "gemm":
            ops.fp16_gemm(a[i & 1], b, w, rows, cols, k)
        else:
            ops.embedding_lookup(table, ids[i & 1], w, rows, cols)
        ops.fp16_gemv(w, x, y[i & 1], rows, cols)
        want = w.double() @ x.double()
        # as above
        bound = cols * 2.0 ** -24 * (w.double().abs() @ x.double().abs()) + 2.0 ** -11 * want.abs() + 2.0 ** -25
        assert ((y[i & 1].double() - want).abs() <= bound).all(), i
