"""Attention of one new token on clusters (csrc/attention_step.cu): edges of a warp's, a CTA's and a cluster's share of the
positions, more positions than one round of copies holds, every group size, against 64 bits; nothing behind the new position is read, and
other sequences and positions of the cache stay as they are."""
import ctypes

import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import _lib
from ternary_llm_b200 import layer_ops as ops
from ternary_llm_b200 import tllm_format as tf

pytestmark = pytest.mark.gpu
THETA = 500000.0


def rotated(x, pos):
    """Rotation in 64 bits, rounded to FP16 as the caches hold it; x [heads, hd]."""
    hd = x.shape[1]
    angle = pos * THETA ** (-2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd)
    u, v = x[:, 0::2].double(), x[:, 1::2].double()
    return torch.stack([u * angle.cos() - v * angle.sin(), u * angle.sin() + v * angle.cos()], dim=-1).reshape(x.shape).half()


def softmax_rows(q, k, v):
    """q [G, hd], k and v [n, hd]: outputs in 64 bits, and their sums of magnitudes."""
    p = torch.softmax(q.double() @ k.double().T * q.shape[1] ** -0.5, dim=1)
    return p @ v.double(), p @ v.double().abs()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("pos", [0, 1, 3, 15, 31, 32, 63, 64, 127, 128, 129, 511, 1000, 1023, 2047, 2300, 4500])
def test_one_sequence(pos, group, hd):
    hk, mx = 3, pos + 5
    gen = torch.Generator().manual_seed(pos * 10 + group)
    q, k, v = (torch.randn(h, hd, generator=gen).half() for h in (hk * group, hk, hk))
    kc, vc = (torch.full((hk, mx, hd), float("nan"), dtype=torch.float16) for _ in range(2))
    kc[:, :pos], vc[:, :pos] = torch.randn(hk, pos, hd, generator=gen).half(), torch.randn(hk, pos, hd, generator=gen).half()
    kd, vd, out = kc.cuda(), vc.cuda(), torch.full((hk * group + 1, hd), 7.0, dtype=torch.float16, device="cuda")
    qd = q.cuda()
    ops.attention_decode(qd, k.cuda(), v.cuda(), kd, vd, out[:-1], hk * group, hk, hd, pos, THETA, mx)
    assert (qd.cpu() == q).all() and (out[-1] == 7.0).all()
    kn, vn = kd.cpu(), vd.cpu()
    assert torch.equal(kn[:, :pos], kc[:, :pos]) and torch.equal(vn[:, :pos], vc[:, :pos])
    assert kn[:, pos + 1:].isnan().all() and vn[:, pos + 1:].isnan().all() and torch.equal(vn[:, pos], v)
    # the angle is an FP32 product of an FP32 power: a few 2^-24 of it, beside one rounding to FP16
    turn = 8 * 2.0 ** -24 * pos + 2.0 ** -10
    assert ((kn[:, pos].double() - rotated(k, pos).double()).abs() <= turn * k.abs().amax() * 1.5 + 1e-6).all()
    qr = rotated(q, pos)
    for h in range(hk):
        want, size = softmax_rows(qr[h * group:(h + 1) * group], kn[h, :pos + 1], vn[h, :pos + 1])
        got = out[h * group:(h + 1) * group].double().cpu()
        # a query off by `turn` moves a score by at most that times |q| |k| / sqrt(hd), and an output by twice that of the magnitudes
        score = turn * (q[h * group:(h + 1) * group].double().norm(dim=1) * kn[h, :pos + 1].double().norm(dim=1).max() * hd ** -0.5)
        bound = (2 * score[:, None] + 2.0 ** -18) * size + 2.0 ** -11 * want.abs() + 1e-7
        assert ((got - want).abs() <= bound).all()
    tl.check_device_errors()


def test_values_that_are_not_finite():
    """Scores of NaN leave a head's output zero; infinities of values seen reach the output, the others of the cluster's parts included."""
    hk, group, hd, pos = 2, 4, 64, 700
    gen = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(h, hd, generator=gen).half().cuda() for h in (hk * group, hk, hk))
    kc, vc = (torch.randn(hk, pos + 1, hd, generator=gen).half().cuda() for _ in range(2))
    q[1, 5] = float("nan")
    vc[1, 3, 7] = float("inf")
    out = torch.empty(hk * group, hd, dtype=torch.float16, device="cuda")
    ops.attention_decode(q, k, v, kc, vc, out, hk * group, hk, hd, pos, THETA, pos + 1)
    assert (out[1] == 0).all() and out[[0, 2, 3]].isfinite().all()
    assert (out[4:, 7] == float("inf")).all() and out[4:, :7].isfinite().all() and out[4:, 8:].isfinite().all()


def test_first_call_under_capture():
    """No scratch: a size that no call has had before may be captured."""
    hk, group, hd, pos, mx = 64, 8, 128, 300, 20000                     # records of this cache would be larger than any other test's
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(h, hd, generator=gen, device="cuda").half() for h in (hk * group, hk, hk))
    kc, vc = (torch.zeros(hk, mx, hd, dtype=torch.float16, device="cuda") for _ in range(2))
    kc[:, :pos], vc[:, :pos] = (torch.randn(hk, pos, hd, generator=gen, device="cuda").half() for _ in range(2))
    out = [torch.zeros(hk * group, hd, dtype=torch.float16, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.attention_decode(q, k, v, kc, vc, out[0], hk * group, hk, hd, pos, THETA, mx)
    graph.replay()
    ops.attention_decode(q, k, v, kc, vc, out[1], hk * group, hk, hd, pos, THETA, mx)
    assert out[1].any() and torch.equal(*out)
    tl.check_device_errors()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
def test_parts_run_at_once(group, hd):
    """A KV head is shared by more CTAs only while all of them run at the same time, whatever the registers of a group's kernel leave;
    one sequence behind a long cache is shared by as many as a cluster has."""
    def plan(batch, pos, hk=8):
        parts, at_once = ctypes.c_int(), ctypes.c_int()
        _lib.check(_lib.lib().tllm_b200_attention_step_plan(group * hk, hk, hd, batch, pos, ctypes.byref(parts), ctypes.byref(at_once)))
        return parts.value, at_once.value
    assert plan(1, 4000)[0] == 8 and plan(1, 64)[0] == 2 and plan(1, 63)[0] == 1 and plan(1000, 4000)[0] == 1
    for batch in range(1, 40):
        parts, at_once = plan(batch, 4000)
        assert parts == 1 or batch * 8 * parts <= at_once


@pytest.mark.parametrize("group,hd", [(8, 64), (8, 128), (4, 128), (1, 128)])
@pytest.mark.parametrize("batch", [3, 4, 18])
def test_lock_step_of_every_group(batch, group, hd):
    """As below, behind more positions than one round of a CTA's copies holds, where groups share a head differently."""
    cfg = tf.TllmConfig(vocab_size=500, hidden_dim=256, intermediate_dim=256, n_layers=2, n_heads=8 * group, n_kv_heads=8, head_dim=hd,
                        max_seq_len=640, rope_theta=10000.0, rms_norm_eps=1e-5)
    dec = tl.Decoder(tf.random_model(cfg, seed=5), int8_decode=False, max_batch=batch)
    rng = np.random.default_rng(batch)
    ctx, last = torch.from_numpy(rng.integers(0, 500, (batch, 600)).astype(np.int32)).cuda(), torch.from_numpy(rng.integers(0, 500, batch).astype(np.int32)).cuda()
    rows = []
    for order in (list(range(batch)), list(range(batch))[::-1]):
        for place, i in enumerate(order):
            dec.forward_seq(place, ctx[i].clone(), 0)
        rows.append(dec.forward_batch(last[order].contiguous(), 600).clone())
    assert torch.equal(rows[0], rows[1].flip(0))
    dec.close()


@pytest.mark.parametrize("batch", [3, 24, 50])
def test_lock_step_equals_single_sequences(batch):
    """Sequences in lock step read their own caches: each gives what the same sequence gives in another place of the batch."""
    cfg = tf.TllmConfig(vocab_size=999, hidden_dim=256, intermediate_dim=256, n_layers=2, n_heads=16, n_kv_heads=8, head_dim=64, max_seq_len=160,
                        rope_theta=10000.0, rms_norm_eps=1e-5)
    dec = tl.Decoder(tf.random_model(cfg, seed=5), int8_decode=False, max_batch=batch)
    rng = np.random.default_rng(batch)
    ctx = rng.integers(0, 999, (batch, 130)).astype(np.int32)
    last = torch.from_numpy(rng.integers(0, 999, batch).astype(np.int32)).cuda()
    order = np.arange(batch)[::-1].copy()
    rows = []
    for perm in (np.arange(batch), order):
        for i in range(batch):
            dec.forward_seq(i, torch.from_numpy(ctx[perm[i]]).cuda(), 0)
        rows.append(dec.forward_batch(last[torch.from_numpy(perm).cuda()].contiguous(), 130).clone())
    assert torch.equal(rows[0], rows[1][torch.from_numpy(order).cuda()])
    dec.close()
