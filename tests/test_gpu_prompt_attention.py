"""Attention of several FP16 queries on tcgen05 (csrc/grouped_prompt.cu) behind attention_forward,
against the numpy restatement in 64 bits: edges of the 128-query and 128-position tiles, queries
behind a context, both head sizes, groups of heads, several sequences, full caches."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import layer_ops as ops

pytestmark = pytest.mark.gpu
f16 = np.float16


def exact(q, kc, vc, kv_len):
    b, s, h, d = q.shape
    group = h // kc.shape[1]
    out = np.empty(q.shape)
    seen = np.arange(kv_len)[None, :] <= kv_len - s + np.arange(s)[:, None]
    for i in range(b):
        for j in range(h):
            k, v = kc[i, j // group, :kv_len].astype(np.float64), vc[i, j // group, :kv_len].astype(np.float64)
            z = np.where(seen, q[i, :, j].astype(np.float64) @ k.T / np.sqrt(d), -np.inf)
            p = np.exp(z - z.max(axis=1, keepdims=True))
            out[i, :, j] = (p / p.sum(axis=1, keepdims=True)) @ v
    return out


@pytest.mark.parametrize("b,hq,hk,hd", [(1, 8, 2, 64), (2, 4, 4, 128), (1, 32, 8, 128)])
@pytest.mark.parametrize("seq,kv_len,mx", [(2, 2, 8), (8, 8, 8), (8, 400, 512), (127, 127, 130), (128, 128, 128), (129, 129, 256), (130, 387, 387),
                                           (300, 300, 512), (257, 640, 640)])
def test_prompt_attention(b, hq, hk, hd, seq, kv_len, mx):
    rng = np.random.default_rng(seq * 1000 + kv_len + hd)
    q = (3.0 * rng.standard_normal((b, seq, hq, hd))).astype(f16)
    kc = rng.standard_normal((b, hk, mx, hd)).astype(f16)
    vc = rng.standard_normal((b, hk, mx, hd)).astype(f16)
    kc[:, :, kv_len:], vc[:, :, kv_len:] = np.nan, np.nan       # nothing behind the last position is used
    out = torch.zeros(q.shape, dtype=torch.float16, device="cuda")
    args = [torch.from_numpy(t).cuda() for t in (q, kc, vc)]
    ops.attention_forward(*args, out, b, hq, hk, hd, seq, kv_len, mx)
    tl.check_device_errors()
    want = exact(q, kc, vc, kv_len)
    # FP16 rounding of the result; scores of up to 30 in FP32 sums of 64 or 128 terms move a weight by
    # less than 30 * 128 * 2^-24 = 2.3e-4 of itself in the worst case, and the mean of values by a tenth of that
    err = np.abs(out.cpu().numpy().astype(np.float64) - want)
    assert (err <= 2.0 ** -11 * np.abs(want) + 2e-5 * np.abs(vc[:, :, :kv_len].astype(np.float64)).max()).all(), err.max()


@pytest.mark.parametrize("b,hq,hk,hd,seq,kv_len", [
    (1, 8, 8, 64, 16, 16), (1, 8, 8, 64, 17, 17), (1, 16, 8, 64, 12, 300), (1, 16, 8, 64, 13, 300), (1, 4, 4, 64, 3, 64), (1, 4, 4, 64, 3, 65),
    (1, 4, 4, 64, 4, 32), (1, 4, 4, 64, 4, 33), (1, 6, 2, 64, 5, 128), (1, 6, 2, 64, 5, 129), (1, 6, 2, 64, 5, 256), (1, 6, 2, 64, 5, 257),
    (1, 4, 4, 128, 5, 256), (1, 4, 4, 128, 5, 257), (1, 8, 2, 64, 8, 8), (1, 8, 2, 64, 9, 9), (2, 32, 32, 64, 2, 300), (2, 32, 32, 64, 3, 300),
    (8, 28, 7, 64, 7, 7), (8, 32, 8, 64, 7, 7)])
def test_both_sides_of_the_lines_for_few_queries(b, hq, hk, hd, seq, kv_len):
    """Few queries stay with the form on the CUDA cores up to lines of their own; on either side of each the result is the same."""
    rng = np.random.default_rng(seq + kv_len)
    q, kc, vc = (rng.standard_normal(s).astype(f16) for s in ((b, seq, hq, hd), (b, hk, kv_len, hd), (b, hk, kv_len, hd)))
    out = torch.zeros(q.shape, dtype=torch.float16, device="cuda")
    ops.attention_forward(*[torch.from_numpy(t).cuda() for t in (q, kc, vc)], out, b, hq, hk, hd, seq, kv_len, kv_len)
    tl.check_device_errors()
    want = exact(q, kc, vc, kv_len)
    # as above
    assert (np.abs(out.cpu().numpy().astype(np.float64) - want) <= 2.0 ** -11 * np.abs(want) + 2e-5 * np.abs(vc.astype(np.float64)).max()).all()


@pytest.mark.parametrize("b,hq,hk,hd,seq,kv_len", [
    (1, 1, 1, 64, 6, 32), (1, 1, 1, 64, 6, 33), (1, 4, 4, 64, 3, 48), (1, 4, 4, 64, 3, 49), (1, 8, 8, 64, 4, 128), (1, 8, 8, 64, 4, 129),
    (1, 8, 8, 64, 8, 208), (1, 8, 8, 64, 8, 209), (1, 9, 9, 64, 8, 200), (1, 4, 4, 128, 4, 160), (1, 4, 4, 128, 4, 161), (1, 8, 4, 64, 4, 160), (1, 8, 4, 64, 4, 161),
    (8, 32, 8, 64, 3, 20), (9, 32, 8, 64, 3, 20), (8, 7, 1, 64, 8, 20), (1, 16, 4, 64, 8, 20), (2, 32, 8, 64, 8, 32), (48, 8, 4, 64, 1, 9), (24, 8, 4, 64, 2, 9),
    (25, 8, 4, 64, 2, 9), (37, 4, 4, 64, 3, 9), (38, 4, 4, 64, 3, 9)])
def test_more_lines_for_few_queries(b, hq, hk, hd, seq, kv_len):
    test_both_sides_of_the_lines_for_few_queries(b, hq, hk, hd, seq, kv_len)


def test_scores_far_apart():
    """One position's score far above the others', first, last or in between: the running maximum
    moves, and the weights of the others are nothing."""
    hd, n = 64, 300
    for hot in (0, 127, 128, 200):
        rng = np.random.default_rng(hot)
        q, kc, vc = (rng.standard_normal(s).astype(f16) for s in ((1, n, 1, hd), (1, 1, n, hd), (1, 1, n, hd)))
        q[..., 0], kc[..., 0], kc[0, 0, hot, 0] = 30.0, 0.0, 30.0
        out = torch.zeros(q.shape, dtype=torch.float16, device="cuda")
        ops.attention_forward(*[torch.from_numpy(t).cuda() for t in (q, kc, vc)], out, 1, 1, 1, hd, n, n, n)
        want = exact(q, kc, vc, n)
        err = np.abs(out.cpu().numpy().astype(np.float64) - want)
        assert (err <= 2.0 ** -11 * np.abs(want) + 1e-4).all(), (hot, err.max())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("seq,kv_len", [(2, 2), (9, 140), (128, 128), (200, 333)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_do_not_travel_back(hd, seq, kv_len, value):
    """A value of one position is in the outputs of the queries that see it and of no other, the queries
    of its own tile in front of it included."""
    rng = np.random.default_rng(seq + hd)
    b, hq, hk, mx = 2, 4, 2, kv_len + 5
    q = rng.standard_normal((b, seq, hq, hd)).astype(f16)
    kc, vc = (rng.standard_normal((b, hk, mx, hd)).astype(f16) for _ in range(2))
    kc[:, :, kv_len:], vc[:, :, kv_len:] = np.nan, np.nan
    want = exact(q, kc, vc, kv_len)
    bound = 2.0 ** -11 * np.abs(want) + 2e-5 * np.abs(vc[:, :, :kv_len].astype(np.float64)).max()     # as above
    for first in (kv_len - 1, kv_len - seq + seq // 2):           # seen by the last query alone, by half of them
        v, k = vc.copy(), kc.copy()
        v[1, 1, first, 3] = value
        if first == kv_len - 1:
            k[1, 1, first] = value                                # its scores as well
        out = torch.zeros(q.shape, dtype=torch.float16, device="cuda")
        ops.attention_forward(*[torch.from_numpy(t).cuda() for t in (q, k, v)], out, b, hq, hk, hd, seq, kv_len, mx)
        tl.check_device_errors()
        got = out.cpu().numpy().astype(np.float64)
        hit = np.zeros(q.shape, dtype=bool)
        sees = np.arange(seq) >= first - (kv_len - seq)
        hit[1, sees, 2:] = True if first == kv_len - 1 else np.arange(hd) == 3
        assert (np.abs(got - want) <= bound)[~hit].all()
        if first != kv_len - 1:
            assert ((got[hit] == value) | (np.isnan(got[hit]) & np.isnan(value))).all()
