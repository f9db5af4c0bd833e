"""Latent attention over a prompt on tcgen05 (csrc/grouped_prompt.cu): edges of the tiles of 128 queries and positions, the
sizes of the key's two parts and of the values, sinks and gates, against 64 bits, and values that are not finite."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu
RANK = 24


def inputs(H, dim, rot, vdim, n, ctx, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    cache = torch.full((ctx + 5, RANK + rot), float("nan"), device="cuda", dtype=torch.bfloat16)     # nothing of it but the keys is read
    cache[:ctx, RANK:] = rand(ctx, rot)
    return 1.5 * rand(n, H, dim + rot), rand(ctx, H, dim), rand(ctx, H, vdim), cache, torch.randn(H, generator=gen, device="cuda") * 3, rand(n, H)


def run(q, k, v, cache, sink, gate, scale):
    n, H, dq = q.shape
    ctx, dim, vdim = k.shape[0], k.shape[2], v.shape[2]
    out = torch.full((n + 1, H, vdim), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.latent_attention_expanded(q, k, v, cache, sink, gate, out, H, dim, dq - dim, vdim, RANK, scale, ctx + 5, n, ctx - n)
    assert (out[n] == 7.0).all()
    return out[:n]


def exact(q, k, v, cache, sink, gate, scale):
    """(outputs, sums of magnitudes of weight and value) in 64 bits."""
    n, H, ctx = q.shape[0], q.shape[1], k.shape[0]
    full = torch.cat([k.double(), cache[:ctx, None, RANK:].double().expand(ctx, H, -1)], dim=2)
    s = torch.einsum("nhd,chd->hnc", q.double(), full) * scale
    s.masked_fill_(torch.arange(ctx, device="cuda")[None, :] > torch.arange(ctx - n, ctx, device="cuda")[:, None], -torch.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(H, n, 1)], dim=2)
    p = torch.softmax(s, dim=2)[:, :, :ctx]
    o, size = torch.einsum("hnc,chd->nhd", p, v.double()), torch.einsum("hnc,chd->nhd", p, v.double().abs())
    if gate is not None:
        g = torch.sigmoid(gate.double())[:, :, None]
        o, size = o * g, size * g
    return o, size


@pytest.mark.parametrize("dim,rot,vdim", [(64, 0, 64), (64, 64, 128), (128, 64, 128), (128, 128, 64), (192, 64, 64)])
@pytest.mark.parametrize("n,start", [(1, 200), (16, 0), (127, 0), (128, 0), (129, 0), (130, 77), (257, 128), (40, 500), (600, 1)])
def test_against_64_bits(dim, rot, vdim, n, start):
    scale = (dim + rot) ** -0.5
    q, k, v, cache, sink, gate = inputs(3, dim, rot, vdim, n, start + n, n + dim)
    for s, g in ((None, None), (sink, gate)):
        got = run(q, k, v, cache, s, g, scale)
        want, size = exact(q, k, v, cache, s, g, scale)
        # scores: sums of dim + rot exact products in FP32, and the exponential's 2^-22; weights in two BF16 parts (2^-17), their sums
        # and products in FP32; one rounding to BF16
        worst = (dim + rot) * 2.0 ** -23 * scale * (q.double().norm(dim=2).max() * (k.double().norm(dim=2).max() + cache[:start + n, RANK:].double().norm(dim=1).max()))
        bound = (2 * worst + 2.0 ** -16 + (start + n) * 2.0 ** -23) * size + 2.0 ** -8 * want.abs() + 1e-6
        assert ((got.double() - want).abs() <= bound).all()
    tl.check_device_errors()


@pytest.mark.parametrize("n,start", [(1, 62), (1, 63), (1, 64), (64, 0), (65, 0), (20, 44), (20, 45)])
def test_both_sides_of_one_tile_of_keys(n, start):
    """Up to 64 positions go another way (csrc/latent_attention.cu)."""
    test_against_64_bits(128, 64, 128, n, start)


def test_values_that_are_not_finite():
    """An infinity among a position's values reaches the queries that see it and no other."""
    n, H, scale = 300, 2, 0.1
    q, k, v, cache, sink, gate = inputs(H, 64, 64, 128, n, n, 3)
    v[140, 1, 5] = float("inf")
    got = run(q, k, v, cache, sink, gate, scale)
    assert got[:, 0].isfinite().all() and got[:140].isfinite().all() and (got[140:, 1, 5] == float("inf")).all()
    want, size = exact(q[:140], k[:140], v[:140], cache[:145], sink, gate[:140], scale)
    assert ((got[:140].double() - want).abs() <= 2.0 ** -7 * size + 1e-6).all()
    assert got[140:, 1, :5].isfinite().all() and got[140:, 1, 6:].isfinite().all()
    tl.check_device_errors()
