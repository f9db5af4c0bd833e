"""Absorbed latent attention (csrc/latent_attention.cu): tiles of 32 and of 64 positions, borders of the splits, partly filled tiles of rows
and several sequences, against 64 bits."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_seq,n,start", [(1, 1, 0), (1, 1, 30), (1, 1, 31), (1, 1, 32), (1, 1, 63), (1, 1, 64), (1, 3, 95), (3, 1, 700), (1, 1, 4200),
                                           (1, 1, 9471), (1, 1, 9472), (37, 1, 255), (37, 1, 256), (2, 9, 33)])
@pytest.mark.parametrize("heads,rank,rot", [(5, 72, 24), (16, 512, 64), (40, 8, 8)])
def test_absorbed_steps(n_seq, n, start, heads, rank, rot):
    gen = torch.Generator(device="cuda").manual_seed(start * 100 + heads)
    dk, ctx, max_seq = rank + rot, start + n, start + n + 3
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, sink, scale = rand(n_seq, n, heads, dk).bfloat16(), rand(heads) if heads == 16 else None, 2 * dk ** -0.5
    cache = torch.full((n_seq, max_seq, dk), float("nan"), device="cuda", dtype=torch.bfloat16)
    cache[:, :ctx] = rand(n_seq, ctx, dk).bfloat16()
    out = torch.full((n_seq * n + 1, heads, rank), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.latent_attention(q, cache, sink, out, heads, rank, rot, scale, max_seq, n_seq, n, start)
    assert (out[n_seq * n] == 7.0).all()
    sees = torch.arange(ctx, device="cuda")[None] <= torch.arange(start, ctx, device="cuda")[:, None]
    for b in range(n_seq):
        k = cache[b, :ctx].double()
        s = torch.einsum("nhd,cd->hnc", q[b].double(), k) * scale
        reach = (torch.einsum("nhd,cd->hnc", q[b].double().abs(), k.abs()) * scale).max()
        s.masked_fill_(~sees, -torch.inf)
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(heads, n, 1)], dim=2)
        p = torch.softmax(s, dim=2)[:, :, :ctx]
        want, size = torch.einsum("hnc,cd->nhd", p, k[:, :rank]), torch.einsum("hnc,cd->nhd", p, k[:, :rank].abs())
        # weights of 16 bits, scores and sums in FP32, the result rounded to BF16
        bound = (2.0 ** -15 + 2 * (dk + ctx) * 2.0 ** -24 * float(reach)) * size + 2.0 ** -8 * want.abs() + 1e-30
        assert ((out[b * n:(b + 1) * n].double() - want).abs() <= bound).all(), b
    tl.check_device_errors()


@pytest.mark.parametrize("n_seq,n,start", [(1, 1, 1023), (1, 1, 1024), (1, 1, 2047), (1, 1, 2048), (4, 1, 1023), (4, 1, 1024), (5, 1, 991), (148, 1, 31),
                                           (149, 1, 31)])
def test_both_sides_of_the_lines_of_tiles(n_seq, n, start):
    """Where tiles go from 32 to 64 positions: by their number, and by the number of records of a row."""
    test_absorbed_steps(n_seq, n, start, 16, 512, 64)
