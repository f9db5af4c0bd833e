"""Selective scan of a BF16 prompt by a channel per thread (csrc/mixers.cu): edges of the tiles of 8 tokens, of the time chunks and of the
blocks of 128 channels, every count of states that it takes, and inputs that it leaves to the general kernel, against 64 bits."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu


def shifted(t, offset):
    """The same values `offset` elements behind an allocation's start."""
    flat = torch.empty(t.numel() + offset, device="cuda", dtype=t.dtype)[offset:]
    return flat.copy_(t.flatten()).view(t.shape)


def exact(x, dt, B, C, z, A, D, S):
    """(outputs, their sums of magnitudes, state, its sums of magnitudes) in 64 bits; S is the state before."""
    M, y, size = S.abs(), [], []
    for t in range(x.shape[1]):
        f, dx = torch.exp(dt[:, t, :, None] * A), (dt[:, t] * x[:, t])[..., None] * B[:, t, None]
        S, M = f * S + dx, f * M + dx.abs()
        g = 1.0 if z is None else z[:, t] * torch.sigmoid(z[:, t])
        d = 0.0 if D is None else D * x[:, t]
        y.append(((S * C[:, t, None]).sum(-1) + d) * g)
        size.append(((M * C[:, t, None].abs()).sum(-1) + abs(d)) * abs(g))
    return torch.stack(y, 1), torch.stack(size, 1), S, M


@pytest.mark.parametrize("channels,states,shift", [(8, 1, 0), (120, 7, 0), (128, 16, 0), (136, 15, 0), (264, 2, 0), (24, 16, 0), (40, 16, 3),
                                                   (40, 17, 0)])
@pytest.mark.parametrize("n,start", [(5, 0), (8, 3), (9, 0), (31, 1), (64, 0), (65, 7), (130, 0), (515, 2)])
def test_selective_scan_tiles(n, start, channels, states, shift):
    gen = torch.Generator(device="cuda").manual_seed(channels * 1000 + n)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    with_gate, with_d, s8 = n % 2 == 1, n % 4 != 0, (states + 7) // 8 * 8
    x, z, bc = rand(2, n, channels).bfloat16(), rand(2, n, channels).bfloat16(), rand(2, n, 2 * s8).bfloat16()
    dt = torch.rand(2, n, channels, generator=gen, device="cuda") * 0.3 + 0.001
    a2, D, state = -torch.exp(rand(channels, states) * 2 - 1), rand(channels), rand(2, channels, states)
    before = state.double() if start else torch.zeros_like(state).double()
    if not start: state.fill_(float("nan"))                     # a new sequence must not read it
    y = torch.full((2, n + 1, channels), 7.0, device="cuda", dtype=torch.bfloat16)
    out = y.flatten()[:2 * n * channels].view(2, n, channels)
    ops.selective_scan(shifted(x, shift), shifted(dt, shift), bc, shifted(z, shift) if with_gate else None, a2, D if with_d else None, state,
                       out, channels, states, 2, n, start)
    assert (y.flatten()[2 * n * channels:] == 7.0).all()
    want, size, S, M = exact(x.double(), dt.double(), bc[..., :states].double(), bc[..., s8:s8 + states].double(), z.double() if with_gate else None,
                             a2.double() * 0.6931471805599453, D.double() if with_d else None, before)
    # FP32 all through: a step rounds the exponent's product, the exponential (2 ulp), the input's product and the sum, and the error of
    # one token stays in the state for the rest of the sequence at most; the output is rounded to BF16 last
    eps = 6 * (n + states) * 2.0 ** -24
    assert ((state.double() - S).abs() <= eps * M + 1e-30).all()
    assert ((out.double() - want).abs() <= eps * size + 2.0 ** -8 * want.abs() + 1e-30).all()
    tl.check_device_errors()


def test_values_that_are_not_finite():
    """An infinite input is felt by its own channel and sequence alone, from its token on."""
    n, C, S = 100, 136, 16
    x = torch.ones(2, n, C, device="cuda", dtype=torch.bfloat16)
    x[1, 70, 130] = float("inf")
    bc, dt = torch.ones(2, n, 2 * S, device="cuda", dtype=torch.bfloat16), torch.full((2, n, C), 0.1, device="cuda")
    y, state = torch.empty_like(x), torch.empty(2, C, S, device="cuda")
    ops.selective_scan(x, dt, bc, None, -torch.ones(C, S, device="cuda"), torch.ones(C, device="cuda"), state, y, C, S, 2, n, 0)
    bad = torch.zeros(2, n, C, device="cuda", dtype=torch.bool)
    bad[1, 70:, 130] = True
    assert (torch.isfinite(y) == ~bad).all() and torch.equal(y[0], y[1].where(~bad[1], y[0]))
    tl.check_device_errors()
