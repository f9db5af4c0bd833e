"""Causal convolution of few and of very many tokens, gated scan of few and of many CTAs (csrc/mixers.cu), against 64 bits."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import mixed_oracle as O
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_conv_of_few_tokens(n, taps, dt):
    gen = torch.Generator(device="cuda").manual_seed(10 * n + taps)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    C, seqs = 264, 2
    x, w, b = rand(seqs, n, C).to(dt), rand(C, taps), rand(C)
    for start in (0, 7):
        state = rand(seqs, taps - 1, C).to(dt)
        before = state.double() if start else torch.zeros_like(state).double()
        if not start: state.fill_(float("nan"))                     # a new sequence must not read it
        y = torch.full((seqs + 1, n, C), 7.0, device="cuda", dtype=dt)
        ops.causal_conv(x, w, b, state, y[:seqs], C, taps, seqs, n, start, "silu")
        full = torch.cat([before, x.double()], dim=1)
        z = sum(full[:, j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
        size = sum(full[:, j:j + n].abs() * w[:, j].double().abs() for j in range(taps)) + b.double().abs()
        want = z * torch.sigmoid(z)
        # taps products and sums in FP32, through SiLU's slope of at most 1.1 and its own FP32 steps, then the type of the result
        bound = 1.1 * (taps + 1) * 2.0 ** -23 * size + 2.0 ** -20 * want.abs() + (2.0 ** -8 if dt == BF16 else 0.0) * want.abs() + 1e-30
        assert ((y[:seqs].double() - want).abs() <= bound).all() and (y[seqs] == 7.0).all()
        assert torch.equal(state.double(), full[:, n:])
    tl.check_device_errors()


@pytest.mark.parametrize("taps", [4, 9])
def test_conv_of_more_chunks_than_a_grid_is_high(taps):
    n, C = 65535 * 16 + 40, 8
    gen = torch.Generator(device="cuda").manual_seed(taps)
    x = torch.randn(n, C, generator=gen, device="cuda").to(BF16)
    w, state = torch.randn(C, taps, generator=gen, device="cuda"), torch.empty(taps - 1, C, device="cuda", dtype=BF16)
    y = torch.empty_like(x)
    ops.causal_conv(x, w, None, state, y, C, taps, 1, n, 0)
    full = torch.cat([torch.zeros(taps - 1, C, device="cuda", dtype=torch.float64), x.double()])
    want, size = (sum(f(full[j:j + n]) * f(w[:, j].double()) for j in range(taps)) for f in (lambda t: t, torch.abs))
    assert ((y.double() - want).abs() <= taps * 2.0 ** -23 * size + 2.0 ** -8 * want.abs() + 1e-30).all()
    assert torch.equal(state, x[n - taps + 1:])
    tl.check_device_errors()


@pytest.mark.parametrize("dt,channels,seqs", [(F32, 1280, 18), (F32, 1280, 19), (BF16, 1280, 40), (BF16, 1288, 41)])
def test_gated_scan_of_many_ctas(dt, channels, seqs):
    """Either side of the line between the second pass's tiles of 8 and 4 tokens, chunks that end inside both."""
    n, C = 67, channels
    rng = np.random.default_rng(seqs)
    u, y = (torch.from_numpy(rng.standard_normal((seqs, n, C))).to(dt) for _ in range(2))
    r, i = (rng.uniform(0.01, 1, (seqs, n, C)).astype(np.float32) for _ in range(2))
    lam = rng.uniform(-12, 1, C).astype(np.float32)
    gates, soft = torch.from_numpy(np.stack([r, i], axis=2)).cuda(), torch.from_numpy(O.softplus(lam.astype(np.float64)).astype(np.float32)).cuda()
    state, out = torch.full((seqs, C), float("nan"), device="cuda"), torch.full((seqs + 1, n, C), 7.0, device="cuda", dtype=dt)
    ops.gated_scan(u.cuda(), gates, soft, y.cuda(), state, out[:seqs], C, 1, seqs, n, 0)
    assert (out[seqs] == 7.0).all()
    for s in (0, 1, seqs - 1):
        want = O.gated_linear_recurrence(u[s].double().numpy(), r[s].astype(np.float64), i[s].astype(np.float64), lam.astype(np.float64)) * O.gelu_tanh(y[s].double().numpy())
        got = out[s].double().cpu().numpy()
        # as the operator's other tests: of the largest value, FP32 sums over the tokens, or the rounding to BF16
        assert np.abs(got - want).max() <= (6e-3 if dt == BF16 else 2e-5) * np.abs(want).max()
    tl.check_device_errors()


@pytest.mark.parametrize("n", [64, 66, 80, 81, 82, 94, 95, 96, 97, 1040, 1056])
def test_gated_scan_of_chunks_of_all_lengths(n):
    """Chunks of 32 to 48 tokens, whose last tile of 16 is whole, nearly whole or nearly empty."""
    C, rng = 72, np.random.default_rng(n)
    u, y = (torch.from_numpy(rng.standard_normal((n, C))).float() for _ in range(2))
    r, i = (rng.uniform(0.01, 1, (n, C)).astype(np.float32) for _ in range(2))
    lam = rng.uniform(-12, 1, C).astype(np.float32)
    soft = torch.from_numpy(O.softplus(lam.astype(np.float64)).astype(np.float32)).cuda()
    state, out = torch.full((1, C), float("nan"), device="cuda"), torch.full((n + 1, C), 7.0, device="cuda")
    ops.gated_scan(u.cuda(), torch.from_numpy(np.stack([r, i], axis=1)).cuda(), soft, y.cuda(), state, out[:n], C, 1, 1, n, 0)
    want = O.gated_linear_recurrence(u.double().numpy(), r.astype(np.float64), i.astype(np.float64), lam.astype(np.float64)) * O.gelu_tanh(y.double().numpy())
    assert np.abs(out[:n].double().cpu().numpy() - want).max() <= 2e-5 * np.abs(want).max() and (out[n] == 7.0).all()
    tl.check_device_errors()
