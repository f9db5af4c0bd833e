"""Causal convolution of very many tokens (csrc/mixers.cu), against 64 bits."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


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
