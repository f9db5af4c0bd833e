"""The dense GEMM of prompts (csrc/dense_gemm.cu) at sizes that take each of its tiles, 64, 128 and 256 features of one CTA,
128 and 256 of a pair, 64 of two, four and eight CTAs that share K: whole and ragged rows, features and columns, one round of tiles and several, against 64 bits."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import mixed_ops as ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [9, 128, 129, 256, 257, 300, 385, 1000])
@pytest.mark.parametrize("n,k", [(64, 64), (500, 4104), (1000, 2056), (2048, 512), (2050, 4104), (4096, 2048), (4100, 72), (9000, 1032)])
@pytest.mark.parametrize("glu", [False, True])
def test_product(m, n, k, glu):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(n * (2 if glu else 1), k, generator=gen, device="cuda") * k ** -0.5).bfloat16()
    bias = None if glu else torch.randn(n, generator=gen, device="cuda")
    y = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16 if glu else torch.float32)
    ops.dense_linear(x, w, y, m, n, k, bias=bias, glu=glu)
    assert (y[m] == 7.0).all()
    # products are exact, K sums in FP32, each cut or rounded once: K * 2^-23 of the sum of magnitudes
    p, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T * (k * 2.0 ** -23)
    if glu:
        want, bound = p[:, :n] * p[:, n:], 1.1 * (size[:, :n] * p[:, n:].abs() + size[:, n:] * p[:, :n].abs()) + 1e-9
        bound = bound + 2.0 ** -8 * want.abs()                                       # BF16
    else:
        want = p + bias.double()
        bound = size + 2.0 ** -23 * want.abs()
    assert ((y[:m].double() - want).abs() <= bound).all()
    tl.check_device_errors()
