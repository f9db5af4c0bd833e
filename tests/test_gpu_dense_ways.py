"""The dense GEMM of prompts (csrc/dense_gemm.cu) at sizes that take each of its tiles, 64, 128 and 256 features of one CTA,
128 and 256 of a pair, 64 of two, four and eight CTAs that share K: whole and ragged rows, features and columns, one round of tiles and several, against 64 bits;
batch entries, gates, ranges of the activation and the second output in each of them."""
import ctypes

import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import _lib
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


NONE = 2 ** 31 - 1
# (features of a tile, pairs of CTAs, CTAs that share K)
WAYS = {(64, 0, 1), (128, 0, 1), (256, 0, 1), (128, 1, 1), (256, 1, 1), (64, 0, 2), (64, 0, 4), (64, 0, 8)}


def ask(**sizes):
    args = _lib.DenseArgs(**dict(dict(batch=1, act_hi=NONE, f32_from=NONE), **sizes))
    out = [ctypes.c_int() for _ in range(3)]
    _lib.check(_lib.lib().tllm_b200_dense_way(ctypes.byref(args), *[ctypes.byref(o) for o in out]))
    return tuple(o.value for o in out)


def test_every_way_occurs():
    """The sizes above take all of them."""
    sizes = [(64, 64), (500, 4104), (1000, 2056), (2048, 512), (2050, 4104), (4096, 2048), (4100, 72), (9000, 1032)]
    assert {ask(rows=m, n=n, cols=k, glu=g) for m in (9, 128, 129, 256, 257, 300, 385, 1000) for n, k in sizes for g in (0, 1)} == WAYS


def product(args, x, w, y, **tensors):
    for name, t in dict(tensors, x=x, w=w, y=y).items():
        setattr(args, name, t.data_ptr())
    _lib.check(_lib.lib().tllm_b200_dense_product(ctypes.byref(args), torch.cuda.current_stream().cuda_stream))
    tl.check_device_errors()


def sums(x, w, k):
    """(products, what FP32 sums of K products may be off), x [batch, m, k], w [batch, n, k]"""
    return torch.einsum("bmk,bnk->mbn", x.double(), w.double()), torch.einsum("bmk,bnk->mbn", x.double().abs(), w.double().abs()) * (k * 2.0 ** -23)


@pytest.mark.parametrize("m,n,k,batch,way", [
    (37, 72, 264, 3, (64, 0, 1)), (37, 1030, 4104, 2, (64, 0, 2)), (37, 520, 2056, 2, (64, 0, 4)), (130, 136, 2056, 3, (64, 0, 4)),
    (37, 72, 2056, 3, (64, 0, 8)), (200, 72, 2056, 2, (64, 0, 8)), (300, 2056, 264, 2, (128, 0, 1)), (300, 1030, 4104, 3, (128, 1, 1)),
    (390, 3000, 264, 3, (256, 0, 1)), (300, 2056, 4104, 3, (256, 1, 1))])
@pytest.mark.parametrize("pad", [0, 8])
def test_batch_entries_and_gates(m, n, k, batch, way, pad):
    """Offsets of an entry in X, Y and W, and a gate per row and entry, with and without whole 16-byte pieces in Y."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    rows = n + pad                                                   # rows of an entry of W, the last of them not asked for
    x, w, gate, bias = rand(m, batch * k + pad), (rand(batch, rows, k).float() * k ** -0.5).bfloat16(), rand(m, batch), torch.randn(batch, n, generator=gen, device="cuda")
    ldy, y_batch = batch * n + 5 * (pad == 0), n
    y = torch.full((m + 1, ldy), 7.0, device="cuda", dtype=torch.bfloat16)
    sizes = dict(rows=m, n=n, cols=k, batch=batch, ldx=batch * k + pad, x_batch=k, ldw=k, w_rows=rows, ldy=ldy, y_batch=y_batch, gate_ld=batch)
    assert ask(**sizes) == way
    product(_lib.DenseArgs(**sizes, act_hi=NONE, f32_from=NONE), x, w, y, gate=gate, bias=bias)
    p, size = sums(x[:, :batch * k].view(m, batch, k).transpose(0, 1), w[:, :n], k)
    g = torch.sigmoid(gate.double())[:, :, None]
    want = (p + bias.double()) * g
    got = y[:m, :batch * n].double().view(m, batch, n)
    # the sums, bias and gate in FP32 (its exponential 2^-21 off), then BF16
    assert ((got - want).abs() <= size * g + (2.0 ** -8 + 2.0 ** -20) * want.abs() + 2.0 ** -22 * bias.double().abs() + 1e-9).all()
    assert (y[m] == 7.0).all() and (y[:, batch * n:] == 7.0).all()


@pytest.mark.parametrize("m,n,k,way", [(37, 330, 264, (64, 0, 1)), (37, 2056, 4104, (64, 0, 2)), (37, 1030, 2056, (64, 0, 4)), (37, 260, 2056, (64, 0, 8)),
                                       (390, 3000, 264, (128, 0, 1)), (390, 3000, 4104, (128, 1, 1)), (1000, 4100, 264, (256, 0, 1)),
                                       (700, 4100, 4104, (256, 1, 1))])
@pytest.mark.parametrize("pad", [0, 3])
def test_ranges_and_second_output(m, n, k, way, pad):
    """Features of the activation from 64 on to a border, the last ones to an FP32 output of their own."""
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(m, k, generator=gen, device="cuda").bfloat16()
    w, bias = (torch.randn(n, k, generator=gen, device="cuda") * k ** -0.5).bfloat16(), torch.randn(n, generator=gen, device="cuda")
    hi, second = n // 128 * 64, n // 64 * 64 - 64
    y, y2 = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16), torch.full((m + 1, n - second + pad), 7.0, device="cuda")
    sizes = dict(rows=m, n=n, cols=k, batch=1, ldx=k, ldw=k, w_rows=n, ldy=n, ldy2=n - second + pad, act=2, act_lo=64, act_hi=hi, f32_from=second)
    assert ask(**sizes) == way
    product(_lib.DenseArgs(**sizes), x, w, y, bias=bias, y2=y2)
    p, size = (t[:, 0] for t in sums(x[None], w[None], k))
    z = p + bias.double()
    want = torch.where((torch.arange(n, device="cuda") >= 64) & (torch.arange(n, device="cuda") < hi), z * torch.sigmoid(z), z)
    # SiLU's slope is at most 1.1; its FP32 steps; BF16 of the first output, FP32 of the second
    bound = 1.1 * size + 2.0 ** -20 * (want.abs() + bias.double().abs()) + 1e-9
    assert ((y[:m, :second].double() - want[:, :second]).abs() <= bound[:, :second] + 2.0 ** -8 * want[:, :second].abs()).all()
    assert ((y2[:m, :n - second].double() - want[:, second:]).abs() <= bound[:, second:]).all()
    assert (y[m] == 7.0).all() and (y[:, second:] == 7.0).all() and (y2[m] == 7.0).all() and (y2[:, n - second:] == 7.0).all()
