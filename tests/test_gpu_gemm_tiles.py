"""The tcgen05 prompt GEMM over its free token tiles (csrc/gemm_tcgen05.cu): token counts around
multiples of 16 and the largest tiles, one to many tiles per SM, splits of K over clusters with uneven shares
(and fewer scale groups than stages), ragged features, against 64 bits."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import oracle
from ternary_llm_b200 import layer_ops as ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 48, 65, 113, 161, 192, 193, 385, 700])
@pytest.mark.parametrize("n,k", [(1, 128), (127, 384), (130, 2176), (1000, 640), (4112, 1152)])
def test_tiles(m, n, k):
    product(m, n, k)


@pytest.mark.parametrize("m,n,k", [(1000, 4112, 1152), (2000, 2000, 1152), (2000, 3456, 2304), (1999, 3460, 2304), (201, 3200, 6144), (205, 3070, 6144)])
def test_tiles_of_one_accumulator(m, n, k):
    """Tiles of more than 192 tokens: one and two rounds of them, whole and ragged, and K split over a cluster."""
    product(m, n, k)


def product(m, n, k):
    nz, sg, sc, x = oracle.make_case(n, k, seed=m + n + k, batch=m)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")
    tl.ternary_gemm_packed(dev[3], w, y, m)
    torch.cuda.synchronize()
    tl.check_device_errors()
    assert (y[m] == 7.0).all()
    wd = torch.from_numpy(oracle.unpack_bitmasks(nz, sg).astype(np.float64) * np.repeat(sc.astype(np.float64), 128, axis=1)).cuda()
    xd = dev[3].double()
    want = xd @ wd.T
    # products are exact; K FP32 sums of at most the magnitudes, cut or rounded, then one rounding to FP16
    bound = k * 2.0 ** -23 * (xd.abs() @ wd.abs().T) + 2.0 ** -11 * want.abs() + 2.0 ** -25
    assert ((y[:m].double() - want).abs() <= bound).all()


def test_chain_of_launches():
    """Launches that start before the one in front of them has ended, weights from HBM in the first layer: every product
    is the one of the input it was given (a slot of codes refilled under its readers showed here, not alone)."""
    m, dims = 300, [(2048, 2048), (8192, 2048), (2048, 8192)]
    prepared, dense = [], []
    for i, (n, k) in enumerate(dims):
        nz, sg, sc, _ = oracle.make_case(n, k, seed=i, batch=1)
        prepared.append(tl.PreparedWeight(*[torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc)],
                                          n, k, register=False))
        dense.append(torch.from_numpy(oracle.unpack_bitmasks(nz, sg).astype(np.float32) * np.repeat(sc.astype(np.float32), 128, axis=1)).cuda())
    ones = [torch.ones(n, dtype=torch.float16, device="cuda") for n, _ in dims]
    x0 = torch.randn(m, 2048, device="cuda").half()
    y = [[torch.zeros(m, n, dtype=torch.float16, device="cuda") for n, _ in dims] for _ in range(6)]
    z = [[torch.zeros_like(t) for t in layer] for layer in y]

    def chain():
        x = x0
        for yl, zl in zip(y, z):
            for i, (n, k) in enumerate(dims):
                tl.ternary_gemm_packed(x, prepared[i], yl[i], m)
                ops.rmsnorm_forward(yl[i], ones[i], zl[i], None, None, m, n, 1e-5)
                x = zl[i]

    chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    cold = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    for _ in range(8):
        cold.zero_()                                     # weights out of L2
        graph.replay()
        torch.cuda.synchronize()
        x = x0
        for yl, zl in zip(y, z):
            for i in range(len(dims)):
                want = x.float() @ dense[i].T
                # a wrong code word shows as several per cent of an output; FP16 rounds to 2^-11
                assert ((yl[i].float() - want).abs() <= 2.0 ** -10 * want.abs() + 2.0 ** -9 * want.std()).all()
                x = zl[i]
    tl.check_device_errors()
    del graph
