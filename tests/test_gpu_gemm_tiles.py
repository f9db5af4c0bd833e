"""The tcgen05 prompt GEMM over its free token tiles (csrc/gemm_tcgen05.cu): token counts around every
multiple of 16 and the largest tile, one to many tiles per SM, splits of K over clusters with uneven shares
(and fewer scale groups than stages), ragged features, against 64 bits."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 48, 65, 113, 161, 192, 193, 385, 700])
@pytest.mark.parametrize("n,k", [(1, 128), (127, 384), (130, 2176), (1000, 640), (4112, 1152)])
def test_tiles(m, n, k):
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
