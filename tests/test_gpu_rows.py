"""Products of a few rows (csrc/gemm_rows.cu) through ternary_gemm_packed and, for matrices packed back to
back, through the decoder: edges of the 16-row blocks, the 64-feature tiles, the groups and their
split over clusters, against the oracle in 64 bits."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4, 5, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("n,k", [(1, 128), (15, 384), (64, 512), (65, 1152), (333, 2048), (130, 4352), (20000, 256)])
def test_rows(m, n, k):
    nz, sg, sc, x = oracle.make_case(n, k, seed=m * 1000 + n + k, batch=m)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (nz, sg, sc, x)]
    w = tl.PreparedWeight(*dev[:3], n, k, register=False)
    y = torch.full((m + 1, n), 7.0, dtype=torch.float16, device="cuda")     # one row more than is asked for
    tl.ternary_gemm_packed(dev[3], w, y, m)
    tl.check_device_errors()
    got = y.cpu().numpy().astype(np.float64)
    assert (got[m] == 7.0).all()
    y64 = oracle.ternary_matvec(nz, sg, sc, x, 128, np.float64)
    # products are exact; K sums in FP32, each rounded once: K * 2^-24 of the sum of magnitudes, then FP16
    bound = k * 2.0 ** -24 * oracle.tolerance_bound(nz, sg, sc, x) / 2e-3 + 2.0 ** -11 * np.abs(y64) + 2.0 ** -25
    assert (np.abs(got[:m] - y64) <= bound).all(), np.max(np.abs(got[:m] - y64) / bound)
