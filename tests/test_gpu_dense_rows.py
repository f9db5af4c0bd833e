"""The dense GEMV of one vector whose rows are whole groups of its ring (csrc/dense_gemv.cu, dense_row_kernel): edges of
the groups and of the rows a CTA owns, gated pairs, and in models as wide the norms in its staging, its tails and chosen experts."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import femolix_oracle, mixed_oracle
from ternary_llm_b200 import mixed_ops as ops
from tests import _femolix as X
from tests import _mixed as M
from tests.test_gpu_mixed_decoder import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("k", [256, 512, 1024, 1536, 8192])
@pytest.mark.parametrize("n", [1, 7, 296, 297, 5001])
def test_product(n, k, dt):
    """Whole groups are 1024 BF16 or 512 FP32 columns of one row, half of that of two."""
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    x = torch.randn(1, k, generator=gen, device="cuda").to(dt)
    w = (torch.randn(2 * n, k, generator=gen, device="cuda") * k ** -0.5).to(dt)
    y = torch.full((n + 8,), 7.0, device="cuda")
    ops.dense_linear(x, w, y, 1, n, k)
    assert (y[n:] == 7.0).all()
    want, size = w[:n].double() @ x[0].double(), w.double().abs() @ x[0].double().abs()
    # a lane's two chains of K / 64 sums, then six over chains and lanes, each rounded to FP32 (products of FP32 too)
    bound = (k / 64 + 7) * 2.0 ** -24
    assert ((y[:n].double() - want).abs() <= bound * size[:n]).all()
    g = torch.full((n + 8,), 7.0, device="cuda", dtype=dt)
    ops.dense_linear(x, w, g, 1, n, k, act=None, glu=True)
    assert (g[n:] == 7.0).all()
    up = w[n:].double() @ x[0].double()
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -23
    assert ((g[:n].double() - want * up).abs() <= eps * (want * up).abs() + 1.1 * bound * (size[:n] * up.abs() + size[n:] * want.abs()) + 1e-9).all()


LAYERS = {
    "petulix": (M.config([M.mamba(inner=1024, state=16, dt_rank=64, conv=4, ff=1024), M.mamba(inner=512, conv=7), M.rglru(width=1024, blocks=2, conv=4),
                          M.attention(heads=4, dim=64, rot_dim=32, vdim=128, kv_rank=512, ff=512)], width=1024), M, mixed_oracle),
    "femolix": (X.config([X.delta(heads=8, kv_heads=4, dim=64, vdim=64, conv=4, mlp=X.dense(1024)), X.parallel(mlp=X.moe(6, 2, 1024)),
                          X.delta(conv=2, mlp=X.moe(5, 3, 512))], width=1024), X, femolix_oracle),
}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("design", list(LAYERS))
def test_steps_of_wide_models(design, dtype):
    cfg, helper, oracle = LAYERS[design]
    raw, W = helper.random_model(cfg, 11)
    toks = np.random.default_rng(3).integers(0, cfg["vocab"], 28).astype(np.int32)
    want = oracle.forward(cfg, W, toks, [])
    dec = tl.Decoder(helper.model(cfg, raw), dtype=dtype, max_batch=2, max_seq_len=32)
    for cuts in ([1] * 28, [9] + [1] * 19):
        err = helper.row_error(run(dec, toks, cuts, seq=1), want)
        # the limits of tests/test_gpu_mixed_decoder.py and, for a router's close calls in BF16, tests/test_gpu_femolix.py
        if dtype == "float32":
            assert err.max() <= 1e-4, err.max()
        else:
            assert (err > 6e-2).mean() <= 0.08 and np.median(err) <= 3e-2, err
    tl.check_device_errors()
    dec.close()
