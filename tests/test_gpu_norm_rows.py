"""Residual chain of many rows (csrc/mixers.cu): widths at the edges of a thread's pieces, and row counts either side of the line, through
models of one layer against the oracle; 32-bit mode, so that a row's sums decide."""
import numpy as np
import pytest
import torch

import ternary_llm_b200 as tl
from oracle import mixed_oracle as O
from tests import _mixed as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 510, 512, 513, 1024, 1030, 2049, 4096, 4100])
def test_chain_widths_and_rows(width):
    cfg = M.config([M.rglru(width=16, blocks=2, conv=2, ff=8)], width=width, vocab=40)
    raw, W = M.random_model(cfg, width)
    toks = np.random.default_rng(width).integers(0, 40, 150).astype(np.int32)
    want = O.forward(cfg, W, toks)
    dec = tl.Decoder(M.model(cfg, raw), dtype="float32", max_seq_len=150)
    for n in (147, 148, 150):
        got = dec.forward_logits(0, torch.from_numpy(toks[:n]).cuda(), 0, list(range(n))).cpu().numpy()
        err = M.row_error(got, want[:n])
        assert err.max() <= 1e-4, f"{n} rows: {err.max():.2e}"
    tl.check_device_errors()
    dec.close()
