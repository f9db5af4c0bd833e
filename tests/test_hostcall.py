"""The native calls of the operators on prepared weights (csrc/hostcall.c): what they take gives what the C ABI gives, on
the stream that is current; what they refuse ends in the checks written in Python, with their words."""
import pytest
import torch

import ternary_llm_b200 as tl
from ternary_llm_b200 import _lib


class Weight:
    def __init__(self, packed, rows, cols):
        self.packed, self.rows, self.cols = packed, rows, cols


def test_refusals_without_a_gpu():
    t = torch.zeros(512, dtype=torch.float16)
    w = Weight(t, 4, 128)
    host = _lib.host()
    for call in (lambda: tl.ternary_gemv_packed(w, t, t), lambda: tl.ternary_gemm_packed(t, w, t, 3), lambda: tl.ternary_gemv_int8_packed(w, t, 1.0, t)):
        with pytest.raises(ValueError, match="must be a CUDA tensor"):
            call()
    with pytest.raises(ValueError, match="positive multiple of 128"):
        tl.ternary_gemv_packed(Weight(t, 4, 130), t, t)
    with pytest.raises(ValueError, match="positive multiple of 128"):
        tl.ternary_gemm_packed(t, Weight(t, 0, 128), t, 3)
    # nothing but plain numbers and tensors is taken, and no exception is left behind
    for bad in (None, 1.5, "x", True, 2 ** 40, -1, 0):
        assert host.gemv_packed(t, bad, 128, t, t, 1) is None
        assert host.gemm_packed(t, t, 4, 128, t, bad) is None
    for bad in (None, 3, object(), [1]):
        assert host.gemv_packed(bad, 4, 128, t, t, 1) is None
    assert host.gemv_packed() is None and host.gemv_int8_packed(t, 4, 128, t, 1, t) is None


@pytest.fixture
def prepared():
    masks = torch.randint(-2 ** 31, 2 ** 31, (2, 100, 12), device="cuda").to(torch.int32)
    scales = torch.rand(100, 3, device="cuda").half()
    return tl.PreparedWeight(masks[0], masks[0] & masks[1], scales, 100, 384, register=False)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 3, 40])
def test_as_the_c_abi(rows, prepared):
    w, lib, side = prepared, _lib.lib(), torch.cuda.Stream()
    x = torch.randn(rows, 384, device="cuda").half()
    q = torch.randint(-127, 128, (384,), device="cuda").to(torch.int8)
    got, want = (torch.full((3, rows + 1, 100), 7.0, device="cuda", dtype=torch.float16) for _ in range(2))
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        if rows <= 16:
            tl.ternary_gemv_packed(w, x, got[0], batch=rows)
        tl.ternary_gemm_packed(x, w, got[1], rows)
        tl.ternary_gemv_int8_packed(w, q, 0.03, got[2])
    p, s = w.packed.data_ptr(), side.cuda_stream
    if rows <= 16:
        assert lib.tllm_b200_gemv_packed(p, x.data_ptr(), want[0].data_ptr(), rows, 100, 384, s) == 0
    assert lib.tllm_b200_gemm_packed(x.data_ptr(), p, want[1].data_ptr(), rows, 100, 384, s) == 0
    assert lib.tllm_b200_gemv_int8_packed(p, q.data_ptr(), 0.03, want[2].data_ptr(), 100, 384, s) == 0
    side.synchronize()
    assert torch.equal(got, want) and (got[:2, rows:] == 7.0).all()


@pytest.mark.gpu
def test_refusals(prepared):
    w = prepared
    x, y = torch.randn(2, 384, device="cuda").half(), torch.zeros(2, 100, device="cuda").half()
    with pytest.raises(TypeError, match="input must be"):
        tl.ternary_gemv_packed(w, x.float(), y)
    with pytest.raises(ValueError, match="holds 384 elements, the call needs 768"):
        tl.ternary_gemv_packed(w, x[:1], y, batch=2)
    with pytest.raises(ValueError, match="contiguous"):
        tl.ternary_gemm_packed(torch.randn(384, 2, device="cuda").half().T, w, y, 2)
    with pytest.raises(ValueError, match="output holds"):
        tl.ternary_gemv_int8_packed(w, torch.zeros(384, dtype=torch.int8, device="cuda"), 1.0, y[0, :99].contiguous())
    with pytest.raises(_lib.TllmError, match="batch 17"):
        tl.ternary_gemv_packed(w, torch.zeros(17, 384, device="cuda").half(), torch.zeros(17, 100, device="cuda").half(), batch=17)
    with pytest.raises(_lib.TllmError, match="aligned"):
        tl.ternary_gemv_packed(w, torch.zeros(400, device="cuda").half()[1:385], y)
    tl.ternary_gemv_int8_packed(w, torch.zeros(384, dtype=torch.int8, device="cuda"), 1, y[0])       # a whole number as the scale
    torch.cuda.synchronize()
    assert (y[0] == 0).all()
