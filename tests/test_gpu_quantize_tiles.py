"""Quantisation of tiles that are not whole: rows around 32 and 128, columns around 64, a pitch, with and without the transpose; the bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols,pad,transpose", [(1, 8, 0, True), (31, 72, 8, True), (129, 64, 0, False), (160, 136, 16, True), (257, 200, 0, True)])
def test_bytes(rows, cols, pad, transpose, dtype):
    from sparse import _ext
    g = torch.Generator(device=DEV).manual_seed(rows * cols)
    x = torch.randn(rows, cols + pad, device=DEV, generator=g).to(dtype)
    x[0, 0], x[-1, cols - 1] = float("inf"), float("nan")
    amax = torch.full((1,), 448.0, device=DEV)                 # scale 1: the conversion alone
    q = torch.full((rows, cols), 85, device=DEV, dtype=torch.uint8)
    t = torch.full((cols, rows + 3), 85, device=DEV, dtype=torch.uint8)
    rc = _ext.lib().sp24_quantize_f8(x.data_ptr(), _ext.dt(dtype), rows, cols, cols + pad, amax.data_ptr(), q.data_ptr(),
                                     t.data_ptr() if transpose else None, rows + 3, _ext.stream())
    assert rc == 0
    want = x[:, :cols].float().clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)      # saturating; NaN stays NaN
    nan = torch.isnan(x[:, :cols])
    assert torch.equal(q[~nan], want[~nan]) and bool((q[nan] & 0x7F == 0x7F).all())
    assert bool((t[:, rows:] == 85).all())
    assert torch.equal(t[:, :rows], q.t()) if transpose else bool((t == 85).all())
