"""Column sums that are set: the bits of those added to zeros, whatever the buffer held, for rows and columns off the tiles and a pitch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols,pad", [(1, 8, 0), (7, 72, 8), (513, 64, 0), (4096, 2304, 0)])
def test_set_is_added_to_zeros(rows, cols, pad, dtype):
    from sparse import _ext
    lib, g = _ext.lib(), torch.Generator(device=DEV).manual_seed(rows + cols)
    x = torch.randn(rows, cols + pad, device=DEV, generator=g).to(dtype)
    a, b = torch.zeros(cols, device=DEV), torch.full((cols,), float("nan"), device=DEV)
    for name, out in (("sp24_column_sums", a), ("sp24_column_sums_set", b)):
        assert getattr(lib, name)(x.data_ptr(), _ext.dt(dtype), rows, cols, cols + pad, out.data_ptr(), _ext.stream()) == 0
    assert torch.equal(a, b)
    ref, mag = x[:, :cols].double().sum(0), x[:, :cols].double().abs().sum(0)
    assert bool(((b.double() - ref).abs() <= (rows + 1) * 2.0 ** -24 * mag).all())
