"""The two passes that a weight gradient's launches take along: clearing the buffer that the GEMM adds to, and adding up the partial
bias sums inside the GEMM."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _compress(g, parts=None, clear=None):
    """MVUE 2:4 compression of g^T (column-major): packed values, metadata in tensor-core order."""
    from sparse import _ext
    k, m = g.shape
    f8 = clear is not None and clear[1]
    packed = torch.empty(m * k // 2, dtype=torch.uint8 if f8 else g.dtype, device=DEV)
    meta = torch.empty(m * k // 16, dtype=torch.int16, device=DEV)
    e_tc = torch.empty(_ext.lib().sp24_meta_tc_bytes(m, k), dtype=torch.uint8, device=DEV)
    x = _ext.PruneExtras()
    x.e_tc, x.row_parts = e_tc.data_ptr(), _ext.ptr(parts)
    if f8:
        x.packed_row_major, x.out_scale = 1, 1.0
    dt, out = _ext.dt(g.dtype), _ext.dt(torch.float8_e4m3fn if f8 else g.dtype)
    if clear is None:
        rc = _ext.lib().sp24_prune_compress_with(g.data_ptr(), dt, m, k, m, 1, packed.data_ptr(), out, m, meta.data_ptr(), _ext.PRUNE_MVUE_FAST,
                                                 None, 0, None, 0, 5, 0, x, _ext.stream())
    else:
        rc = _ext.lib().sp24_mvue_compress_clearing(g.data_ptr(), dt, m, k, m, packed.data_ptr(), out, k // 2 if f8 else m, meta.data_ptr(), 5, 0, x,
                                                    clear[0].data_ptr(), clear[0].numel() * 4, _ext.stream())
    assert rc == 0
    return packed, e_tc


@pytest.mark.parametrize("f8", [False, True])
@pytest.mark.parametrize("pieces", [1, 255, 4097, 1 << 20])
def test_compression_clears_exactly_the_buffer(pieces, f8):
    g = torch.randn(256, 128, device=DEV).half()
    room = torch.ones(pieces * 4 + 8, device=DEV)
    _compress(g, clear=(room[4:-4], f8))
    assert bool((room[4:-4] == 0).all()) and bool((room[:4] == 1).all()) and bool((room[-4:] == 1).all())


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (384, 512, 1152), (1024, 256, 1088), (2304, 264, 2048), (128, 512, 1152), (384, 128, 1088)])
def test_gemm_adds_up_the_row_sums(m, n, k, accumulate):
    """The same bits as the launch of its own (one fixed order), for sizes that the pair kernel takes and two that it does not (a single row
    block, few columns)."""
    from sparse import _ext
    from sparse.spmm import check_status
    lib = _ext.lib()
    gen = torch.Generator(device=DEV).manual_seed(m + k)
    g = torch.randn(k, m, device=DEV, generator=gen).half()
    x = torch.randn(k, n, device=DEV, generator=gen).half()
    n_parts = lib.sp24_row_parts(k, _ext.dt(g.dtype))
    parts = torch.empty(n_parts, m, device=DEV)
    packed, e_tc = _compress(g, parts)
    start = torch.randn(m, device=DEV, generator=gen)
    want, got = start.clone(), start.clone()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    d0, d1 = torch.zeros(m, n, device=DEV), torch.zeros(m, n, device=DEV)
    a = (packed.data_ptr(), _ext.dt(g.dtype), 1, m, e_tc.data_ptr(), m, k, x.data_ptr(), n, n)
    assert lib.sp24_sum_parts(parts.data_ptr(), n_parts, m, want.data_ptr(), accumulate, _ext.stream()) == 0
    assert lib.sp24_spmm_accumulate_f32(*a, d0.data_ptr(), n, 1, status.data_ptr(), _ext.stream()) == 0
    assert lib.sp24_spmm_accumulate_sums_f32(*a, d1.data_ptr(), n, 1, parts.data_ptr(), n_parts, got.data_ptr(), accumulate, status.data_ptr(),
                                             _ext.stream()) == 0
    assert int(status) == 0
    check_status()
    assert torch.equal(got, want) and torch.equal(d0, d1)
    ref = g.double().sum(0) + (start.double() if accumulate else 0)
    assert bool(((got.double() - ref).abs() <= (k + 2) * 2.0 ** -24 * (g.double().abs().sum(0) + start.double().abs())).all())
