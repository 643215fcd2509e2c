"""The fast MVUE compression, two groups at a time with two-lane float32 arithmetic, against the dense-shaped kernel, which works group
by group: the same bits at the edges of its tiles (32-row remainders, word columns that do not fill a tile, fewer and more tiles than
resident blocks), for every type and both storage orders, with infinities and NaN among the values, and its row sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAMES = {torch.float32: "f32", torch.float16: "f16", torch.bfloat16: "bf16"}


def _x(m, k, dtype, col, special=False):
    g = torch.Generator(device=DEV).manual_seed(m * 7 + k)
    x = torch.randn(m, k, device=DEV, generator=g) * 1e-2
    x.mul_(torch.where(torch.rand(m, k, device=DEV, generator=g) < 0.02, 100.0, 1.0))
    x[torch.rand(m, k, device=DEV, generator=g) < 0.05] = 0
    x[torch.rand(m, k, device=DEV, generator=g) < 0.01] *= -0.0
    if special:
        f = x.view(-1)
        f[5::97], f[11::131], f[17::211] = float("inf"), float("-inf"), float("nan")
    x = x.to(dtype)
    return x.t().contiguous().t() if col else x


def _bits(t):
    """Bit patterns, every NaN alike."""
    i = t.contiguous().view(torch.int16)
    return torch.where(t.isnan().contiguous(), torch.full_like(i, 0x7FFF), i)


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("dtype", list(NAMES), ids=NAMES.get)
@pytest.mark.parametrize("m,k", [(32, 64), (96, 192), (64, 128), (160, 1088), (1056, 2624)])
def test_compression_has_the_dense_kernels_bits(m, k, dtype, col, special):
    import sparse
    from sparse import _ext
    from sparse._semi_structured_conversions import prune_compress, sparse_semi_structured_to_dense
    x = _x(m, k, dtype, col, special)
    out = torch.float16 if dtype == torch.float32 else dtype
    packed = torch.empty(k // 2, m, dtype=out, device=DEV).t() if col else torch.empty(m, k // 2, dtype=out, device=DEV)
    meta = torch.empty(m, k // 16, dtype=torch.int16, device=DEV)
    prune_compress(x, packed, meta, mode=_ext.PRUNE_MVUE_FAST, seed=77, offset=3)
    back = sparse_semi_structured_to_dense(packed.contiguous(), meta)
    want = sparse.MVUE24_approx_triton(x, seed=77, offset=3, exact=False).to(out)
    same = _bits(back) == _bits(want)
    # a group with an infinity or NaN may draw one position twice: the packed form then stores a second one, which the dense form drops
    odd = (~x.contiguous().isfinite()).view(m, k // 4, 4).any(-1, keepdim=True).expand(-1, -1, 4).reshape(m, k)
    assert bool((same | (odd & (want == 0) & back.isnan())).all())


@pytest.mark.parametrize("dtype", list(NAMES), ids=NAMES.get)
@pytest.mark.parametrize("m,k", [(1184, 8256), (2080, 4160)])
def test_blocks_of_many_tiles_have_the_dense_kernels_bits(m, k, dtype):
    """19 x 65 and 33 x 33 tiles on two blocks an SM: every stage is refilled after its operands were written over, and both buffers of
    staged metadata are used again; remainders of 32 rows and 64 columns."""
    test_compression_has_the_dense_kernels_bits(m, k, dtype, True, False)


@pytest.mark.parametrize("dtype", list(NAMES), ids=NAMES.get)
@pytest.mark.parametrize("m,k", [(128, 64), (384, 1088), (2176, 2112)])
def test_pitches_metadata_copy_and_sums(m, k, dtype):
    """Row pitches wider than the matrix on either side (16-byte steps), the metadata copy in tensor-core order where K ends inside an
    atom, and row sums added by the same launch: the bits of the plain call, nothing written beside the rows."""
    from sparse import _ext
    lib, out = _ext.lib(), torch.float16 if dtype == torch.float32 else dtype
    x = _x(m, k, dtype, True).t()                        # storage (k, m)
    wide = torch.full((k, m + 24), float("nan"), dtype=dtype, device=DEV)
    wide[:, 8:m + 8] = x
    atoms = lib.sp24_meta_tc_bytes(m, k)

    def call(src, packed, ld, ld_p):
        meta, e_tc = torch.zeros(m * k // 16, dtype=torch.int16, device=DEV), torch.full((atoms,), 0x5A, dtype=torch.uint8, device=DEV)
        sums = torch.full((m,), 3.0, device=DEV)
        _ext.check(lib.sp24_prune_compress_ex(src.data_ptr(), _ext.dt(dtype), m, k, ld, 1, packed.data_ptr(), _ext.dt(out), ld_p, meta.data_ptr(),
                                              _ext.PRUNE_MVUE_FAST, None, 0, None, 0, 7, 2, None, e_tc.data_ptr(), sums.data_ptr(), _ext.stream()),
                   "prune_compress_ex")
        return meta, e_tc, sums

    plain = torch.empty(k // 2, m, dtype=out, device=DEV)
    room = torch.full((k // 2, m + 40), 7.0, dtype=out, device=DEV)
    meta, e_tc, sums = call(x, plain, m, m)
    meta2, e_tc2, sums2 = call(wide[:, 8:], room[:, 16:], m + 24, m + 40)
    assert torch.equal(_bits(room[:, 16:m + 16]), _bits(plain)) and torch.equal(meta, meta2) and torch.equal(e_tc, e_tc2)
    assert bool((room[:, :16] == 7).all()) and bool((room[:, m + 16:] == 7).all())
    want = torch.empty_like(e_tc)
    _ext.check(lib.sp24_meta_to_tc(meta.data_ptr(), 2, m, k, want.data_ptr(), _ext.stream()), "meta_to_tc")
    assert torch.equal(e_tc, want)
    ref, mag = 3.0 + x.double().sum(0), 3.0 + x.double().abs().sum(0)
    for s in (sums, sums2):                              # k float32 additions in whatever order the blocks come
        assert bool(((s.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("m,k", [(32, 64), (96, 192), (1056, 2624)])
def test_row_sums(m, k):
    """The row sums taken along the way: k float32 additions of exact values, against float64."""
    from sparse import _ext
    from sparse._semi_structured_conversions import prune_compress
    x = _x(m, k, torch.bfloat16, True)
    packed, meta = torch.empty(k // 2, m, dtype=torch.bfloat16, device=DEV).t(), torch.empty(m, k // 16, dtype=torch.int16, device=DEV)
    sums = torch.full((m,), 2.0, device=DEV)
    prune_compress(x, packed, meta, mode=_ext.PRUNE_MVUE_FAST, seed=1, row_sums=sums)
    ref, mag = 2.0 + x.double().sum(1), 2.0 + x.double().abs().sum(1)
    assert bool(((sums.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("dtype", list(NAMES), ids=NAMES.get)
@pytest.mark.parametrize("m,k", [(32, 128), (96, 256), (160, 1152)])
def test_float8_compression_rounds_the_dense_kernels_values(m, k, dtype, col):
    """Unscaled e4m3 in either storage order: the dense-shaped kernel's float32 quotients, saturated and rounded once."""
    import sparse
    from sparse import _ext
    from sparse._semi_structured_conversions import prune_compress, sparse_semi_structured_to_dense
    f8 = torch.float8_e4m3fn
    x = _x(m, k, dtype, col)
    packed = torch.empty(k // 2, m, dtype=f8, device=DEV).t() if col else torch.empty(m, k // 2, dtype=f8, device=DEV)
    meta = torch.empty(m, k // 32, dtype=torch.int32, device=DEV)
    prune_compress(x, packed, meta, mode=_ext.PRUNE_MVUE_FAST, seed=9, offset=1)
    back = sparse_semi_structured_to_dense(packed.contiguous(), meta)
    want = sparse.MVUE24_approx_triton(x.float(), seed=9, offset=1, exact=False).clamp(-448, 448).to(f8)
    assert torch.equal(back.contiguous().view(torch.uint8), want.contiguous().view(torch.uint8))
