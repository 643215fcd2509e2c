"""Layer-norm backward at every width's number of warps (16; 12 at d = 1024; the widths beside that line) and row counts around a block's."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("extras", [False, True])
@pytest.mark.parametrize("rows", [1, 13, 17, 2369])
@pytest.mark.parametrize("d", [128, 768, 896, 1024])
def test_against_float64(d, rows, extras, dtype):
    from sparse import _ext
    g = torch.Generator(device=DEV).manual_seed(d + rows)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x, dy, dres, gamma = rnd(rows, d), rnd(rows, d).to(dtype), rnd(rows, d), rnd(d)
    mean = x.mean(1)
    rstd = (x.var(1, correction=0) + 1e-5).rsqrt()
    dx, dd, dg, db = torch.empty_like(x), torch.empty_like(dy), torch.zeros(d, device=DEV), torch.zeros(d, device=DEV)
    p = lambda t: t.data_ptr()  # noqa: E731
    lib, tail = _ext.lib(), (p(dg), p(db), rows, d, _ext.stream())
    if extras:
        rc = lib.sp24_add_layernorm_bwd(p(dy), _ext.dt(dtype), p(dres), p(x), p(gamma), p(mean), p(rstd), p(dx), p(dd), *tail)
    else:
        rc = lib.sp24_layernorm_bwd(p(dy), _ext.dt(dtype), p(x), p(gamma), p(mean), p(rstd), p(dx), *tail)
    assert rc == 0
    y, gd, rs = dy.double(), gamma.double(), rstd.double()[:, None]
    xh = (x.double() - mean.double()[:, None]) * rs
    gy = y * gd
    want = rs * (gy - gy.mean(1, keepdim=True) - xh * (gy * xh).mean(1, keepdim=True)) + (dres.double() if extras else 0)
    # A value takes a dozen roundings and two sums of d terms (32 lanes of d / 32), each term at most the row's largest.
    big = rs * gy.abs().amax(1, keepdim=True) * (1 + xh.abs().amax(1, keepdim=True)) ** 2 + dres.double().abs()
    assert bool(((dx.double() - want).abs() <= (d / 32 + 20) * 2.0 ** -24 * big).all())
    if extras:
        assert torch.equal(dd, dx.to(dtype))
    # Sums of `rows` terms of three roundings each.
    for got, terms in ((dg, y * xh), (db, y)):
        mag = (y.abs() * (xh.abs() + 1)).sum(0)
        assert bool(((got.double() - terms.sum(0)).abs() <= (rows + 4) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,d", [(1, 128), (9, 768), (2369, 896), (1003, 1024)])
def test_the_residual_stream_may_be_written_in_place(rows, d, dtype):
    """res_out = x gives the bits of a separate buffer; the sum is float32's own, and the output that of the plain norm of it."""
    from sparse import _ext
    g = torch.Generator(device=DEV).manual_seed(rows + d)
    x, delta = torch.randn(rows, d, device=DEV, generator=g), torch.randn(rows, d, device=DEV, generator=g).to(dtype)
    gamma, beta = torch.randn(d, device=DEV, generator=g), torch.randn(d, device=DEV, generator=g)
    p, lib, got = lambda t: t.data_ptr(), _ext.lib(), []  # noqa: E731
    want = x + delta.float()
    for inp, branch, res in ((x, delta, torch.empty_like(x)), (x, delta, x), (want, None, None)):
        out, mean, rstd = torch.empty(rows, d, device=DEV, dtype=dtype), torch.empty(rows, device=DEV), torch.empty(rows, device=DEV)
        tail = (p(gamma), p(beta), p(out), _ext.dt(dtype), p(mean), p(rstd), rows, d, 1e-5, _ext.stream())
        rc = lib.sp24_add_layernorm_fwd(p(inp), p(branch), p(res), *tail) if res is not None else lib.sp24_layernorm_fwd(p(inp), *tail)
        assert rc == 0 and (res is None or torch.equal(res, want))
        got.append((out, mean, rstd))
    assert all(torch.equal(a, b) for run in got[1:] for a, b in zip(run, got[0]))
