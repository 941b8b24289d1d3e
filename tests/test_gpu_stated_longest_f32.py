"""FP32 products of a CSR that states its longest row: what it may state ends
without an error, what 128 rows show to be too short is reported, and an error
never reaches another call.

Bound of a row's sum as in test_gpu_spmv_any: (len + 32) 2^-24 sum |a||x|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

F32 = torch.float32


def system(lens, seed):
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n = len(lens)
    rng = np.random.default_rng(seed)
    cols = rng.integers(0, n, ro[-1]).astype(np.int32)
    vals, x = rng.normal(size=ro[-1]).astype(np.float32), rng.normal(size=n).astype(np.float32)
    prod = vals.astype(np.float64) * x[cols]
    rows = np.repeat(np.arange(n), lens)
    exact, size = np.zeros(n), np.zeros(n)
    np.add.at(exact, rows, prod)
    np.add.at(size, rows, np.abs(prod))
    dev = [torch.from_numpy(a).cuda() for a in (ro, cols, vals, x)]
    return dev, exact, (np.asarray(lens) + 32) * 2.0**-24 * size


@pytest.mark.parametrize("n", [1, 33, 127, 129, 20011])
@pytest.mark.parametrize("length,stated", [(27, 27), (32, 32), (20, 27), (1, 1)])
def test_right_length(n, length, stated):
    (ro, cols, vals, x), exact, bound = system(np.full(n, length), 1)
    A = M.CSRMatrix(ro, cols, vals, max_row_len=stated)
    ctx = M.Context()
    ctx.bind_torch_stream()
    y = torch.full_like(x, 7.0)
    M.matvec(A, x, y, ctx=ctx)
    ctx.synchronize()
    assert (np.abs(y.cpu().numpy() - exact) <= bound).all()
    d = M.matvec_and_dot(A, x, y, ctx=ctx)
    yx = y.double() * x.double()
    assert abs(d - float(yx.sum())) <= 1e-5 * float(yx.abs().sum())
    # the next solve of the context has nothing to report either
    B, b = M.build_system(6, 5, 7, ctx=ctx)
    s = torch.zeros_like(b)
    r = M.cg_solve(B, b, s, max_iter=200, tol=1e-9, tol_mode="relative", ctx=ctx)
    assert r.status == 0
    ctx.close()


# 128 rows of 27 are 3456 entries, three off a 16-byte boundary at most; with 26
# stated they may take 3336, with 27 3464.  One group of 32 rows of 27 beside
# three of 26 (3360) is more than 26 allow, beside three of 24 (3168) it is not.
@pytest.mark.parametrize("rest,stated,refused", [(27, 26, True), (26, 26, True), (24, 26, False), (27, 4, True)])
def test_stated_too_short(rest, stated, refused):
    i = np.arange(128 * 20)
    (ro, cols, vals, x), exact, bound = system(np.where(i % 128 < 32, 27, rest), 2)
    A = M.CSRMatrix(ro, cols, vals, max_row_len=stated)
    ctx = M.Context()
    ctx.bind_torch_stream()
    y = torch.full_like(x, 7.0)
    M.matvec(A, x, y, ctx=ctx)
    if refused:
        with pytest.raises(M.MiniFEError):
            ctx.synchronize()
    else:
        ctx.synchronize()
        assert (np.abs(y.cpu().numpy() - exact) <= bound).all()
    ctx.close()


def test_box_with_unaligned_x():
    # (the box kernel wants 16-byte alignment; the CSR one takes the product)
    A, b = M.build_system(12, 11, 13)
    A32 = M.to_f32(A)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    off = torch.randn(A.nrows + 1, device="cuda", dtype=F32, generator=g)[1:]
    assert off.data_ptr() % 16
    ctx = M.Context()
    ctx.bind_torch_stream()
    y, ref = torch.empty(A.nrows, device="cuda", dtype=F32), torch.empty_like(b)
    M.matvec(A32, off, y, ctx=ctx)
    ctx.synchronize()
    M.matvec(A, off.double(), ref, ctx=ctx)
    ctx.synchronize()
    # sum |a||x| <= 27 max |a| max |x|; the values themselves are rounded to FP32
    size = 27 * float(A.packed_coefs.abs().max()) * float(off.abs().max())
    assert float((y.double() - ref).abs().max()) <= (27 + 32 + 1) * 2.0**-24 * size
    ctx.close()
