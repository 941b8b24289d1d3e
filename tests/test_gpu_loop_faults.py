"""The resident solver loops where they cannot run.  Bounded waits: the blocks of the
next loop wait for one that never arrives, give up after 20 ms, and the solve returns
MFE_TIMEOUT from each form of the loop; the same context then solves as if nothing had
been.  A refused launch: the solve runs as a graph."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

# CSR values, the stencil in FP64 and in fixed point (tiles of two sizes), mixed
LOOPS = [((9, 8, 7), dict(f64_operator="csr")), ((30, 30, 30), dict(f64_operator="csr")),
         ((30, 30, 30), {}), ((82, 80, 81), {}), ((99, 99, 99), {}), ((520, 30, 40), {}),
         ((24, 24, 24), dict(precision="mixed")), ((100, 97, 99), dict(precision="mixed"))]


@pytest.mark.parametrize("dims,kw", LOOPS)
def test_timeout(dims, kw):
    ctx = M.Context()
    ctx.bind_torch_stream()
    A, b = M.build_system(*dims, ctx=ctx)
    kw = dict(kw, max_iter=3000, tol=1e-9, tol_mode="relative", ctx=ctx)
    x = torch.zeros_like(b)
    r = M.cg_solve(A, b, x, **kw)
    for _ in range(2):
        M.inject_loop_fault(20_000_000, ctx=ctx)
        y = torch.zeros_like(b)
        with pytest.raises(M.MiniFEError) as ei:
            M.cg_solve(A, b, y, **kw)
        assert ei.value.status == 6  # MFE_TIMEOUT
        y = torch.zeros_like(b)
        r2 = M.cg_solve(A, b, y, **kw)
        assert (r2.status, r2.num_iters, r2.normr) == (0, r.num_iters, r.normr)
        assert torch.equal(x, y)
    ctx.close()


@pytest.mark.parametrize("dims,kw", LOOPS)
def test_refused(dims, kw):
    # a device that cannot hold the loop: the solve runs as a graph instead.  Both
    # end within the tolerance: ||A (x - y)|| <= 2 tol ||b|| up to the products'
    # rounding (28 2^-53 of the row sums |A||x| each)
    ctx = M.Context()
    ctx.bind_torch_stream()
    A, b0 = M.build_system(*dims, ctx=ctx)
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    b = torch.randn(b0.shape, dtype=b0.dtype, device="cuda", generator=g)
    kw = dict(kw, max_iter=3000, tol=1e-9, tol_mode="relative", ctx=ctx)
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    r = M.cg_solve(A, b, x, **kw)
    M.inject_loop_fault(0, ctx=ctx)
    r2 = M.cg_solve(A, b, y, **kw)
    assert r.status == r2.status == 0 and r.inner_operator == r2.inner_operator
    d = torch.empty_like(b)
    M.matvec(A, x - y, d, ctx=ctx)
    rnd = 28 * 2.0**-53 * 27 * float(A.packed_coefs.abs().max()) * float(x.norm())
    # (the FP64 loop tests the residual norm that the recurrence carries)
    assert float(d.norm()) <= 2 * 1e-9 * float(b.norm()) * (1 + 1e-6) + 4 * rnd
    assert not torch.equal(x, y)  # (other sums: the graph did run)
    ctx.close()
