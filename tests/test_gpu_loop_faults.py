"""The resident solver loops' bounded waits: the blocks of the next loop wait for one
that never arrives, give up after 20 ms, and the solve returns MFE_TIMEOUT from each
form of the loop; the same context then solves as if nothing had been."""
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
