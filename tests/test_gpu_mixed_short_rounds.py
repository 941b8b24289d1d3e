"""Mixed solves whose reliable updates come every few iterations: the resident loop
gives way to the graph, so that such a solve takes no longer than one that runs as a
graph from the start (the launch refused, mfe_inject_loop_fault), and both end within
the tolerance: ||b - A x|| <= tol ||b||, the check's own product rounding by at most
28 2^-53 of the row sums |A||x|."""
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


def system(dims):
    A, b0 = M.build_system(*dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    return A, torch.randn(b0.shape, dtype=b0.dtype, device="cuda", generator=g)


@pytest.mark.parametrize("kw", [dict(refine_k=1), dict(refine_k=2), dict(refine_k=3), dict(refine_k=4),
                                dict(inner_tol=0.9)])
@pytest.mark.parametrize("dims", [(9, 8, 7), (24, 24, 24), (64, 64, 64)])
def test_solution(dims, kw):
    A, b = system(dims)
    x = torch.zeros_like(b)
    r = M.cg_solve(A, b, x, max_iter=2000, tol=1e-11, tol_mode="relative", precision="mixed", **kw)
    assert r.status == 0 and r.refinements >= (r.num_iters // kw["refine_k"] if "refine_k" in kw else 2)
    y = torch.empty_like(b)
    M.matvec(A, x, y)
    rnd = 28 * 2.0**-53 * 27 * float(A.packed_coefs.abs().max()) * float(x.norm())
    assert float((b - y).norm()) <= 1e-11 * float(b.norm()) + 2 * rnd


def test_time():
    A, b = system((24, 24, 24))

    def ms(refuse):
        times = []
        for i in range(9):
            x = torch.zeros_like(b)
            if refuse:
                M.inject_loop_fault(0)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            M.cg_solve(A, b, x, max_iter=2000, tol=1e-11, tol_mode="relative", precision="mixed", refine_k=1)
            times.append(time.perf_counter() - t0)
        return 1e3 * min(times[2:])

    assert ms(False) <= 1.2 * ms(True)
