"""The cooperative CG loop against the same solve issued kernel by kernel
(MFE_CG_EAGER=1).

Both form the same rows and differ in the order of the dots' sums (2^-53 sqrt(n)
relative at most) and, for the stencil operator, in how a product is rounded
(2^-53 of its norm): alpha and beta of the first two iterations differ by about
1e-15, and so does x, the norms of r and p being within a factor of ten of b's.
(Further iterations amplify without a simple bound: the Dirichlet rows are an
eigenspace that CG resolves at once.)  The boxes lie
on both sides of the lines where the loop (on 152 SMs) changes its block size
(91,200 rows with the stencil, 212,800 with the CSR values), no longer holds all
CSR values in shared memory (about 134,000), changes its form of the stencil
product (500,000) and gives way to the graph (1,000,000 rows with the CSR
values, 2,000,000 with the stencil)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

BOXES = [(1, 1, 1), (2, 1, 3), (7, 4, 5), (33, 32, 33), (34, 33, 32), (58, 57, 57), (58, 58, 57),
         (44, 44, 44), (45, 44, 44), (50, 50, 50), (51, 51, 50), (60, 58, 58), (61, 58, 58), (78, 78, 79),
         (79, 79, 79), (99, 99, 98), (99, 99, 99), (600, 12, 20)]


def solve(A, b, x, **kw):
    r = M.cg_solve(A, b, x, record_history=True, **kw)
    return r, x


@pytest.mark.parametrize("operator", ["csr", "auto"])
@pytest.mark.parametrize("dims", BOXES)
def test_two_iterations(dims, operator, monkeypatch):
    A, b0 = M.build_system(*dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    b = torch.randn(b0.shape, dtype=b0.dtype, device="cuda", generator=g)
    kw = dict(max_iter=2, tol=1e-9, tol_mode="relative", f64_operator=operator)
    off = torch.zeros(b.numel() + 1, dtype=b.dtype, device="cuda")[1:]  # not 16-byte aligned
    r, x = solve(A, b, torch.zeros_like(b), **kw)
    r1, x1 = solve(A, b, off, **kw)
    monkeypatch.setenv("MFE_CG_EAGER", "1")
    r2, x2 = solve(A, b, torch.zeros_like(b), **kw)
    assert r.num_iters == r1.num_iters == r2.num_iters and r.inner_operator == r2.inner_operator
    for v in (x, x1):  # (an unaligned x takes another kernel for the first residual)
        assert float((v - x2).norm()) <= 1e-13 * float(x2.norm())
    assert r.history == pytest.approx(r2.history, rel=1e-12)


@pytest.mark.parametrize("dims", [(10, 10, 10), (30, 30, 30), (24, 61, 40)])
def test_absolute_stop(dims, monkeypatch):
    # p.Ap falls far below the breakdown pre-test's first threshold
    A, b = M.build_system(*dims)
    kw = dict(max_iter=1000, tol=M.DBL_EPSILON, tol_mode="absolute")
    r, x = solve(A, b, torch.zeros_like(b), **kw)
    monkeypatch.setenv("MFE_CG_EAGER", "1")
    r2, x2 = solve(A, b, torch.zeros_like(b), **kw)
    assert r.status == r2.status == 0
    assert abs(r.num_iters - r2.num_iters) <= 2
    assert float((x - x2).norm()) <= 1e-12 * float(x2.norm())
