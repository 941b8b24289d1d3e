"""Multi-RHS dots on both sides of the number of blocks (160) up to which their
partial sums are one group: products of 32 rows a block, and right-hand sides of 1 to 32
columns.

Every column's first iterations against the same column solved alone.  The sums differ
in their order only: 2^-53 sqrt(n) relative at most, so alpha and beta of two iterations
by a few 1e-15, and x with them (r and p within a factor of ten of b)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


@pytest.mark.parametrize("nrhs", [1, 4, 32])
@pytest.mark.parametrize("dims", [(3, 3, 3), (15, 15, 15), (16, 16, 16), (17, 16, 16), (19, 19, 19), (33, 34, 35)])
def test_two_iterations(dims, nrhs):
    A, b = M.build_system(*dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    B = torch.randn((b.numel(), nrhs), dtype=b.dtype, device="cuda", generator=g)
    kw = dict(max_iter=2, tol=1e-12, tol_mode="relative")
    X = torch.zeros_like(B)
    for _ in range(2):  # (the second call meets the tickets that the first left)
        X.zero_()
        M.cg_solve_multi(A, B, X, precision="f64", **kw)
    for j in range(nrhs):
        x = torch.zeros_like(b)
        M.cg_solve(A, B[:, j].contiguous(), x, f64_operator="csr", **kw)
        assert float((X[:, j] - x).norm()) <= 1e-13 * float(x.norm())
