"""The FP64 ELL product with one stage per warp (a million rows and more) and, just
below the line, with two: plain, and as the residual that CG starts from.

Bound: a row's K products in two chains rounded K + 2 times, each by at most 2^-53
of sum |a||x|; the FP64 reference (torch, K sequential additions) likewise.  The
residual's norm: rounded to (2 K + 8) 2^-53 of || |b| + |A||x| ||, the sum of
squares with it."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


@pytest.mark.parametrize("n", [999999, 1000000, 1000033])
@pytest.mark.parametrize("K", [1, 7, 32])
def test_rows(n, K):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + K)
    c = torch.randint(0, n, (n, K), device="cuda", generator=g, dtype=torch.int32)
    c[:, 0] = torch.arange(n, device="cuda")
    v = torch.randn((n, K), device="cuda", generator=g, dtype=torch.float64)
    x = torch.randn(n, device="cuda", generator=g, dtype=torch.float64)
    E = M.ELLMatrix(c.ravel(), v.ravel(), K)
    y = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    M.matvec_ell(E, x, y)
    ref, size = torch.zeros_like(x), torch.zeros_like(x)
    for k in range(K):
        t = v[:, k] * x[c[:, k].long()]
        ref += t
        size += t.abs()
    assert bool(((y - ref).abs() <= 2 * (K + 2) * 2.0**-53 * size).all())
    b = torch.randn(n, device="cuda", generator=g, dtype=torch.float64)
    r = M.cg_solve_ell(E, b, x.clone(), max_iter=0, tol=1e-3, tol_mode="relative")
    want = float((b - ref).norm())
    assert abs(r.normr0 - want) <= 2 * (2 * K + 8) * 2.0**-53 * float((b.abs() + size).norm()) + 1e-12 * want
