"""The mixed solver's cooperative loop against the same solve issued kernel by
kernel (MFE_CG_EAGER=1).

Both run CG in FP32 with FP64-accurate dots and refine to the same FP64 residual;
the FP32 products group their sums differently.  The solutions are checked against
what the stop promises: ||b - A x|| <= tol ||b|| for each, so ||A (x - x2)|| <=
2 tol ||b||; the check's own product rounds by at most 28 2^-53 of the row sums
|A| |x|.  The boxes lie on both sides of the lines where the loop changes its
block size (912,000 padded rows on 152 SMs) and gives way to the graph (2,000,000
rows), with shares that end inside a line, paddings of 0 to 3 and blocks of few
rows."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

BOXES = [(4, 4, 4), (5, 4, 6), (6, 9, 4), (7, 30, 5), (33, 32, 31), (200, 6, 5), (5, 6, 300),
         (95, 95, 97), (96, 97, 97), (124, 125, 124), (125, 126, 125)]


@pytest.mark.parametrize("dims", BOXES)
def test_against_eager(dims, monkeypatch):
    A, b0 = M.build_system(*dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = torch.randn(b0.shape, dtype=b0.dtype, device="cuda", generator=g)
    tol = 1e-11
    out = []
    for eager in (False, True):
        if eager:
            monkeypatch.setenv("MFE_CG_EAGER", "1")
        x = torch.zeros_like(b)
        r = M.cg_solve(A, b, x, max_iter=4000, tol=tol, tol_mode="relative", precision="mixed",
                       record_history=True)
        assert r.status == 0 and r.inner_operator == "stencil"
        out.append((r, x))
    (r, x), (r2, x2) = out
    # the recursive residuals agree while FP32 rounding has not separated them
    assert r.history[:2] == pytest.approx(r2.history[:2], rel=1e-5)
    bn = float(b.norm())
    rnd = 28 * 2.0**-53 * 27 * float(A.packed_coefs.abs().max()) * float(x.norm())
    y = torch.empty_like(b)
    for v in (x, x2):
        M.matvec(A, v, y)
        assert float((b - y).norm()) <= tol * bn + 2 * rnd
    M.matvec(A, x - x2, y)
    assert float(y.norm()) <= 2 * tol * bn + 4 * rnd


def test_iteration_limit():
    A, b = M.build_system(20, 20, 20)
    x = torch.zeros_like(b)
    r = M.cg_solve(A, b, x, max_iter=7, tol=1e-12, tol_mode="relative", precision="mixed")
    assert r.num_iters == 7 and r.status == 5
