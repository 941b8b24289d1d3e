"""The FP64 CG's fixed-point stencil product against the CG on the CSR values.

Both run three iterations from x = 0.  The operators differ by at most 2^-39 of
a row's largest entry per entry, so a product by at most 2^-39 sum |a||p|, and
with sum |a||p| / |A p| up to about 8 three products move x by at most
3 * 8 * 2^-39 = 4.4e-11 of its norm; the fixed-point sums themselves add
2^-55.  The boxes put the plane at the edges of the tiles (1024 and 2048
positions), the node lines at the lengths where the launch changes (255 / 256
and 511 / 512), and one plane wider than a tile's window."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

TOL = 4.4e-11
BOXES = [(4, 4, 4), (31, 31, 6), (40, 24, 7), (63, 31, 5), (49, 40, 9), (46, 43, 40), (254, 6, 5),
         (255, 6, 5), (510, 5, 6), (511, 5, 5), (2600, 4, 5), (120, 130, 11)]


def three_iterations(dims, b):
    A, _ = M.build_system(*dims)
    xs = []
    for op in ("auto", "csr"):
        x = torch.zeros_like(b)
        r = M.cg_solve(A, b, x, max_iter=3, tol=1e-9, tol_mode="relative", f64_operator=op)
        assert r.num_iters == 3
        assert r.inner_operator == ("stencil64" if op == "auto" else "none")
        xs.append(x)
    return xs


def normal(dims, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nx, ny, nz = dims
    return torch.randn((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("dims", BOXES)
def test_three_iterations_match_csr(dims):
    b = normal(dims, 3)
    x, ref = three_iterations(dims, b.reshape(-1))
    assert float((x - ref).norm()) <= TOL * float(ref.norm())


@pytest.mark.parametrize("step", [-10, -40])
def test_steep_vectors(step):
    # entries falling by 2^step per node along x, as at the front of the first iterations
    dims = (37, 20, 12)
    b = normal(dims, 4)
    b *= torch.exp2(step * torch.arange(dims[0] + 1, dtype=torch.float64, device="cuda") / 2)
    x, ref = three_iterations(dims, b.reshape(-1))
    assert float((x - ref).norm()) <= TOL * float(ref.norm())


def test_rows_outside_the_fixed_point_range():
    # planes of entries near 2^-1000, far enough from the others that three
    # products do not reach them (a thread's exponent covers three planes): all
    # their rows take the FP64 form
    dims = (14, 12, 40)
    b = normal(dims, 5)
    b[14:22] = 0.0
    b[22:] *= 2.0**-1000
    x, ref = (v.view_as(b)[26:] for v in three_iterations(dims, b.reshape(-1)))
    scale = 2.0**990
    assert float(((x - ref) * scale).norm()) <= TOL * float((ref * scale).norm()) > 0.0
