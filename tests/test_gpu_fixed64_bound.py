"""One fixed-point stencil product of the FP64 CG (mfe_fixed64.cuh) row by row, against
the same operator in extended precision.

The kernel by kernel form of the solve (MFE_CG_EAGER=1) runs that product at any size.
From x = 0 the first iteration leaves x1 = a1 b, and the second x2 = x1 + a2 p2 with
p2 = b - a1 A b + beta b, so x1 and x2 hold A b up to the roundings of those steps.

Bound of the product.  A thread's rows share the largest exponent of the three-plane
window that its four positions read.  In units of the last place of the sum V:
entries floored 1/4; weights rounded 27 / 2 / 16 = 0.85; four dropped low products of
at most 1/4 in each of three plane parts 3; their rounding 3 / 2; exponents aligned
between planes 2: 7.6 units, each at most 2^-56 of sum |w| times the window's largest
entry, so 2^-53 of it; and one rounding of the result.
The steps beside it: a1 from x1 (2 roundings), r, p2, x2 one each, beta and a2 (a
projection) a few: 8 roundings of every term cover them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

LD = np.longdouble
# planes within a tile and over several (of 1024 and 2048 positions), lines of the
# lengths where the window changes its form, few planes and many
BOXES = [(4, 4, 4), (31, 31, 6), (40, 24, 7), (63, 31, 5), (254, 6, 5), (510, 5, 6), (511, 5, 5),
         (600, 9, 6), (20, 70, 41)]


def vectors(dims, kind):
    nx, ny, nz = dims
    b = np.random.default_rng(6).standard_normal((nz + 1, ny + 1, nx + 1))
    if kind == "steep in x":
        b *= np.exp2(-2.0 * (np.arange(nx + 1) % 50))
    if kind == "planes apart":  # exponents that differ from plane to plane
        b *= np.exp2(np.array([0, -9, 14, 3, -30, 40])[np.arange(nz + 1) % 6])[:, None, None]
    return b


def apply(w, dd, p):
    """S p in extended precision, and sum |w| over a row's entries."""
    q = np.zeros(p.shape, LD)
    q[1:-1, 1:-1, 1:-1] = p[1:-1, 1:-1, 1:-1]
    y = LD(dd) * p.astype(LD)
    acc = np.zeros(tuple(s - 2 for s in p.shape), LD)
    nz, ny, nx = p.shape
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                c = w[4 * abs(dz) + 2 * abs(dy) + abs(dx)]
                acc += LD(c) * q[1 + dz:nz - 1 + dz, 1 + dy:ny - 1 + dy, 1 + dx:nx - 1 + dx]
    y[1:-1, 1:-1, 1:-1] = acc
    mult = [1, 2, 2, 4, 2, 4, 4, 8]
    return y, sum(m * abs(c) for m, c in zip(mult, w))


def window_max(p):
    """The largest |p~| that the thread of each row reads, in the row's three planes."""
    nz, ny, nx = p.shape
    q = np.zeros_like(p)
    q[1:-1, 1:-1, 1:-1] = np.abs(p[1:-1, 1:-1, 1:-1])
    flat = q.reshape(nz, ny * nx)
    out = np.zeros_like(flat)
    pad = np.zeros((nz, ny * nx + 2 * nx + 12))
    pad[:, nx + 4:nx + 4 + ny * nx] = flat
    # four positions from a multiple of four on: -1 .. 4, and a line before and after.
    # A tile begins at a multiple of four too.
    starts = np.arange(0, ny * nx, 4)
    m = np.zeros((nz, starts.size))
    for line in (-nx, 0, nx):
        for t in range(-1, 5):
            m = np.maximum(m, pad[:, np.minimum(starts + nx + 4 + line + t, pad.shape[1] - 1)])
    m3 = m.copy()
    m3[1:] = np.maximum(m3[1:], m[:-1])
    m3[:-1] = np.maximum(m3[:-1], m[1:])
    for r in range(4):
        at = starts + r
        ok = at < ny * nx
        out[:, at[ok]] = m3[:, ok]
    return out.reshape(p.shape)


@pytest.mark.parametrize("kind", ["normal", "steep in x", "planes apart"])
@pytest.mark.parametrize("dims", BOXES)
def test_product(dims, kind, monkeypatch):
    monkeypatch.setenv("MFE_CG_EAGER", "1")
    A, _ = M.build_system(*dims)
    w, dd = M.Stencil64(A).weights
    b = vectors(dims, kind)
    dev = torch.from_numpy(b.reshape(-1)).cuda()
    xs = []
    for k in (1, 2):
        x = torch.zeros_like(dev)
        r = M.cg_solve(A, dev, x, max_iter=k, tol=1e-9, tol_mode="relative")
        assert r.num_iters == k and r.inner_operator == "stencil64"
        xs.append(x.cpu().numpy().reshape(b.shape).astype(LD))
    x1, x2 = xs
    i = np.unravel_index(np.argmax(np.abs(b)), b.shape)
    a1 = x1[i] / LD(b[i])
    y, sumw = apply(w, dd, b)
    r1 = b - a1 * y
    beta = (r1 * r1).sum() / (b.astype(LD) ** 2).sum()
    p2 = r1 + beta * b
    d = x2 - x1
    a2 = (d * p2).sum() / (p2 * p2).sum()
    err = np.abs(d / a2 - p2)
    steps = np.abs(b) + 2 * np.abs(a1 * y) + 2 * np.abs(r1) + np.abs(beta * b) + np.abs(p2) + np.abs(x2 / a2)
    bound = np.abs(a1) * LD(2.0**-53) * sumw * window_max(b)
    assert (err <= bound + 8 * LD(2.0**-53) * steps).all()
