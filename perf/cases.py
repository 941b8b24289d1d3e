"""What this framework is measured on: the calls that programs make through its
Python entry points (minife_gb300), over the sizes, storage forms, data types and
stopping rules that they use, each as one case.

A case is a dict of plain values; "op" says which path it takes:

  blas1     the reference's vector kernels: waxpby, dot and fused_waxpby
  cg        cg_solve on device vectors (FP64 or mixed precision)
  multi     cg_solve_multi: many right-hand sides of one matrix
  batch     Batch.solve: uneven boxes solved together
  assemble  build_system with one conductivity per element
  adjoint   adjoint.grad_l2: gradient of a loss in the conductivities
  matvec    the product y = A x, A a box matrix, any CSR, or ELL
  host      cg_solve_host: matrix and vectors in host memory

The systems are miniFE's: an nx x ny x nz box of Hex8 elements with its six faces
prescribed.  Right-hand sides are N(0, 1), as in the 32-column benchmark (the
batch assembles its own).  The solves stop at tolerances that determine the
solution to about nine digits, so that two correct solvers return the same x.
"""
from __future__ import annotations

import math

import torch

import minife_gb300 as M
from minife_gb300 import adjoint

F64 = torch.float64


def listed():
    return [
        # the smallest calls: a 30^3 box's vectors (the reference's CPU-sized
        # case), where launch and read-back latency is all there is
        {"name": "blas1 30^3", "op": "blas1", "n": 29791},
        # the reference's own run at that size: its default stop (absolute
        # DBL_EPSILON), which keeps the CSR values
        {"name": "cg 30^3 default stop", "op": "cg", "nx": 30, "ny": 30, "nz": 30,
         "precision": "f64", "tol": M.DBL_EPSILON, "mode": "absolute"},
        # an ordinary FP64 solve on an odd, uneven box to a relative residual
        {"name": "cg 97x64x83", "op": "cg", "nx": 97, "ny": 64, "nz": 83,
         "precision": "f64", "tol": 2e-11, "mode": "relative"},
        # the benchmark's system, FP64, solved to the end
        {"name": "cg 256^3", "op": "cg", "nx": 256, "ny": 256, "nz": 256,
         "precision": "f64", "tol": 2e-11, "mode": "relative"},
        # mixed precision to near-FP64 accuracy on a box that is no cube
        {"name": "cg mixed 160x192x144", "op": "cg", "nx": 160, "ny": 192, "nz": 144,
         "precision": "mixed", "tol": 1e-12, "mode": "relative"},
        # load cases of one structure: 32 right-hand sides together
        {"name": "multi 64^3 x 32", "op": "multi", "nx": 64, "ny": 64, "nz": 64, "nrhs": 32,
         "tol": 1e-12},
        # a parameter study: uneven boxes together
        {"name": "batch 24 boxes 16..96", "op": "batch", "boxes": 24, "lo": 16, "hi": 96,
         "shapes": 20261204, "tol": 1e-13},
        # one assembly of an inverse problem: a new conductivity field each time
        {"name": "assemble 160x128x144", "op": "assemble", "nx": 160, "ny": 128, "nz": 144},
        # one gradient of an inverse problem: assembly, forward and adjoint
        # solve, element contraction
        {"name": "adjoint 48x40x56", "op": "adjoint", "nx": 48, "ny": 40, "nz": 56, "tol": 1e-13},
        # the product alone, as a program with its own Krylov method calls it
        {"name": "matvec box 160^3 f64", "op": "matvec", "nx": 160, "ny": 160, "nz": 160,
         "storage": "box", "dtype": "f64"},
        # the product with a CSR that is no box: rows of 4 to 27 entries
        # around the diagonal, as a mesh with hanging or mixed elements gives
        {"name": "matvec csr 1.5M f64", "op": "matvec", "nx": 113, "ny": 113, "nz": 113,
         "storage": "csr", "dtype": "f64"},
        # the drop-in call of a host program: CSR and vectors in pinned host
        # memory, x copied back
        {"name": "host 80x72x96", "op": "host", "nx": 80, "ny": 72, "nz": 96, "tol": 2e-11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return {d: max(lo, min(hi, int(round(n * rng.uniform(0.7, 1.4))))) for d in ("nx", "ny", "nz")}


def draw(rng):
    op = rng.choice(["blas1", "cg", "cg", "cg", "multi", "batch", "assemble", "adjoint",
                     "matvec", "matvec", "host"])
    if op == "blas1":
        return {"op": op, "n": _log_int(rng, 1000, 8_000_000)}
    if op == "cg":
        kind = rng.choice(["default", "f64", "mixed"])
        if kind == "default":
            return {"op": op, **_box(rng, 12, 80), "precision": "f64", "tol": M.DBL_EPSILON,
                    "mode": "absolute"}
        if kind == "f64":
            return {"op": op, **_box(rng, 20, 220), "precision": "f64", "tol": 2e-11,
                    "mode": "relative"}
        return {"op": op, **_box(rng, 24, 220), "precision": "mixed", "tol": 1e-12,
                "mode": "relative"}
    if op == "multi":
        return {"op": op, **_box(rng, 24, 96), "nrhs": rng.choice([4, 8, 32]), "tol": 1e-12}
    if op == "batch":
        return {"op": op, "boxes": rng.randint(4, 32), "lo": 16, "hi": rng.randint(40, 96),
                "shapes": rng.randint(1, 10**6), "tol": 1e-13}
    if op == "assemble":
        return {"op": op, **_box(rng, 16, 180)}
    if op == "adjoint":
        return {"op": op, **_box(rng, 16, 64), "tol": 1e-13}
    if op == "matvec":
        return {"op": op, **_box(rng, 20, 180), "storage": rng.choice(["box", "csr", "ell"]),
                "dtype": rng.choice(["f64", "f64", "f32"])}
    return {"op": op, **_box(rng, 24, 110), "tol": 2e-11}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _rows(case):
    nx, ny, nz = _dims(case)
    return (nx + 1) * (ny + 1) * (nz + 1)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(n, seed, dtype=F64):
    shape = n if isinstance(n, tuple) else (n,)
    return torch.randn(shape, dtype=F64, device="cuda", generator=_gen(seed)).to(dtype)


def _kappa(case, seed):
    """Log-normal conductivities around 1."""
    nx, ny, nz = _dims(case)
    return torch.exp(0.5 * _normal(nx * ny * nz, seed))


def _ragged_csr(case, seed):
    """(row offsets, columns, values) of rows with 4 to 27 ascending columns taken
    from the 27-point neighbourhood's distances, clamped into the matrix."""
    nx, ny, nz = _dims(case)
    n = _rows(case)
    g = _gen(seed)
    dev = "cuda"
    plane, line = (nx + 1) * (ny + 1), nx + 1
    off = torch.tensor([dz * plane + dy * line + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1)
                        for dx in (-1, 0, 1)], device=dev)
    cols = torch.arange(n, device=dev)[:, None] + off[None, :]
    keep = torch.rand((n, 27), device=dev, generator=g) < torch.rand((n, 1), device=dev,
                                                                     generator=g) * 0.85 + 0.15
    keep[:, 11:15] = True
    keep &= (cols >= 0) & (cols < n)
    ro = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    ro[1:] = torch.cumsum(keep.sum(1), 0)
    cols = cols[keep].to(torch.int32)
    return ro, cols, _normal(cols.numel(), seed + 1)


def _batch_dims(case, seed):
    """The study's boxes (their shapes are the case's), in an order of the seed's."""
    g = torch.Generator()
    g.manual_seed(case["shapes"])
    d = torch.randint(case["lo"], case["hi"] + 1, (case["boxes"], 3), generator=g).tolist()
    g.manual_seed(seed)
    return [tuple(d[i]) for i in torch.randperm(case["boxes"], generator=g).tolist()]


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "blas1":
        s["x"], s["y"] = _normal(case["n"], seed), _normal(case["n"], seed + 1)
        s["w"], s["w2"], s["w3"] = (torch.empty_like(s["x"]) for _ in range(3))
        return s
    if op == "batch":
        s["batch"] = M.Batch(_batch_dims(case, seed))
        return s
    n = _rows(case)
    if op == "assemble":
        s["kappa"] = _kappa(case, seed)
        return s
    if op == "adjoint":
        s["kappa"] = _kappa(case, seed)
        s["target"] = 0.25 * _normal(n, seed + 1)
        return s
    if op == "matvec":
        if case["storage"] == "csr":
            A = M.CSRMatrix(*_ragged_csr(case, seed))
        else:
            A, _ = M.build_system(*_dims(case))
        if case["dtype"] == "f32":
            A = M.to_f32(A)
        s["A"] = M.ELLMatrix.from_csr(A) if case["storage"] == "ell" else A
        s["x"] = _normal(n, seed + 2, torch.float32 if case["dtype"] == "f32" else F64)
        s["y"] = torch.empty_like(s["x"])
        return s
    if op == "host":
        A, _ = M.build_system(*_dims(case))
        s["csr"] = [t.cpu().pin_memory() for t in (A.row_offsets, A.packed_cols, A.packed_coefs)]
        s["b"] = _normal(n, seed).cpu().pin_memory()
        s["x"] = torch.empty_like(s["b"]).pin_memory()
        return s
    s["A"], _ = M.build_system(*_dims(case))
    s["b"] = _normal((n, case["nrhs"]) if op == "multi" else n, seed)
    return s


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "blas1":
        M.waxpby(1.0, s["x"], -0.5, s["y"], s["w"])
        d = M.dot(s["w"], s["x"])
        M.fused_waxpby(1.0, s["x"], 0.25, s["w"], s["w2"], 1.0, s["y"], -0.25, s["w"], s["w3"])
        return {"w": s["w"], "dot": d, "w2": s["w2"], "w3": s["w3"]}
    if op == "cg":
        x = torch.zeros_like(s["b"])
        M.cg_solve(s["A"], s["b"], x, max_iter=5000, tol=case["tol"], tol_mode=case["mode"],
                   precision=case["precision"])
        return x
    if op == "multi":
        x = torch.zeros_like(s["b"])
        M.cg_solve_multi(s["A"], s["b"], x, max_iter=5000, tol=case["tol"], tol_mode="relative")
        return x
    if op == "batch":
        x, _ = s["batch"].solve(max_iter=5000, tol=case["tol"], tol_mode="relative")
        return x
    if op == "assemble":
        A, b = M.build_system(*_dims(case), kappa=s["kappa"])
        return {"values": A.packed_coefs, "b": b}
    if op == "adjoint":
        loss, g, u = adjoint.grad_l2(s["kappa"], _dims(case), s["target"], tol=case["tol"])
        return {"loss": loss, "gradient": g, "u": u}
    if op == "matvec":
        f = M.matvec_ell if case["storage"] == "ell" else M.matvec
        return f(s["A"], s["x"], s["y"])
    s["x"].zero_()
    M.cg_solve_host(*s["csr"], s["b"], s["x"], max_iter=5000, tol=case["tol"],
                    tol_mode="relative")
    return s["x"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _nnz(case):
    nx, ny, nz = _dims(case)
    return (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)


def _iterations(dims, tol):
    """About what CG takes: proportional to the longest side and to the digits."""
    return 0.25 * max(dims) * -math.log10(tol) + 10


def work(case):
    op = case["op"]
    if op == "blas1":
        return {"bytes": 8 * 5 * case["n"], "flops": 11 * case["n"]}
    if op == "batch":
        by = fl = 0.0
        for d in _batch_dims(case, 0):
            c = dict(zip(("nx", "ny", "nz"), d))
            by += 8 * _nnz(c) + 8 * _rows(c)
            fl += _iterations(d, case["tol"]) * (2 * _nnz(c) + 10 * _rows(c))
        return {"bytes": by, "flops": fl}
    n, nnz = _rows(case), _nnz(case)
    ne = case["nx"] * case["ny"] * case["nz"]
    if op == "assemble":
        return {"bytes": 8 * ne + 8 * nnz + 8 * n, "flops": 3500 * ne}
    if op == "adjoint":
        it = 2 * _iterations(_dims(case), case["tol"])
        return {"bytes": 16 * ne + 16 * n, "flops": 4000 * ne + it * (2 * nnz + 10 * n)}
    if op == "matvec":
        v = 4 if case["dtype"] == "f32" else 8
        if case["storage"] == "csr":
            nnz = int(n * 17.5)  # the kept share of 27 columns, on average
        cols = 0 if case["storage"] == "box" else 4
        return {"bytes": (v + cols) * nnz + 2 * v * n, "flops": 2 * nnz}
    k = case.get("nrhs", 1)
    it = _iterations(_dims(case), max(case["tol"], 1e-16))
    return {"bytes": 8 * nnz + 16 * n * k, "flops": it * k * (2 * nnz + 10 * n)}


# ---------------------------------------------------------------------------
# the same in 64 bits, from the mathematics: on a box of equal elements the
# assembled operator is Kx My Mz + Mx Ky Mz + Mx My Kz with the one-dimensional
# stiffness K and mass M of 2-point Gauss quadrature
# ---------------------------------------------------------------------------
_GAUSS = 0.577350269  # the reference's truncated point


def _pair(n):
    """(K, M) as (diagonal, neighbour) along n elements of length 1 / n."""
    h, a2 = 1.0 / n, _GAUSS * _GAUSS
    return (2.0 / h, -1.0 / h), (h / 2 * (1 + a2), h / 2 * (1 - a2) / 2)


def _tri(u, dim, c):
    """c[0] u + c[1] (u's neighbours along dim); u is zero on the faces."""
    y = c[0] * u
    m = u.shape[dim]
    y.narrow(dim, 1, m - 1).add_(u.narrow(dim, 0, m - 1), alpha=c[1])
    y.narrow(dim, 0, m - 1).add_(u.narrow(dim, 1, m - 1), alpha=c[1])
    return y


def _inside(t):
    return t[1:-1, 1:-1, 1:-1]


def _apply(dims, x):
    nx, ny, nz = dims
    (kx, mx), (ky, my), (kz, mz) = _pair(nx), _pair(ny), _pair(nz)
    u = torch.zeros_like(x)
    _inside(u)[:] = _inside(x)
    mxu, kxu = _tri(u, 2, mx), _tri(u, 2, kx)
    w = _tri(_tri(mxu, 1, ky).add_(_tri(kxu, 1, my)), 0, mz).add_(_tri(_tri(mxu, 1, my), 0, kz))
    y = x.clone()
    _inside(y)[:] = _inside(w)
    return y


def _solve(dims, b):
    """The box operator's inverse by diagonalising each direction; b (nz+1, ny+1, nx+1)."""
    vecs, vals = [], []
    for n in dims:
        k, m = _pair(n)
        one = torch.ones(max(n - 2, 0), dtype=F64, device="cuda")
        band = torch.diag(one, 1) + torch.diag(one, -1)
        eye = torch.eye(n - 1, dtype=F64, device="cuda")
        inv = torch.linalg.inv(torch.linalg.cholesky(m[0] * eye + m[1] * band))
        lam, q = torch.linalg.eigh(inv @ (k[0] * eye + k[1] * band) @ inv.T)
        vals.append(lam)
        vecs.append(inv.T @ q)
    t = torch.einsum("zyx,xi,yj,zk->kji", _inside(b), *vecs)
    t = t / (vals[0][None, None, :] + vals[1][None, :, None] + vals[2][:, None, None])
    x = b.clone()
    _inside(x)[:] = torch.einsum("kji,xi,yj,zk->zyx", t, *vecs)
    return x


_CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _element(dims):
    """The 8 x 8 matrix of one element with unit conductivity."""
    nx, ny, nz = dims
    km = []
    for n in dims:
        k, m = _pair(n)
        km.append(((k[0] / 2, k[1]), (m[0] / 2, m[1])))
    e = torch.zeros((8, 8), dtype=F64)
    for i, ci in enumerate(_CORNERS):
        for j, cj in enumerate(_CORNERS):
            d = [abs(p - q) for p, q in zip(ci, cj)]
            for axis in range(3):
                t = 1.0
                for a in range(3):
                    t *= km[a][0 if a == axis else 1][d[a]]
                e[i, j] += t
    return e


def _corner(t, c):
    """The nodes at corner c of every element, as a view of node values t."""
    nz, ny, nx = (v - 1 for v in t.shape)
    return t[c[2]:c[2] + nz, c[1]:c[1] + ny, c[0]:c[0] + nx]


def _faces(dims):
    """(nodes prescribed 0 or 1, nodes prescribed 1, the latter off the other faces)."""
    nx, ny, nz = dims
    shape = (nz + 1, ny + 1, nx + 1)
    bc = torch.ones(shape, dtype=torch.bool, device="cuda")
    _inside(bc)[:] = False
    one = torch.zeros_like(bc)
    one[:, :, -1] = True
    lift = torch.zeros_like(bc)
    lift[1:-1, 1:-1, -1] = True
    return bc, one, lift


def _k_apply(dims, kappa, u):
    e = _element(dims)
    y = torch.zeros_like(u)
    for i, ci in enumerate(_CORNERS):
        s = sum(_corner(u, cj) * float(e[i, j]) for j, cj in enumerate(_CORNERS))
        _corner(y, ci).add_(s.mul_(kappa))
    return y


def _rhs(dims, kappa):
    nx, ny, nz = dims
    bc, one, lift = _faces(dims)
    b = torch.full(bc.shape, 1.0 / (nx * ny * nz), dtype=F64, device="cuda")
    if kappa is None:
        kappa = torch.ones((nz, ny, nx), dtype=F64, device="cuda")
    b -= _k_apply(dims, kappa, lift.to(F64))
    b[bc] = 0.0
    b[one] = 1.0
    return b


def _cg(apply, b):
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), float((r * r).sum())
    stop = 1e-30 * rr
    for _ in range(3000):
        if rr <= stop:
            break
        q = apply(p)
        a = rr / float((p * q).sum())
        x += a * p
        r -= a * q
        rr, old = float((r * r).sum()), rr
        p = r + (rr / old) * p
    return x


def _exact_assemble(dims, kappa):
    nx, ny, nz = dims
    e = _element(dims)
    bc, _, _ = _faces(dims)
    vals = torch.zeros((27,) + tuple(bc.shape), dtype=F64, device="cuda")
    for i, ci in enumerate(_CORNERS):
        for j, cj in enumerate(_CORNERS):
            slot = sum((cj[a] - ci[a] + 1) * 3**a for a in range(3))
            _corner(vals[slot], ci).add_(kappa, alpha=float(e[i, j]))
    there = torch.zeros(vals.shape, dtype=torch.bool, device="cuda")
    pad = torch.nn.functional.pad(bc.to(torch.uint8), (1, 1, 1, 1, 1, 1), value=2)
    for s in range(27):
        dx, dy, dz = s % 3, s // 3 % 3, s // 9
        near = pad[dz:dz + nz + 1, dy:dy + ny + 1, dx:dx + nx + 1]
        there[s] = near != 2
        vals[s][(near == 1) | bc] = 0.0
    vals[13][bc] = 1.0
    order = (1, 2, 3, 0)
    return vals.permute(order).reshape(-1)[there.permute(order).reshape(-1)]


def exact(case, seed):
    op = case["op"]
    if op == "blas1":
        x, y = _normal(case["n"], seed), _normal(case["n"], seed + 1)
        w = x - 0.5 * y
        return {"w": w, "dot": float((w * x).sum()), "w2": x + 0.25 * w, "w3": y - 0.25 * w}
    if op == "batch":
        return torch.cat([_solve(d, _rhs(d, None)).reshape(-1) for d in _batch_dims(case, seed)])
    dims = _dims(case)
    shape = (dims[2] + 1, dims[1] + 1, dims[0] + 1)
    n = _rows(case)
    if op in ("assemble", "adjoint"):
        kappa = _kappa(case, seed).view(dims[2], dims[1], dims[0])
        b = _rhs(dims, kappa)
        if op == "assemble":
            return {"values": _exact_assemble(dims, kappa), "b": b.reshape(-1)}
        bc, one, _ = _faces(dims)

        def apply(v):
            return _k_apply(dims, kappa, v).masked_fill_(bc, 0.0)

        u = _cg(apply, b.masked_fill(bc, 0.0)) + one.to(F64)
        off = u - (0.25 * _normal(n, seed + 1)).view(shape)
        lam = _cg(apply, off.masked_fill(bc, 0.0))
        e = _element(dims)
        g = torch.zeros_like(kappa)
        for i, ci in enumerate(_CORNERS):
            for j, cj in enumerate(_CORNERS):
                g.sub_(_corner(lam, ci) * _corner(u, cj), alpha=float(e[i, j]))
        return {"loss": float(0.5 * (off * off).sum()), "gradient": g.reshape(-1),
                "u": u.reshape(-1)}
    if op == "matvec":
        x = _normal(n, seed + 2, torch.float32 if case["dtype"] == "f32" else F64).to(F64)
        if case["storage"] != "csr":
            return _apply(dims, x.view(shape)).reshape(-1)
        ro, cols, vals = _ragged_csr(case, seed)
        if case["dtype"] == "f32":
            vals = vals.to(torch.float32).to(F64)
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (ro[1:] - ro[:-1]).long())
        return torch.zeros(n, dtype=F64, device="cuda").index_add_(0, rows, vals * x[cols.long()])
    if op == "multi":
        b = _normal((n, case["nrhs"]), seed)
        return torch.stack([_solve(dims, b[:, j].reshape(shape)).reshape(-1)
                            for j in range(case["nrhs"])], 1)
    x = _solve(dims, _normal(n, seed).view(shape)).reshape(-1)
    return x.cpu() if op == "host" else x
