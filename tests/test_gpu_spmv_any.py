"""Products with CSR rows of any lengths (k_spmv_any): rows in pairs and alone,
empty rows, groups of 32 rows larger than the stage, long rows among short ones,
the last partial group, and the dot's epilogue.

Bound: each row is at most its length in FMAs plus the additions that join its
partial sums (32 at most), every rounding at most 2^-53 of the sum of |a||x| so far:
(len + 32) 2^-53 sum |a||x| against the same sum in extended precision (whose
own rounding is 2^-11 of that).  FP32 rows the same with 2^-24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

SHAPES = {
    "ragged": lambda r, n: r.integers(4, 28, n),
    # pairs of rows: 18 entries a lane, 19 (no pairs), the longest that pairs take
    "0 and 36": lambda r, n: np.arange(n) % 2 * 36,
    "0 and 37": lambda r, n: np.arange(n) % 2 * 37,
    "one of 54 in 4": lambda r, n: np.where(np.arange(n) % 4 == 1, 54, 2),
    "even": lambda r, n: np.full(n, 27),
    "short": lambda r, n: r.integers(0, 3, n),
    "one long row per group": lambda r, n: np.where(np.arange(n) % 32 == 17, 200, 1),
    "longer than the stage": lambda r, n: np.where(np.arange(n) == n // 2, 3000, 3),
    "empty ends": lambda r, n: np.where((np.arange(n) % 32 < 5) | (np.arange(n) % 32 > 28), 0, 9),
    "all empty but one": lambda r, n: np.where(np.arange(n) == n - 1, 5, 0),
}


@pytest.mark.parametrize("n", [1, 31, 33, 20011])
@pytest.mark.parametrize("shape", SHAPES)
def test_uneven_rows(shape, n):
    rng = np.random.default_rng(3)
    lens = SHAPES[shape](rng, n).astype(np.int64)
    ncol = max(n, 3001)
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = rng.integers(0, ncol, ro[-1]).astype(np.int32)
    vals, x = rng.normal(size=ro[-1]), rng.normal(size=ncol)
    dev = [torch.from_numpy(a).cuda() for a in (ro, np.append(cols, [0] * 4).astype(np.int32),
                                                np.append(vals, [0.0] * 4), x)]
    A = M.CSRMatrix(dev[0], dev[1][:ro[-1]], dev[2][:ro[-1]], num_cols=ncol)
    y = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    M.matvec(A, dev[3], y)
    prod = vals.astype(np.longdouble) * x[cols].astype(np.longdouble)
    rows = np.repeat(np.arange(n), lens)
    exact = np.zeros(n, dtype=np.longdouble)
    size = np.zeros(n, dtype=np.longdouble)
    np.add.at(exact, rows, prod)
    np.add.at(size, rows, np.abs(prod))
    err = np.abs(y.cpu().numpy().astype(np.longdouble) - exact)
    assert (err <= (lens + 32) * 2.0**-53 * size).all()
    if n == ncol:
        d = M.matvec_and_dot(A, dev[3], y)
        yy = y.cpu().numpy()
        assert abs(d - float(np.dot(yy.astype(np.longdouble), x))) <= (n + 64) * 2.0**-53 * float(np.abs(yy * x).sum())


@pytest.mark.parametrize("n", [33, 20011])
@pytest.mark.parametrize("shape", SHAPES)
def test_uneven_rows_f32(shape, n):
    rng = np.random.default_rng(4)
    lens = SHAPES[shape](rng, n).astype(np.int64)
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = rng.integers(0, n, ro[-1]).astype(np.int32)
    vals, x = (rng.normal(size=k).astype(np.float32) for k in (ro[-1], n))
    dev = [torch.from_numpy(a).cuda() for a in (ro, np.append(cols, [0] * 4).astype(np.int32),
                                                np.append(vals, np.zeros(4, np.float32)), x)]
    A = M.CSRMatrix(dev[0], dev[1][:ro[-1]], dev[2][:ro[-1]])
    y = torch.full((n,), 7.0, dtype=torch.float32, device="cuda")
    M.matvec(A, dev[3], y)
    prod = vals.astype(np.float64) * x[cols].astype(np.float64)
    rows = np.repeat(np.arange(n), lens)
    exact, size = np.zeros(n), np.zeros(n)
    np.add.at(exact, rows, prod)
    np.add.at(size, rows, np.abs(prod))
    assert (np.abs(y.cpu().numpy() - exact) <= (lens + 32) * 2.0**-24 * size).all()


@pytest.mark.parametrize("stated,refused", [(27, False), (26, False), (25, True), (4, True)])
def test_stated_longest_row(stated, refused):
    # one row of 27 per group of 32, the others of 25 (26 where 25 is stated): 802
    # or 833 entries a group, where 32 rows of the stated length may take 872, 840,
    # 808 and 136 with the rounding to 16 bytes
    n = 32 * 50
    lens = np.where(np.arange(n) % 32 == 3, 27, 26 if refused and stated == 25 else 25)
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    rng = np.random.default_rng(5)
    cols, vals, x = rng.integers(0, n, ro[-1]).astype(np.int32), rng.normal(size=ro[-1]), rng.normal(size=n)
    dev = [torch.from_numpy(a).cuda() for a in (ro, cols, vals, x)]
    A = M.CSRMatrix(*dev[:3], max_row_len=stated)
    ctx = M.Context()
    y = torch.empty_like(dev[3])
    M.matvec(A, dev[3], y, ctx=ctx)
    if refused:
        with pytest.raises(M.MiniFEError):
            ctx.synchronize()
    else:
        ctx.synchronize()
        ref = np.add.reduceat(vals * x[cols], ro[:-1])
        size = np.add.reduceat(np.abs(vals * x[cols]), ro[:-1])
        assert (np.abs(y.cpu().numpy() - ref) <= 2 * (27 + 32) * 2.0**-53 * size).all()
    ctx.close()
