"""CSR products whose row lengths come in regions, so that whole groups of 32 rows
are larger than the stage that the mean row gives: they go through it in parts, and
rows too long for one lane are shared by several.

Bound as in test_gpu_spmv_any: (len + 32) roundings of the sum of |a||x| so far.
The time of a matrix of two regions is held against those of its halves alone: a
group that goes through the stage in two parts may take half as long again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

SHAPES = {
    # parts of 16 rows, of 8, of 4 and 2, of one row, and rows past the stage
    "4..7 | 27..32": lambda r, n: np.where(np.arange(n) < n // 2, r.integers(4, 8, n), r.integers(27, 33, n)),
    "2 | 30, a tenth": lambda r, n: np.where(np.arange(n) < n * 9 // 10, 2, 30),
    "1 | 54": lambda r, n: np.where(np.arange(n) < n * 9 // 10, 1, 54),
    "1 | 55..108": lambda r, n: np.where(np.arange(n) < n * 19 // 20, 1, r.integers(55, 109, n)),
    "0 | 109..432": lambda r, n: np.where(np.arange(n) < n * 49 // 50, 0, r.integers(109, 433, n)),
    "3 | 433..2000": lambda r, n: np.where(np.arange(n) < n * 99 // 100, 3, r.integers(433, 2001, n)),
    # staged groups with rows that one lane does not take
    "one of 100 a group": lambda r, n: np.where(np.arange(n) % 32 == 7, 100, 12),
    "8, 56": lambda r, n: np.where(np.arange(n) % 2 == 0, 8, 56),
    "empty rows among long": lambda r, n: np.where(np.arange(n) % 3 == 0, 0, np.where(np.arange(n) < n // 2, 5, 48)),
}


def make(lens, dtype, seed, spread=3000):
    rng = np.random.default_rng(seed)
    n = len(lens)
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    near = np.repeat(np.arange(n), lens) + rng.integers(-spread, spread + 1, ro[-1])
    cols = np.clip(near, 0, n - 1).astype(np.int32)
    vals, x = rng.normal(size=ro[-1]).astype(dtype), rng.normal(size=n).astype(dtype)
    return ro, cols, vals, x


@pytest.mark.parametrize("dtype,unit", [(np.float64, 2.0**-53), (np.float32, 2.0**-24)])
@pytest.mark.parametrize("n", [50, 20011])
@pytest.mark.parametrize("shape", SHAPES)
def test_regions(shape, n, dtype, unit):
    lens = SHAPES[shape](np.random.default_rng(6), n).astype(np.int64)
    ro, cols, vals, x = make(lens, dtype, 7)
    dev = [torch.from_numpy(a).cuda() for a in (ro, cols, vals, x)]
    prod = vals.astype(np.longdouble) * x[cols].astype(np.longdouble)
    rows = np.repeat(np.arange(n), lens)
    exact, size = np.zeros(n, dtype=np.longdouble), np.zeros(n, dtype=np.longdouble)
    np.add.at(exact, rows, prod)
    np.add.at(size, rows, np.abs(prod))
    ctx = M.Context()
    ctx.bind_torch_stream()
    # the longest row unknown, or stated where that keeps the kernel
    for stated in [0] + ([int(lens.max())] if lens.max() <= 32 else []):
        A = M.CSRMatrix(*dev[:3], max_row_len=stated)
        y = torch.full_like(dev[3], 7.0)
        M.matvec(A, dev[3], y, ctx=ctx)
        ctx.synchronize()
        err = np.abs(y.cpu().numpy().astype(np.longdouble) - exact)
        assert (err <= (lens + 32) * unit * size).all()
        d = M.matvec_and_dot(A, dev[3], y, ctx=ctx)
        yx = y.cpu().numpy().astype(np.longdouble) * x
        assert abs(d - float(yx.sum())) <= (n + 64) * 2.0**-53 * float(np.abs(yx).sum())
    ctx.close()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_time_of_two_regions(dtype):
    rng = np.random.default_rng(8)
    half = 600_000

    def us(lens):
        ro, cols, vals, x = make(lens, np.float64, 9, 30)
        ro, cols, vals, x = (torch.from_numpy(a).cuda() for a in (ro, cols, vals, x))
        A = M.CSRMatrix(ro, cols, vals.to(dtype))
        x = x.to(dtype)
        y = torch.empty_like(x)
        times = []
        for i in range(13):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            M.matvec(A, x, y)
            e.record()
            e.synchronize()
            times.append(s.elapsed_time(e))
        return min(times[3:])

    short, long = rng.integers(4, 8, half), rng.integers(27, 33, half)
    assert us(np.concatenate([short, long])) <= 1.5 * (us(short) + us(long))
