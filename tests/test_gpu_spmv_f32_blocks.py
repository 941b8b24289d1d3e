"""FP32 CSR products on both sides of the mean row length (19) from which a block has
eight warps instead of two, at row numbers around a block's share (64 and 256 rows)
and around those (four groups a warp of 152 SMs) from which they may be eight.

Bound as in test_gpu_spmv_any: (len + 32) 2^-24 sum |a||x|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


@pytest.mark.parametrize("length", [17, 18, 19, 20, 27, 32])
@pytest.mark.parametrize("n", [1, 63, 65, 255, 257, 4 * 32 * 24 * 152 - 1, 4 * 32 * 24 * 152, 4 * 32 * 24 * 152 + 257])
def test_rows(n, length):
    rng = np.random.default_rng(length)
    lens = np.clip(rng.integers(length - 2, length + 3, n), 1, 32)
    ro = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = np.clip(np.repeat(np.arange(n), lens) + rng.integers(-3000, 3001, ro[-1]), 0, n - 1).astype(np.int32)
    vals, x = rng.normal(size=ro[-1]).astype(np.float32), rng.normal(size=n).astype(np.float32)
    A = M.CSRMatrix(*(torch.from_numpy(a).cuda() for a in (ro, cols, vals)))
    xd = torch.from_numpy(x).cuda()
    y = torch.full_like(xd, 7.0)
    d = M.matvec_and_dot(A, xd, y)
    prod = vals.astype(np.float64) * x[cols]
    exact, size = np.add.reduceat(prod, ro[:-1]), np.add.reduceat(np.abs(prod), ro[:-1])
    yh = y.cpu().numpy().astype(np.float64)
    assert (np.abs(yh - exact) <= (lens + 32) * 2.0**-24 * size).all()
    assert abs(d - float(yh @ x)) <= (n + 64) * 2.0**-52 * float(np.abs(yh * x).sum())
