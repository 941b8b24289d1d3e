"""A new context's products report no error of another's: the word that they
record errors in starts at zero, also where its memory was used before."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


def test_new_context_starts_clean():
    n = 320
    ro = torch.arange(0, 27 * n + 1, 27, dtype=torch.int32, device="cuda")
    cols = (torch.arange(27 * n, device="cuda") % n).to(torch.int32)
    vals, x = torch.ones(27 * n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    good, bad = M.CSRMatrix(ro, cols, vals), M.CSRMatrix(ro, cols, vals, max_row_len=4)
    for _ in range(20):
        ctx = M.Context()
        M.matvec(good, x, torch.empty_like(x), ctx=ctx)
        ctx.synchronize()
        # leave a recorded error behind when the context goes
        M.matvec(bad, x, torch.empty_like(x), ctx=ctx)
        torch.cuda.synchronize()
        ctx.close()
