"""Solves whose iterations run in one resident kernel, from several threads at
once, each with its own context and stream: their kernels fill the device one
after another, none waits for blocks that cannot start, and every solve gives the
bits that it gives alone (the sums' order does not depend on the others)."""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

JOBS = [((40, 40, 40), "f64", "auto"), ((30, 30, 30), "f64", "csr"), ((82, 80, 81), "f64", "auto"),
        ((64, 64, 64), "mixed", "auto"), ((24, 24, 24), "mixed", "auto")]


def solve(i, ctx):
    dims, precision, operator = JOBS[i]
    A, b = M.build_system(*dims, ctx=ctx)
    x = torch.zeros_like(b)
    r = M.cg_solve(A, b, x, max_iter=2000, tol=1e-9, tol_mode="relative", precision=precision,
                   f64_operator=operator, ctx=ctx)
    return r.status, r.num_iters, x


def test_concurrent_loops():
    alone = [solve(i, M.default_context()) for i in range(len(JOBS))]
    torch.cuda.synchronize()
    got, errors = {}, []

    def work(i):
        try:
            ctx = M.Context()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    got[i] = solve(i, ctx)
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # reported below, in the main thread
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(JOBS))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i, (status, iters, x) in enumerate(alone):
        assert got[i][:2] == (status, iters) and status == 0
        assert torch.equal(got[i][2], x)
