"""Resident solver loops of several threads: those that fit the device together run
side by side, and a solve that a stream capture refused leaves nothing behind that
another context meets."""
import os
import subprocess
import sys
import threading
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CAPTURE = """
import sys; sys.path.insert(0, %r)
import torch, minife_gb300 as M
A, b = M.build_system(9, 8, 7)
kw = dict(max_iter=300, tol=1e-9, tol_mode="relative", f64_operator="csr")
x, y = torch.zeros_like(b), torch.zeros_like(b)
torch.cuda.synchronize()
ctx = M.Context()
g = torch.cuda.CUDAGraph()
with torch.cuda.stream(torch.cuda.Stream()):
    g.capture_begin(capture_error_mode="relaxed")
    ctx.bind_torch_stream()
    try:
        M.cg_solve(A, b, x, ctx=ctx, **kw)
    except M.MiniFEError:
        print("refused")
    try:
        g.capture_end()
    except RuntimeError:
        pass
r = M.cg_solve(A, b, y, **kw)
print("status", r.status)
"""


def test_after_a_refused_capture():
    # in a process of its own: the first loop of all is the captured one
    p = subprocess.run([sys.executable, "-c", CAPTURE % ROOT], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert "refused" in p.stdout and "status 0" in p.stdout


def test_small_loops_run_side_by_side():
    # eight boxes of 729 rows, 12 blocks each, fit 152 SMs together: eight solves that
    # wait in a barrier nobody completes (0.2 s each) are over in the time of three,
    # where one after another they take eight
    n, wait = 8, 200_000_000
    ctxs = [M.Context() for _ in range(n)]
    systems = [M.build_system(8, 8, 8, ctx=c) for c in ctxs]
    x = [torch.zeros_like(b) for _, b in systems]
    torch.cuda.synchronize()
    status = [None] * n
    start = threading.Barrier(n + 1)

    def work(i):
        A, b = systems[i]
        M.cg_solve(A, b, x[i], max_iter=50, tol=1e-9, tol_mode="relative", ctx=ctxs[i])
        M.inject_loop_fault(wait, ctx=ctxs[i])
        start.wait()
        try:
            M.cg_solve(A, b, x[i], max_iter=50, tol=1e-30, tol_mode="absolute", ctx=ctxs[i])
        except M.MiniFEError as e:
            status[i] = e.status

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    start.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    assert status == [6] * n
    assert time.perf_counter() - t0 < 3 * wait * 1e-9
    for c in ctxs:
        c.close()
