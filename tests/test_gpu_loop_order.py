"""Resident solver loops of several contexts: a solve that a stream capture refused
leaves nothing behind that another context meets."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

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
