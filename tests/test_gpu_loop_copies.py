"""Loop bodies of one and several iterations: solves that end after a few, whose
reliable updates come every few, and that run on, in the graph against the same
kernels issued one by one (MFE_CG_EAGER=1): the same bits.  And the time of updates in
every iteration: a body of several iterations would run its rest empty each time."""
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402

STOPS = [dict(max_iter=1), dict(max_iter=7), dict(max_iter=300), dict(max_iter=300, refine_k=1),
         dict(max_iter=300, refine_k=3), dict(max_iter=300, refine_k=5), dict(max_iter=300, inner_tol=0.5)]


def normal(shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def both(run, monkeypatch):
    x, n = run()
    monkeypatch.setenv("MFE_CG_EAGER", "1")
    y, m = run()
    assert n == m
    assert torch.equal(x, y)


@pytest.mark.parametrize("kw", STOPS)
@pytest.mark.parametrize("dims", [(5, 4, 3), (20, 18, 24)])
def test_multi(dims, kw, monkeypatch):
    A, b = M.build_system(*dims)
    B = normal((b.numel(), 32))

    def run():
        X = torch.zeros_like(B)
        r = M.cg_solve_multi(A, B, X, tol=1e-11, tol_mode="relative", **kw)
        return X, [(v.num_iters, v.status, v.refinements) for v in r]

    both(run, monkeypatch)


@pytest.mark.parametrize("kw", STOPS)
@pytest.mark.parametrize("precision", ["mixed", "f64"])
@pytest.mark.parametrize("boxes", [[(3, 3, 3)] * 4, [(20, 18, 24), (5, 40, 7), (16, 16, 16)]])
def test_batch(boxes, precision, kw, monkeypatch):
    batch = M.Batch(boxes)

    def run():
        x, r = batch.solve(tol=1e-11, tol_mode="relative", precision=precision, **kw)
        return x.clone(), [(v.num_iters, v.status, v.refinements) for v in r]

    both(run, monkeypatch)
    batch.close()


@pytest.mark.parametrize("kw", STOPS[:2] + [dict(max_iter=60, refine_k=1), dict(max_iter=60, refine_k=5)])
def test_mixed(kw, monkeypatch):
    A, b = M.build_system(127, 126, 125)  # past the resident loop
    b = normal(b.shape)

    def run():
        x = torch.zeros_like(b)
        r = M.cg_solve(A, b, x, tol=1e-11, tol_mode="relative", precision="mixed", **kw)
        return x, (r.num_iters, r.status, r.refinements)

    both(run, monkeypatch)


def test_time_of_frequent_updates():
    # an update is two kernels beside the iteration's three, so five of them in place
    # of one cannot take a solve past (1 + 1) / (1 + 1 / 5) = 1.67 of its time
    A, b = M.build_system(8, 8, 8)
    B = normal((b.numel(), 32))
    X = torch.zeros_like(B)

    def ms(k):
        times = []
        for _ in range(9):
            X.zero_()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            M.cg_solve_multi(A, B, X, max_iter=60, tol=1e-12, tol_mode="relative", refine_k=k)
            times.append(time.perf_counter() - t0)
        return 1e3 * min(times[2:])

    assert ms(1) <= 1.67 * ms(5)
