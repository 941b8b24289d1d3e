"""tune_multi also times the solver's own z steps (z_chunk 0) and keeps the faster,
driven by solve times from a table (no GPU)."""
import pytest

from minife_gb300 import autotune


class _Vec:
    shape = (8, 32)

    def zero_(self):
        return self


class _Box:
    box = (16, 16, 16)


class _CG:
    def __init__(self, t, status):
        self.status = status
        self.times = (0.0, 0.0, 0.0, 0.0, t)


@pytest.mark.parametrize("own,status,chosen", [(0.9, 0, 0), (1.0, 0, 32), (0.5, 5, 32), (1.3, 0, 32)])
def test_own_choice(own, status, chosen, tmp_path, monkeypatch):
    import minife_gb300 as M
    monkeypatch.setenv("MFE_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune, "_device_key", lambda: "fake/sm1")
    applied = [None]

    def solve(A, B, X, max_iter, tol, tol_mode, precision, refine_k, inner_tol):
        z = applied[-1]
        if z == 0:
            return [_CG(own, status)] * 2
        return [_CG(1.0 + abs(z - 32) / 100 + abs(refine_k - 50) / 1000, 5 if tol == 0.0 else 0)] * 2

    monkeypatch.setattr(M, "set_multi_tuning", applied.append)
    monkeypatch.setattr(M, "cg_solve_multi", solve)
    cfg = autotune.tune_multi(_Box(), _Vec(), _Vec(), reps=1)
    assert cfg["z_chunk"] == chosen == applied[-1]
    assert cfg["solve_seconds"] == (own if chosen == 0 else 1.0)
    again = autotune.tune_multi(_Box(), _Vec(), _Vec(), reps=1)
    assert again["cached"] and again["z_chunk"] == chosen == applied[-1]
