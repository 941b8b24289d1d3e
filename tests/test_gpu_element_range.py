"""Element matrices whose conductivities leave the integer multiplication's
range (zero, negative, subnormal, huge): the assembly stays the oracle's bit for
bit, in elements side by side with ordinary ones and on flat boxes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only machines
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import minife_gb300 as M  # noqa: E402


@pytest.mark.parametrize("dims", [(5, 4, 3), (9, 7, 18), (3000, 2, 2), (2, 2, 700)])
def test_extreme_conductivities_bitexact(dims):
    rng = np.random.default_rng(5)
    kappa = np.exp(rng.normal(size=dims[0] * dims[1] * dims[2]))
    special = np.array([0.0, -0.0, -1.5, 5e-324, 1e-250, -1e-190, 1e-60, 1e60, 1e190, -1e250])
    at = rng.choice(kappa.size, size=min(kappa.size // 2, 60), replace=False)
    kappa[at] = special[np.arange(at.size) % special.size]
    A, b = M.build_system(*dims, kappa=torch.from_numpy(kappa).cuda())
    ro, cols, vals, bo = O.build_system(*dims, kappa=kappa)
    assert np.array_equal(A.packed_coefs.cpu().numpy().view(np.int64), vals.view(np.int64))
    assert np.array_equal(b.cpu().numpy().view(np.int64), bo.view(np.int64))
