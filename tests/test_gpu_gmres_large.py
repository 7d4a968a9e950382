"""GMRES on vectors on either side of the length from which a kernel adds up the dot products -- needs a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npatch", [4096, 4097, 4160])          # 32 chunks of 2048 rows, 33 with a short one, 33
def test_gpu_gmres_long_vectors(lib, npatch):
    """Against the batched solve, whose dot products are another kernel's: both stop below 1e-9 of the right-hand
    side, and the operator's condition is some tens."""
    k = 60.0
    fm = lib.ForwardMap(0.001, [lib.Kite()], (), 1.0, k, Np=16, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, 0)
    b = -np.exp(1j * k * fm.xs_)
    x = fm.gmres(b, tol=1e-9)
    its = fm.last_solve["iters"]
    r = b - fm.compute_Ax_acc(x)
    assert np.linalg.norm(r) < 2e-9 * np.linalg.norm(b)
    xb = fm.gmres_batch(b[:, None], tol=1e-9)[:, 0]
    assert np.linalg.norm(x - xb) < 1e-7 * np.linalg.norm(xb)
    assert abs(its - fm.last_solve["iters"][0]) <= 1
