"""The FP64 form's fixed-point sums at the ends of FP64's range and in large boxes -- needs a GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(lib, Ps=5, Pang=5, k=60.0, npatch=64, nlevels=0):
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=16, Ps=Ps, Pang=Pang, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, nlevels)
    return fm


@pytest.mark.parametrize("Ps,Pang", [(5, 5), (7, 7)])
def test_gpu_densities_near_the_ends_of_the_range(lib, Ps, Pang):
    """A density times 2^e gives the result times 2^e: the exact products scale, and where parts become
    subnormal each of some hundred roundings is below 2^-1074, 2^-80 of the smallest result here."""
    fm = _map(lib, Ps, Pang)
    n = fm.total_num_unknowns_
    g = np.random.default_rng(3)
    X = g.standard_normal((n, 13)) + 1j * g.standard_normal((n, 13))
    t = np.linspace(0, 2 * np.pi, 65)
    tx, ty = 1.8 * np.cos(t), 2.2 * np.sin(t)
    y, Y, u = fm.compute_Ax_acc(X[:, 0]), fm.apply_batch(X), fm.propagate_acc(tx, ty, X[:, 0])
    e = np.array([-990, -985, -960, -950, -940, -930, 0, 900, 980, 990, 1000, 1003, 1005])
    Ye = fm.apply_batch(X * np.exp2(e.astype(float)))
    for r in range(13):
        assert np.linalg.norm(Ye[:, r] * 2.0 ** float(-e[r]) - Y[:, r]) <= 1e-15 * np.linalg.norm(Y[:, r]), e[r]
    for q in e:
        z = fm.compute_Ax_acc(X[:, 0] * 2.0 ** float(q)) * 2.0 ** float(-q)
        assert np.linalg.norm(z - y) <= 1e-15 * np.linalg.norm(y), q
        v = fm.propagate_acc(tx, ty, X[:, 0] * 2.0 ** float(q)) * 2.0 ** float(-q)
        assert np.linalg.norm(v - u) <= 1e-15 * np.linalg.norm(u), q
