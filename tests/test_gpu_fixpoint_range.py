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


def _weights(npatch, Np=16):
    """the kite's quadrature weights: Fejer's first rule on equal parts of the parameter, times the arc length"""
    th = np.pi * (2 * np.arange(Np) + 1) / (2 * Np)
    w = 2 / Np * (1 - 2 * sum(np.cos(2 * m * th) / (4 * m * m - 1) for m in range(1, Np // 2 + 1)))
    t = (np.pi / npatch) * (2 * np.arange(npatch)[:, None] + 1 + np.cos(th)[None, :])
    return ((np.pi / npatch) * w[None, :] * np.hypot(-np.sin(t) - 1.3 * np.sin(2 * t), 1.5 * np.cos(t))).ravel()


@pytest.mark.parametrize("npatch,nlevels", [(1024, 3), (512, 4)])
def test_gpu_small_densities_beside_a_large_one_in_a_large_box(lib, npatch, nlevels):
    """Leaf boxes of several hundred to a thousand points: one intensity of 1 and, around it, others of 5 units
    of 2^-53.  Densities keep 54 bits in a box of any size, so the small ones are held exactly; coefficients
    and results are rounded at 2^-53 of the large one's field, some 2e-2 of the small ones' few hundred."""
    fm = _map(lib, k=20.0, npatch=npatch, nlevels=nlevels)
    n = fm.total_num_unknowns_
    w = _weights(npatch)
    j = n // 5
    d = np.hypot(fm.xs_ - fm.xs_[j], fm.ys_ - fm.ys_[j])
    spike, small = np.zeros(n, complex), np.zeros(n, complex)
    spike[j] = 1.0
    small[(d < 0.3) & (d > 0)] = 5 * 2.0 ** -53
    far = d > 1.6                                       # beyond the neighbour boxes

    def check(a, b, c):
        assert np.linalg.norm((c - a - b)[far]) < 0.1 * np.linalg.norm(b[far])

    check(fm.ifgf_far(spike), fm.ifgf_far(small), fm.ifgf_far(spike + small))
    for nrhs in (13, 40):
        X = np.zeros((n, nrhs), complex)
        X[:, 0], X[:, 5], X[:, nrhs - 1] = spike / w, small / w, (spike + small) / w
        Y = fm.apply_batch(X)
        check(Y[:, 0], Y[:, 5], Y[:, nrhs - 1])
        assert not Y[:, 1].any()


@pytest.mark.parametrize("k,npatch,nlevels,chunks", [(20.0, 256, 3, 5), (500.0, 512, 0, 2)])
def test_gpu_leaf_shapes(lib, k, npatch, nlevels, chunks):
    """The set-up takes five threads a coefficient for few leaf cones and two for many; integer sums are the
    same in every shape.  A shape that was set stays over the next set-up."""
    fm = _map(lib, k=k, npatch=npatch, nlevels=nlevels)
    g = np.random.default_rng(npatch)
    x = g.standard_normal(fm.total_num_unknowns_) + 1j * g.standard_normal(fm.total_num_unknowns_)
    y = fm.compute_Ax_acc(x)
    t = fm.get_tuning()
    assert t[0] == chunks
    for c in (1, 2, 5, 10):
        t[0] = c
        fm.set_tuning(t)
        fm.precomps_and_setup(k, nlevels)
        assert fm.get_tuning()[0] == c
        assert np.array_equal(fm.compute_Ax_acc(x), y)


def test_gpu_parts_of_a_falling_density(lib, oracle):
    """A density that falls by 1e-30 along the curve, quarter by quarter: the far field of each quarter alone has
    the oracle's digits (1e-11, the tables' rounding, as in test_gpu_fixpoint.py), however small the quarter is,
    single vector and batch; the whole is the sum of the quarters to the rounding of the largest."""
    k, npatch = 60.0, 64
    fm = _map(lib, k=k, npatch=npatch)
    om = oracle.OracleForwardMap([oracle.curve_kite()], 16, 0.02, 1.0, k, patches_per_curve=npatch, formulation="combined")
    om.precompute(k)
    om.setup_ifgf(k, fm.nlevels)
    n = fm.total_num_unknowns_
    g = np.random.default_rng(5)
    x = (g.standard_normal(n) + 1j * g.standard_normal(n)) * np.exp(-np.linspace(0.0, 69.0, n))
    parts = np.zeros((n, 13), complex)
    for q in range(4):
        parts[q * n // 4:(q + 1) * n // 4, 3 * q] = x[q * n // 4:(q + 1) * n // 4]
    Y = fm.apply_batch(parts)
    whole = fm.compute_Ax_acc(x)
    for q in range(4):
        p = parts[:, 3 * q]
        far, faro = fm.ifgf_far(p), om.ifgf_far(p)
        assert np.linalg.norm(far - faro) < 1e-11 * np.linalg.norm(faro), q
        y = fm.compute_Ax_acc(p)
        assert np.linalg.norm(Y[:, 3 * q] - y) <= 4e-15 * np.linalg.norm(y), q
        whole = whole - y
    assert np.linalg.norm(whole) < 4e-15 * np.linalg.norm(Y[:, 0])
