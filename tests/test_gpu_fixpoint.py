"""The FP64 form's fixed-point cone sums at the edges of their range -- needs a GPU.

Blocks of coefficients carry a binary exponent, so scaling a density by a power of two scales the
result exactly as long as no exponent leaves the range; the arithmetic error of an apply, seen in
the additivity defect A(x1 + x2) - A x1 - A x2 with x1 + x2 exact, stays at FP64's rounding (2^-53
per sum of a few hundred terms: 4e-15 of the result bounds it ten times over); zeros, isolated
sources and non-finite values behave as in FP64 arithmetic.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [(3, 3), (5, 5), (6, 6), (5, 7), (7, 7)]


def _map(lib, Ps=5, Pang=5, k=100.0, npatch=110):
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=16, Ps=Ps, Pang=Pang, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, 0)
    return fm


def _f32(g, n):
    return g.standard_normal(n).astype(np.float32).astype(float) + 1j * g.standard_normal(n).astype(np.float32).astype(float)


@pytest.mark.parametrize("Ps,Pang", ORDERS)
def test_gpu_fixpoint_scaling_and_rounding(lib, Ps, Pang):
    fm = _map(lib, Ps, Pang)
    n = fm.total_num_unknowns_
    g = np.random.default_rng(Ps * 10 + Pang)
    x1, x2 = _f32(g, n), _f32(g, n)
    y = fm.compute_Ax_acc(x1)
    for e in (-600, 600):
        s = 2.0 ** e
        assert np.array_equal(fm.compute_Ax_acc(x1 * s), y * s)
    d = fm.compute_Ax_acc(x1 + x2) - y - fm.compute_Ax_acc(x2)
    assert np.linalg.norm(d) < 4e-15 * np.linalg.norm(y)
    # a density of magnitudes falling by 1e-30 along the curve: every part keeps its own relative error
    w = np.exp(-np.linspace(0.0, 69.0, n))
    a, b = x1 * w, np.zeros(n, complex)
    b[: n // 2] = a[: n // 2]
    c = a - b
    d = fm.compute_Ax_acc(a) - fm.compute_Ax_acc(b) - fm.compute_Ax_acc(c)
    assert np.linalg.norm(d) < 4e-15 * np.linalg.norm(fm.compute_Ax_acc(a))


def test_gpu_fixpoint_zero_isolated_and_nonfinite(lib, oracle):
    import torch
    k, npatch = 100.0, 110
    fm = _map(lib, k=k, npatch=npatch)
    n = fm.total_num_unknowns_
    assert not np.any(fm.compute_Ax_acc(np.zeros(n, complex)))
    om = oracle.OracleForwardMap([oracle.curve_kite()], 16, 0.02, 1.0, k, patches_per_curve=npatch, formulation="combined")
    om.precompute(k)
    om.setup_ifgf(k, fm.nlevels)
    x = np.zeros(n, complex)
    x[n // 3] = 1.0 - 2.0j                       # one source: all other boxes' blocks are zero
    y, yo = fm.compute_Ax_acc(x), om.compute_Ax_acc(x)
    assert np.linalg.norm(y - yo) < 1e-6 * np.linalg.norm(yo)     # the singular weights' one-ulp sensitivity
    far, faro = fm.ifgf_far(x), om.ifgf_far(x) if hasattr(om, "ifgf_far") else None
    if faro is not None:
        assert np.linalg.norm(far - faro) < 1e-11 * np.linalg.norm(faro)
    for bad in (np.nan, np.inf):
        v = torch.from_numpy(_f32(np.random.default_rng(1), n)).cuda()
        v[n // 2] = complex(bad, 0.0)
        out = torch.empty_like(v)
        torch.cuda.synchronize()
        fm.apply_device(v, out)
        torch.cuda.synchronize()
        assert not bool(torch.isfinite(torch.view_as_real(out)).all(dim=1).any())


@pytest.mark.parametrize("Ps,Pang,npatch,nlevels", [(5, 5, 300, 4), (3, 3, 110, 0), (7, 7, 64, 0)])
def test_gpu_fixpoint_near_and_leaf_sums(lib, oracle, Ps, Pang, npatch, nlevels):
    """Leaf boxes beyond one staged chunk of sources (256) and near rows beyond one (512) on a shallow
    tree; boxes of a few sources on a deep one.  The far sums against the oracle's to the tables' rounding,
    batches of 1, 33 and 64 against the single vector to the bound above."""
    import torch
    k = 60.0
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=16, Ps=Ps, Pang=Pang, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, nlevels)
    om = oracle.OracleForwardMap([oracle.curve_kite()], 16, 0.02, 1.0, k, patches_per_curve=npatch, formulation="combined")
    om.precompute(k)
    om.setup_ifgf(k, fm.nlevels, Ps, Pang)
    n = fm.total_num_unknowns_
    g = np.random.default_rng(npatch)
    X = np.stack([_f32(g, n) for _ in range(64)], axis=1)
    X[:, 3] = 0
    X[:, 5] *= 2.0 ** -600
    far, faro = fm.ifgf_far(X[:, 0]), om.ifgf_far(X[:, 0])
    assert np.linalg.norm(far - faro) < 1e-11 * np.linalg.norm(faro)
    Y = np.stack([fm.compute_Ax_acc(X[:, r]) for r in range(64)], axis=1)
    for B in (1, 33, 64):
        Yb = fm.apply_batch(X[:, :B])
        s = 2.0 ** np.array([600.0 if r == 5 else 0.0 for r in range(B)])
        assert np.all(np.linalg.norm((Yb - Y[:, :B]) * s, axis=0) <= 4e-15 * np.linalg.norm(Y[:, :B] * s, axis=0)), B
    x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    y, yn = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    fm.apply_batch_device(x, y, 64)
    x[7, n // 2] = complex(np.nan, 0.0)           # a column's NaN stays in it
    torch.cuda.synchronize()
    fm.apply_batch_device(x, yn, 64)
    torch.cuda.synchronize()
    fin = torch.isfinite(torch.view_as_real(yn)).all(dim=2)
    keep = torch.arange(64, device="cuda") != 7
    assert not bool(fin[7].any()) and bool(fin[keep].all()) and torch.equal(yn[keep], y[keep])
