"""The fixed-point Green values (csrc/green_fx.cuh) against scipy over their range -- needs a GPU.

One unit density makes the direct field at a target the Green value times the source's quadrature weight.
Arguments x = k r from 1e-3 (FP64 series below 1) over every piece of the phase-free tables and their
edges to 1e5; both formulations; wavenumbers whose mantissas are at the ends of their range.  The bound: a
dozen FP64 roundings (4e-15 covers scipy's as well) plus x times the rounding of k and r (5e-16).
"""
import numpy as np
import pytest
from scipy.special import hankel1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,k", [("combined", 500.0), ("combined", 64.0), ("single_layer", 127.99999999999999), ("single_layer", 10.0)])
@pytest.mark.parametrize("count", [300, 45000])           # a block per target, a thread per target
def test_gpu_green_values(lib, form, k, count):
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=10, patches_per_curve=20, formulation=form)
    fm.compute_precomputations(k)
    n, j = fm.total_num_unknowns_, 77
    g = np.random.default_rng(int(k))
    edges = np.concatenate([2.0 ** np.arange(0, 10) * f for f in (1 - 1e-6, 1.0, 1 + 1e-6)] + [1.0 + np.arange(64) / 64.0])
    x = np.concatenate([edges, np.exp(g.uniform(np.log(1e-3), np.log(1e5), count - edges.size))])
    th = g.uniform(0, 2 * np.pi, count)
    tx, ty = fm.xs_[j] + x / k * np.cos(th), fm.ys_[j] + x / k * np.sin(th)
    d = np.zeros(n, complex)
    d[j] = 1.0
    out = fm.propagate_unacc(tx, ty, d)
    dx, dy = tx - fm.xs_[j], ty - fm.ys_[j]
    r = np.hypot(dx, dy)
    h0, h1 = hankel1(0, k * r), hankel1(1, k * r)
    if form == "combined":
        a, b = 0.25j * k * (dx * fm.nxs_[j] + dy * fm.nys_[j]) / r * h1, 0.25 * k * h0
    else:
        a, b = 0.25j * h0, np.zeros(count)
    e, scale = a + b, np.abs(a) + np.abs(b)
    w = (out[:64] / e[:64]).real.mean()
    err = np.abs(out / w - e) / scale
    assert np.all(err < 4e-15 + 5e-16 * k * r), (np.max(err), k * r[np.argmax(err / (4e-15 + 5e-16 * k * r))])
