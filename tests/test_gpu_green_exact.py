"""The fixed-point Green values where |d|^2 is exact -- needs a GPU and mpmath.

The targets lie on a horizontal line through the source at distances of 24 bits, so that target minus source
and its square are exact and nothing but the Green value is rounded.  The bound is fourteen FP64 roundings
(1.6e-15) of the terms' magnitudes: d.n, the amplitude (mantissa, scale, their product), the value, its products
with the weight and their sum, and as many for the weight; and k r times the unit in which r enters the phase
(2^-58 of a power of two, twice that at worst).  The weight, the factor between field and Green value, is taken
from the arguments below 1, which the FP64 series evaluates, and compared with the quadrature rule.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["combined", "single_layer"])
@pytest.mark.parametrize("k", [40.0, 977.0, 262143.0])
def test_gpu_green_values_of_exact_distances(lib, form, k):
    mp = pytest.importorskip("mpmath")
    npatch, Np = 20, 10
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=Np, patches_per_curve=npatch, formulation=form)
    fm.compute_precomputations(k)
    n = fm.total_num_unknowns_
    j = int(np.argmax(np.where((fm.xs_ > 0.5) & (fm.xs_ < 1.0), np.abs(fm.nxs_), 0.0)))
    g = np.random.default_rng(int(k))
    # a fifth below x = 1, then each octave's ends and points of all octaves
    top = 0.49 * k
    x = np.concatenate([g.uniform(0.2, 0.9, 64), 2.0 ** np.arange(0, np.log2(top)) * 1.0005, np.exp(g.uniform(0.0, np.log(top), 200))])
    dx = (x / k).astype(np.float32).astype(float)
    tx, ty = fm.xs_[j] - dx, np.full(dx.size, fm.ys_[j])
    assert np.array_equal(fm.xs_[j] - tx, dx)
    d = np.zeros(n, complex)
    d[j] = 1.0
    out = fm.propagate_unacc(tx, ty, d)
    mp.mp.dps = 40
    e, scale = np.zeros(dx.size, complex), np.zeros(dx.size)
    for i, v in enumerate(dx):
        z = mp.mpf(k) * mp.mpf(float(v))
        h0 = mp.hankel1(0, z)
        if form == "combined":
            a, b = mp.mpc(0, 0.25) * k * mp.mpf(float(-fm.nxs_[j])) * mp.hankel1(1, z), mp.mpf(k) / 4 * h0
        else:
            a, b = mp.mpc(0, 0.25) * h0, mp.mpf(0)
        e[i], scale[i] = complex(a + b), float(abs(a) + abs(b))
    t = np.pi * (2 * np.arange(Np) + 1) / (2 * Np)
    f = 2 / Np * (1 - 2 * sum(np.cos(2 * m * t) / (4 * m * m - 1) for m in range(1, Np // 2 + 1)))
    s = (np.pi / npatch) * (2 * (j // Np) + 1 + np.cos(t[j % Np]))
    rule = (np.pi / npatch) * f[j % Np] * np.hypot(-np.sin(s) - 1.3 * np.sin(2 * s), 1.5 * np.cos(s))
    small = k * dx < 1
    w = np.median((out[small] / e[small]).real)
    assert abs(w - rule) < 1e-13 * rule
    err = np.abs(out / w - e) / scale
    assert np.all(err < 1.6e-15 + 2.0 ** -57 * k * dx), (err.max(), k * dx[err.argmax()])
