"""The complex64 leaf sums and the last kernel by leaf box at the edges of their shares -- needs a GPU.

Near rows beyond one staged chunk of densities (1024) and boxes beyond one share of targets (32) on a
shallow tree, boxes of a few points on deep ones.  The bound on the complex64 form is the one the batched
form has (FP32 rounding of sums of some hundred terms, 2e-6); by box and by target differ by no more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ps,Pang,k,npatch,nlevels", [(5, 5, 60.0, 300, 4), (3, 3, 60.0, 110, 0), (7, 7, 60.0, 64, 0), (5, 7, 100.0, 33, 0)])
def test_gpu_mixed_by_box(lib, Ps, Pang, k, npatch, nlevels):
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=16, Ps=Ps, Pang=Pang, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, nlevels)
    g = np.random.default_rng(npatch)
    x = g.standard_normal(fm.total_num_unknowns_) + 1j * g.standard_normal(fm.total_num_unknowns_)
    y = fm.compute_Ax_acc(x)
    table = fm.get_tuning()
    out = {}
    for by_box in (True, False):
        t = table.copy()
        t[-1] = t[-1] | fm.SINGLE_INTERP_BY_BOX_C64 if by_box else t[-1] & ~fm.SINGLE_INTERP_BY_BOX_C64
        for chunks in (1, 2, 5, 10):
            t[1] = chunks
            fm.set_tuning(t)
            out[by_box, chunks] = fm.compute_Ax_acc(x, mixed=True)
            assert np.linalg.norm(out[by_box, chunks] - y) < 2e-6 * np.linalg.norm(y)
    assert np.array_equal(out[True, 5], (fm.set_tuning(table), fm.compute_Ax_acc(x, mixed=True))[1])


@pytest.mark.parametrize("nrhs", [1, 11, 12, 64 + 11, 64 + 12])
def test_gpu_batch_few_columns(lib, nrhs):
    """FP64 batches up to 11 columns, and remainders of that size, go column by column: on either side of the
    line each column is the single vector's, to the rounding of both (4e-15, as test_gpu_fixpoint.py)."""
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, 60.0, Np=16, patches_per_curve=64, formulation="combined")
    fm.precomps_and_setup(60.0, 0)
    g = np.random.default_rng(nrhs)
    X = g.standard_normal((fm.total_num_unknowns_, nrhs)) + 1j * g.standard_normal((fm.total_num_unknowns_, nrhs))
    Y = fm.apply_batch(X)
    for r in range(nrhs):
        y = fm.compute_Ax_acc(X[:, r])
        assert np.linalg.norm(Y[:, r] - y) <= 4e-15 * np.linalg.norm(y)
