"""FP64 batches on either side of the line below which columns go one by one -- needs a GPU.

Tolerance of a column against the same column by another route: 4e-15, as in test_gpu_fixpoint.py.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(lib, k=60.0, npatch=64):
    fm = lib.ForwardMap(0.02, [lib.Kite()], (), 1.0, k, Np=16, patches_per_curve=npatch, formulation="combined")
    fm.precomps_and_setup(k, 0)
    return fm


@pytest.mark.parametrize("nrhs,shift", [(1, 0), (3, 0), (11, 0), (12, 0), (64 + 5, 0), (64 + 12, 0), (5, 1), (11, 3), (5, -1)])
def test_gpu_batch_in_place(lib, nrhs, shift):
    """Results written over the densities, at the same place or some columns on: a chunk's columns are read
    before any of its results is written."""
    import torch
    fm = _map(lib)
    n = fm.total_num_unknowns_
    g = torch.Generator().manual_seed(nrhs)
    x = torch.complex(torch.randn(nrhs, n, generator=g, dtype=torch.float64), torch.randn(nrhs, n, generator=g, dtype=torch.float64)).cuda()
    y = torch.empty_like(x)
    buf = torch.empty(nrhs + abs(shift), n, dtype=torch.complex128, device="cuda")
    at = max(0, -shift)
    buf[at:at + nrhs] = x
    torch.cuda.synchronize()
    fm.apply_batch_device(x, y, nrhs)
    fm.apply_batch_device(buf[at:], buf[at + shift:], nrhs)
    torch.cuda.synchronize()
    z = buf[at + shift:at + shift + nrhs]
    assert bool(((z - y).norm(dim=1) <= 4e-15 * y.norm(dim=1)).all())


@pytest.mark.parametrize("nrhs", [13, 33, 40, 64, 64 + 13])
def test_gpu_batch_passes_against_single(lib, nrhs):
    """Column counts whose every column takes a pass of the batched kernels."""
    fm = _map(lib)
    g = np.random.default_rng(nrhs)
    X = g.standard_normal((fm.total_num_unknowns_, nrhs)) + 1j * g.standard_normal((fm.total_num_unknowns_, nrhs))
    Y = fm.apply_batch(X)
    for r in range(nrhs):
        y = fm.compute_Ax_acc(X[:, r])
        assert np.linalg.norm(Y[:, r] - y) <= 4e-15 * np.linalg.norm(y), r
