"""Conjugate gradients of large systems of long chains: the preconditioner takes whole fragments (512
unknowns at most), whose rows one grid block owns, and still has to fit into shared memory.

Tolerances: both forms are accepted on their true FP64 residual (1e-12 of the right-hand side; 1e-10), so
energies agree to the FP32 coordination numbers of the mixed form (some 1e-9 of 1 Eh per atom of a
chain; 1e-6 is the mixed form's bar), gradients to 1e-5 (the same)."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, MIXED, workloads

pytestmark = pytest.mark.gpu


def rods(count, nc=170):
    """count parallel all-trans alkanes, 6 A apart"""
    Z, X = workloads.alkane(nc, noise=False)
    X = X - X.mean(axis=0)
    X = X @ np.linalg.svd(X, full_matrices=False)[2].T
    side = int(np.ceil(np.sqrt(count)))
    return np.tile(Z, count), np.concatenate([X + np.array([0, 6.0 * (k % side), 6.0 * (k // side)])
                                              for k in range(count)])


def test_whole_chains_at_20951_unknowns():
    Z, X = rods(41)
    x = X + np.random.default_rng(0).normal(scale=0.02, size=X.shape)
    out = []
    for precision in (FP64, MIXED):
        g = GFNFF(precision=precision)
        assert g.setMolecule(Z, X), g.getErrorMessage()
        assert g.eeqSolver() == "pcg"
        g.updateGeometry(x)
        e = g.calculateEnergy(True)
        assert not g.hasError(), g.getErrorMessage()
        assert 1 <= g.eeqIterations() < 120   # 59; cut chains take 200
        if precision == MIXED:
            assert g.eeqFP64Products() >= 1   # the FP32 matrix inside FP64 refinement
        out.append((e, g.getGradient().copy()))
        g.close()
    assert abs(out[0][0] - out[1][0]) < 1e-6
    assert np.abs(out[0][1] - out[1][1]).max() < 1e-5
