"""The batched EEQ by conjugate gradients with the set-up inverse (k_eeq_cg): sizes at the edges of
its row groups and on both sides of every cluster size, geometries off the set-up, several
fragments, and a molecule whose matrix is not positive definite (left to the Cholesky kernel).

Tolerances: the FP64 solve is accepted at a true residual of 1e-12 max|b| and runs to 1e-15; the
charges of these matrices (smallest eigenvalue >= 0.1) then agree to 1e-11 at worst, energies
(stationary in the charges) to rounding, gradients to 1e-11."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, workloads
from tests.indefinite_systems import h2_chain
from tests.oracle_api import Oracle

pytestmark = pytest.mark.gpu


# unknowns 7 .. 304: one CTA, clusters of 2, 4 and 8; multiples of four rows and their neighbours
@pytest.mark.parametrize("nc", [2, 3, 9, 16, 21, 32, 33, 61, 87, 100])
def test_single_alkane(nc, monkeypatch):
    monkeypatch.setenv("GFNFF_EEQ_SOLVER", "batched")
    Z, X = workloads.alkane(nc, nc)
    g = GFNFF(precision=FP64)
    assert g.setMolecule(Z, X), g.getErrorMessage()
    assert g.eeqSolver() == "batched"
    rng = np.random.default_rng(nc)
    for step in range(3):   # the set-up geometry, then off it
        x = X + (0.03 * step) * rng.normal(size=X.shape).clip(-2, 2)
        g.updateGeometry(x)
        e = g.calculateEnergy(True)
        assert not g.hasError(), g.getErrorMessage()
        T, G, q, cn = Oracle(Z, X).engrad(x)
        assert abs(e - T["total"]) < 1e-9
        assert np.abs(g.getCharges() - q).max() < 1e-10
        assert np.abs(g.getGradient() - G).max() < 1e-9
        assert 1 <= g.eeqIterations() < 60


def test_batch_mixed_sizes_and_fragments():
    mols = [workloads.alkane(n, n) for n in (1, 2, 8, 30, 64, 100)]
    mols += [workloads.water_cluster(n, n) for n in (1, 7, 40)]
    g = GFNFF(precision=FP64)
    assert g.setMoleculeBatch(mols), g.getErrorMessage()
    for _ in range(3):   # repeated: no state of one evaluation reaches the next
        e, st = g.calculateEnergyBatch()
        assert (st == 0).all()
        Q = np.split(g.getCharges(), np.cumsum([len(z) for z, _ in mols])[:-1])
        for (Z, X), em, qm in zip(mols, e, Q):
            T, G, q, cn = Oracle(Z, X).engrad(X)
            assert abs(em - T["total"]) < 1e-9
            assert np.abs(qm - q).max() < 1e-10


def test_batch_with_indefinite_molecule(monkeypatch):
    """Same statuses and energies as the Cholesky kernel alone gives."""
    mols = [workloads.alkane(12, 1), h2_chain(), workloads.alkane(50, 2)]
    out = []
    for direct in (False, True):
        if direct:
            monkeypatch.setenv("GFNFF_BATCH_TC", "0")
        g = GFNFF(precision=FP64)
        assert g.setMoleculeBatch(mols), g.getErrorMessage()
        out.append(g.calculateEnergyBatch())
    (e0, s0), (e1, s1) = out
    assert (s0 == s1).all()
    assert s0[0] == 0 and s0[2] == 0
    assert np.abs(e0 - e1).max() < 1e-9
