"""The batched EEQ by conjugate gradients with the set-up inverse (k_eeq_cg): sizes at the edges of
its row groups and on both sides of every cluster size, geometries off the set-up, several
fragments, and molecules whose matrix is not, or hardly, positive definite (left to the elimination).

Tolerances: the FP64 solve is accepted at a true residual of 1e-12 max|b| and runs to 1e-15; the
charges of these matrices (smallest eigenvalue >= 0.1) then agree to 1e-11 at worst, energies
(stationary in the charges) to rounding, gradients to 1e-11."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, MIXED, _lib, workloads
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
    assert g.eeqSolver() == "batched" and g.batchKernel() == "cg"
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
    """At the set-up geometry, where the preconditioner is the matrix's own inverse, off it, and there again"""
    mols = [workloads.alkane(n, n) for n in (1, 2, 8, 30, 64, 100)]
    mols += [workloads.water_cluster(n, n) for n in (1, 7, 40)]
    g = GFNFF(precision=FP64)
    assert g.setMoleculeBatch(mols), g.getErrorMessage()
    assert g.batchKernel() == "cg"
    rng = np.random.default_rng(4)
    noise = [rng.normal(size=x.shape).clip(-2, 2) for _, x in mols]
    iterations = []
    for scale in (0.0, 0.02, 0.06, 0.0):   # no state of one evaluation reaches the next
        xs = [x + scale * d for (_, x), d in zip(mols, noise)]
        g.updateGeometry(np.concatenate(xs))
        e, st = g.calculateEnergyBatch()
        assert (st == 0).all()
        iterations.append(g.eeqIterations())
        cuts = np.cumsum([len(z) for z, _ in mols])[:-1]
        for (Z, X), x, em, qm, gm in zip(mols, xs, e, np.split(g.getCharges(), cuts), np.split(g.getGradient(), cuts)):
            T, G, q, cn = Oracle(Z, X).engrad(x)
            assert abs(em - T["total"]) < 1e-9
            assert np.abs(qm - q).max() < 1e-10
            assert np.abs(gm - G).max() < 1e-9
    assert iterations[0] == iterations[3] < iterations[1] < iterations[2] < 30, iterations


def test_batch_with_indefinite_molecule(monkeypatch):
    """Same statuses and energies as the Cholesky kernel alone gives."""
    mols = [workloads.alkane(12, 1), h2_chain(), workloads.alkane(50, 2)]
    out = []
    for direct in (False, True):
        if direct:
            monkeypatch.setenv("GFNFF_BATCH_TC", "0")
        g = GFNFF(precision=FP64)
        assert g.setMoleculeBatch(mols), g.getErrorMessage()
        assert g.batchKernel() == ("cholesky" if direct else "cg")
        out.append(g.calculateEnergyBatch())
    (e0, s0), (e1, s1) = out
    assert (s0 == s1).all()
    assert s0[0] == 0 and s0[2] == 0
    assert np.abs(e0 - e1).max() < 1e-9


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("setup_bond", [0.471, 0.74])
def test_indefinite_with_a_symmetric_right_hand_side(setup_bond, precision, monkeypatch):
    """H2 at 0.471 A: one unknown, a negative matrix and a right-hand side of zero; four of them on
    the corners of a square (tilted, so that the matrix has no zeros) have right-hand sides without
    the antisymmetric modes.  Both are not positive definite whatever the right-hand side, as the
    Cholesky kernel says, and whichever molecules they are evaluated with."""
    z = np.array([1, 1], dtype=np.int32)

    def square(bond):
        u = bond / 2 * np.array([0.6, 0.8, 0.0])
        v = bond / 2 * np.array([-0.8, 0.6, 0.0])
        c = 4.0 * np.array([[1, 0, 0], [0, 1, 0], [-1, 0, 0], [0, -1, 0]])
        return np.concatenate([np.stack([c[k] - (v if k % 2 else u), c[k] + (v if k % 2 else u)]) for k in range(4)])

    def mols(bond):
        return [workloads.alkane(8, 1), (z, np.array([[0.0, 0, 0], [bond, 0, 0]])),
                (np.tile(z, 4), square(bond)), workloads.alkane(50, 2)]

    for direct in (False, True):
        if direct:
            monkeypatch.setenv("GFNFF_BATCH_TC", "0")
        g = GFNFF(precision=precision)
        assert g.setMoleculeBatch(mols(setup_bond)), g.getErrorMessage()
        g.updateGeometry(np.concatenate([x for _, x in mols(0.471)]))
        e, st = g.calculateEnergyBatch()
        assert list(st) == [0, 3, 3, 0], (direct, st)   # 3: GFNFF_NOT_SPD
        g.updateGeometry(np.concatenate([x for _, x in mols(0.74)]))   # and definite here
        e, st = g.calculateEnergyBatch()
        assert (st == 0).all(), (direct, st)
        assert np.abs(g.getCharges()[26:28]).max() == 0.0


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_coordinate_that_is_not_a_number(precision, monkeypatch):
    """Through the device entry point, which cannot look at its coordinates: the molecule's matrix holds
    NaN, and it gets the status that the Cholesky kernel gives it; its neighbours are not touched."""
    import torch

    mols = [workloads.alkane(8, 1), workloads.alkane(20, 3), workloads.alkane(50, 2)]
    x = np.concatenate([x for _, x in mols]) / 0.529177210903
    x[30, 1] = np.nan
    d_x = torch.from_numpy(x).cuda()
    for direct in (False, True):
        if direct:
            monkeypatch.setenv("GFNFF_BATCH_TC", "0")
        g = GFNFF(precision=precision)
        assert g.setMoleculeBatch(mols), g.getErrorMessage()
        e, _ = g.calculateEnergyBatch()
        d_e = torch.zeros(3, dtype=torch.float64, device="cuda")
        d_st = torch.full((3,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        st = _lib.load().gfnff_energy_and_gradient_device(g.handle, d_x.data_ptr(), d_e.data_ptr(), None,
                                                          d_st.data_ptr())
        assert st == 0
        torch.cuda.synchronize()
        assert d_st.tolist() == [0, 3, 0], (direct, d_st.tolist())
        assert abs(float(d_e[0]) - e[0]) < 1e-9 and abs(float(d_e[2]) - e[2]) < 1e-9


def _near_singular(bond):
    """H2 between two waters: positive definite from a bond of 0.527 A on"""
    w = workloads.water_geometry()
    w = w - w[0]
    z = np.array([1, 1, 8, 1, 1, 8, 1, 1], dtype=np.int32)
    h2 = np.array([[0.0, -bond / 2, 0.0], [0.0, bond / 2, 0.0]])
    return z, np.concatenate([h2, w + np.array([2.9, 0.3, 0.1]), w + np.array([-2.9, 0.7, 1.1])])


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_nearly_singular_matrix_on_the_device_entry(precision, monkeypatch):
    """A matrix that the Cholesky kernel still factorises gets status 0 where nothing on the host can
    evaluate it again.  One eigenvalue l is almost 0: E ~ -b^2 / (2 l), so an error of some 1e-15 in M
    (its elements are of order 1) shows as 1e-15 / l = 1e-15 * 2 |E| / b^2 of E; b^2 > 1e-5 here."""
    import torch

    lib = _lib.load()
    d_e = torch.zeros(1, dtype=torch.float64, device="cuda")
    d_st = torch.full((1,), -1, dtype=torch.int32, device="cuda")

    def handle(solver):
        monkeypatch.setenv("GFNFF_EEQ_SOLVER", solver)
        g = GFNFF(precision=precision)
        assert g.setMolecule(*_near_singular(0.74)), g.getErrorMessage()
        assert g.eeqSolver() == solver
        return g

    def evaluate(g, bond):
        d_x = torch.from_numpy(_near_singular(bond)[1] / 0.529177210903).cuda()
        torch.cuda.synchronize()
        assert lib.gfnff_energy_and_gradient_device(g.handle, d_x.data_ptr(), d_e.data_ptr(), None,
                                                    d_st.data_ptr()) == 0
        torch.cuda.synchronize()
        return int(d_st[0]), float(d_e[0])

    tiled, cg = handle("tiled"), handle("batched")
    lo, hi = 0.471, 0.74
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (lo, mid) if evaluate(tiled, mid)[0] == 0 else (mid, hi)
    for d in (1e-11, 1e-10, 1e-9, 1e-8, 1e-6, 1e-4, 1e-2):
        (s0, e0), (s1, e1) = evaluate(tiled, hi + d), evaluate(cg, hi + d)
        assert (s0, s1) == (0, 0), (d, s0, s1)
        assert abs(e1 - e0) < 1e-10 * e0 * e0 + 1e-9, (d, e0, e1)
    for d in (1e-9, 1e-6, 1e-2):
        assert evaluate(tiled, lo - d)[0] == evaluate(cg, lo - d)[0] == 3


def test_mixed_charges_end_far_below_the_bar(monkeypatch):
    """The same right-hand sides solved by the FP64 Cholesky kernels: the recurrence ends at a residual
    of 1e-14, so the charges agree to 1e-14 sqrt(n) / l_min < 2e-12 (n <= 300, smallest eigenvalue
    >= 0.1); a solve that stops at the bar of 1e-10 is 1e-10 off."""
    def perturbed(mols):
        x = np.concatenate([x for _, x in mols])
        return x + np.random.default_rng(1).normal(scale=0.03, size=x.shape)

    for mols in (workloads.conformer_batch(24, 7), [workloads.water_cluster(k, k) for k in (3, 10, 30, 60)]):
        q = []
        for direct in (False, True):
            monkeypatch.setenv("GFNFF_BATCH_TC", "0") if direct else monkeypatch.delenv("GFNFF_BATCH_TC", False)
            g = GFNFF(precision=MIXED)
            assert g.setMoleculeBatch(mols), g.getErrorMessage()
            g.updateGeometry(perturbed(mols))
            assert (g.calculateEnergyBatch()[1] == 0).all()
            q.append(g.getCharges().copy())
        assert np.abs(q[0] - q[1]).max() < 2e-12
    for mol in (workloads.alkane(8, 8), workloads.alkane(100, 1)):
        q = []
        for solver in ("batched", "tiled"):
            monkeypatch.setenv("GFNFF_EEQ_SOLVER", solver)
            g = GFNFF(precision=MIXED)
            assert g.setMolecule(*mol), g.getErrorMessage()
            g.updateGeometry(perturbed([mol]))
            g.calculateEnergy(True)
            assert not g.hasError() and g.eeqSolver() == solver
            q.append(g.getCharges().copy())
        assert np.abs(q[0] - q[1]).max() < 2e-12


@pytest.mark.parametrize("solver", ["tiled", "pcg", "batched"])
def test_fragments_whose_squared_distance_overflows(solver, monkeypatch):
    """Two flat waters, one 1e160 A away along its normal: no interaction, elements 1/r = 0.  Energy and
    gradient are those at 1e6 A (device entry; the host entry would look for a new topology)."""
    import torch

    w = workloads.water_geometry()
    w = w - w[0]
    flat = np.stack([np.zeros(3), w[:, 0], w[:, 1]], axis=1)

    def waters(dx):
        return np.concatenate([flat, flat + np.array([dx, 0.0, 0.0])])

    monkeypatch.setenv("GFNFF_EEQ_SOLVER", solver)
    g = GFNFF(precision=FP64)
    assert g.setMolecule(np.array([8, 1, 1, 8, 1, 1], dtype=np.int32), waters(4.0)), g.getErrorMessage()
    assert g.eeqSolver() == solver
    out = []
    for dx in (1e6, 1e160):
        d_x = torch.from_numpy(waters(dx) / 0.529177210903).cuda()
        d_e = torch.zeros(1, dtype=torch.float64, device="cuda")
        d_g = torch.zeros(d_x.shape, dtype=torch.float64, device="cuda")
        d_st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert _lib.load().gfnff_energy_and_gradient_device(g.handle, d_x.data_ptr(), d_e.data_ptr(), d_g.data_ptr(),
                                                            d_st.data_ptr()) == 0
        torch.cuda.synchronize()
        assert int(d_st[0]) == 0
        out.append((float(d_e[0]), d_g.cpu().numpy()))
    assert abs(out[0][0] - out[1][0]) < 1e-6    # 1 / (1e6 A) per pair of charges at most
    assert np.abs(out[0][1] - out[1][1]).max() < 1e-6


@pytest.mark.parametrize("nc", [8, 30, 64])
@pytest.mark.parametrize("angle", [0.5, 1.5])
def test_chain_bent_far_from_its_setup(nc, angle, monkeypatch):
    """One half of a chain turned about its middle: the set-up inverse is no longer that of the matrix, by
    many Angstrom at the ends (device entry: no topology refresh).  Against the oracle at that geometry;
    the products stay below those after which the solve is left to the elimination."""
    import torch

    monkeypatch.setenv("GFNFF_EEQ_SOLVER", "batched")
    Z, X = workloads.alkane(nc, nc)
    axis = int(np.argmax(np.ptp(X, axis=0)))
    other = (axis + 1) % 3
    c = X.mean(axis=0)
    turn = np.eye(3)
    turn[axis, axis] = turn[other, other] = np.cos(angle)
    turn[other, axis], turn[axis, other] = np.sin(angle), -np.sin(angle)
    x = X.copy()
    half = X[:, axis] > c[axis]
    x[half] = (X[half] - c) @ turn.T + c
    g = GFNFF(precision=FP64)
    assert g.setMolecule(Z, X), g.getErrorMessage()
    d_x = torch.from_numpy(x / 0.529177210903).cuda()
    d_e = torch.zeros(1, dtype=torch.float64, device="cuda")
    d_g = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    d_st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert _lib.load().gfnff_energy_and_gradient_device(g.handle, d_x.data_ptr(), d_e.data_ptr(), d_g.data_ptr(),
                                                        d_st.data_ptr()) == 0
    torch.cuda.synchronize()
    assert int(d_st[0]) == 0
    T, G, q, cn = Oracle(Z, X).engrad(x)
    scale = max(1.0, np.abs(G).max())   # atoms near the hinge come close
    assert abs(float(d_e[0]) - T["total"]) < 1e-9 * max(1.0, abs(T["total"]))
    assert np.abs(d_g.cpu().numpy() - G).max() < 1e-9 * scale
    assert np.abs(g.getCharges() - q).max() < 1e-10
    assert g.eeqIterations() < 20 + 2 * (len(Z) - 1) // 5, g.eeqIterations()
