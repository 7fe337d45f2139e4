"""The tiled Coulomb and D4 pair kernels at the edges of their tiles (32 rows, 8 partners a step,
16 to 64 partners a tile), against the oracle: sizes around the multiples, every tile shape, a
geometry translated far from the set-up, and one where D4 pairs of the evaluated geometry are not on
the set-up list (distances up to 60 bohr there).

Tolerances: both sides sum FP64 terms of at most ~1 Eh over n^2 / 2 < 1e4 pairs (rounding below
1e-12); the charges are solved to a residual of 1e-12 of the right-hand side, which moves the
energies by its square and the gradient by about 1e-12."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, _lib, workloads
from tests.oracle_api import Oracle

pytestmark = pytest.mark.gpu

VARIANTS = ["sym32", "sym64", "sym64_occ10"]


def _compare(Z, X, variant, monkeypatch):
    monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
    g = GFNFF(precision=FP64)
    assert g.setMolecule(Z, X), g.getErrorMessage()
    e = g.calculateEnergy(True)
    assert not g.hasError(), g.getErrorMessage()
    T, G, q, cn = Oracle(Z, X).engrad(X)
    D = g.getEnergyDecomposition()
    assert abs(D["coulomb"] - T["coulomb"]) < 1e-10
    assert abs(D["dispersion"] - T["dispersion"]) < 1e-10
    assert abs(e - T["total"]) < 1e-10
    assert np.abs(g.getGradient() - G).max() < 1e-10
    return g, e


@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("n_water", [1, 5, 10, 11, 21, 22, 43])   # 3 .. 129 atoms: 30|33, 63|66, 129
def test_tile_edges_water(n_water, variant, monkeypatch):
    _compare(*workloads.water_cluster(n_water, 100 + n_water), variant, monkeypatch)


@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("size", [24, 31, 40, 65, 97])   # C/H/N/O: 17 packed references
def test_tile_edges_chain(size, variant, monkeypatch):
    _compare(*workloads.random_chain(size, np.random.default_rng(size)), variant, monkeypatch)


def test_far_from_setup(monkeypatch):
    Z, X = workloads.water_cluster(20, 3)
    g, e = _compare(Z, X, "sym32", monkeypatch)
    g0 = g.getGradient()
    g.updateGeometry(X + np.array([4.0, -2.0, 1.0]))   # 7.6 bohr: beyond the free displacement
    assert abs(g.calculateEnergy(True) - e) < 1e-9
    assert np.abs(g.getGradient() - g0).max() < 1e-9


# largest coordinate change below and above 2.8 bohr, up to which no pair within 50 bohr can be off the
# list (50 + 2 sqrt(3) 2.8 < 60) and the kernels do not look; and far beyond it
@pytest.mark.parametrize("variant", VARIANTS + ["rows"])
@pytest.mark.parametrize("shift_bohr", [2.79, 2.81, 14.0, 22.0])
def test_d4_list_membership(shift_bohr, variant, monkeypatch):
    """Two water clusters 42 to 75 bohr apart at set-up, one moved towards the other: pairs that are now within
    50 bohr but were beyond 60 do not count (device entry: the host one would detect a new topology)."""
    import torch

    za, xa = workloads.water_cluster(12, 5)
    zb, xb = workloads.water_cluster(14, 6)
    Z = np.concatenate([za, zb])
    X = np.concatenate([xa - xa.mean(axis=0), xb - xb.mean(axis=0) + np.array([31.0, 0.0, 0.0])])
    x = X.copy()
    x[len(za):, 0] -= shift_bohr * 0.529177210903
    d0, d = (np.linalg.norm(y[:len(za), None] - y[None, len(za):], axis=-1) / 0.529177210903 for y in (X, x))
    excluded = int(((d0 > 60.0) & (d <= 50.0)).sum())
    assert (excluded > 0) == (shift_bohr > 10.0) and (d <= 50.0).sum() > 10
    monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
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
    # the excluded pairs (302 and 641) are 1.1e-7 and 5.1e-7 Eh, 1.2e-9 and 5.8e-9 Eh/bohr together
    assert abs(float(d_e[0]) - T["total"]) < 2e-12 * len(Z)
    assert np.abs(d_g.cpu().numpy() - G).max() < 1e-11


def test_batch_of_ragged_molecules(monkeypatch):
    rng = np.random.default_rng(8)
    mols = [workloads.random_chain(n, rng) for n in (20, 33, 64, 70)] + [workloads.water_cluster(1, 2)]
    for variant in VARIANTS:
        monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
        g = GFNFF(precision=FP64)
        assert g.setMoleculeBatch(mols), g.getErrorMessage()
        e, st = g.calculateEnergyBatch()
        assert (st == 0).all()
        G = np.split(g.getGradient(), np.cumsum([len(z) for z, _ in mols])[:-1])
        for (Z, X), em, gm in zip(mols, e, G):
            T, Go, q, cn = Oracle(Z, X).engrad(X)
            assert abs(em - T["total"]) < 1e-10
            assert np.abs(gm - Go).max() < 1e-10


def test_tiles_far_from_the_origin(monkeypatch):
    """800 bohr of waters (tiles of every distance) translated to 5e7 and 1e8 bohr: the tile kernels leave
    out no pair that the row kernel has.  Same coordinates, same charges: the energies (-130 Eh) differ
    by the order of summation, some 1e-11; the pairs that FP32 box gaps lose are 4e-10 to 1e-9."""
    import torch

    w = workloads.water_geometry()
    w = w - w[0]
    X = np.concatenate([w + 3.1 * np.array([k // 4, k % 4 // 2, k % 2]) for k in range(400)])
    Z = np.tile(np.array([8, 1, 1], dtype=np.int32), 400)
    lib = _lib.load()
    out = {}
    for variant in ["rows"] + VARIANTS:
        monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
        g = GFNFF(precision=FP64)
        assert g.setMolecule(Z, X), g.getErrorMessage()
        for shift in (3e7, 6e7):
            d_x = torch.from_numpy((X + shift) / 0.529177210903).cuda()
            d_e = torch.zeros(1, dtype=torch.float64, device="cuda")
            d_st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            assert lib.gfnff_energy_and_gradient_device(g.handle, d_x.data_ptr(), d_e.data_ptr(), None,
                                                        d_st.data_ptr()) == 0
            torch.cuda.synchronize()
            assert int(d_st[0]) == 0
            out[variant, shift] = float(d_e[0])
            assert abs(out[variant, shift] - out["rows", shift]) < 1e-10, (variant, shift)
