"""The set-up autotuner of the Coulomb + D4 pair kernel: every variant it chooses from gives
the same energy and gradient (each pair's arithmetic is the same; only the summation order
differs), and the pick is one of them.  Single molecule (1000 waters) and a conformer batch,
both precision forms."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, MIXED, workloads

pytestmark = pytest.mark.gpu

VARIANTS = ["sym32", "sym64", "sym64_occ10", "rows"]


def _run(mols, precision, monkeypatch, variant=None):
    if variant:
        monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
    else:
        monkeypatch.delenv("GFNFF_PAIRS_VARIANT", raising=False)
    g = GFNFF(precision=precision)
    if len(mols) == 1:
        assert g.setMolecule(*mols[0]), g.getErrorMessage()
        e = np.array([g.calculateEnergy(True)])
    else:
        assert g.setMoleculeBatch(mols), g.getErrorMessage()
        e, st = g.calculateEnergyBatch()
        assert (st == 0).all()
    assert not g.hasError(), g.getErrorMessage()
    return g.pairKernel(), e, g.getGradient()


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("system", ["water1000", "batch24"])
def test_variants_agree_and_tuner_picks_one(system, precision, monkeypatch):
    mols = ([workloads.water_cluster(1000, 1002)] if system == "water1000"
            else workloads.conformer_batch(24, 17, lo=20, hi=200))
    pick, e0, g0 = _run(mols, precision, monkeypatch)
    assert pick in VARIANTS
    for v in VARIANTS:
        name, e, g = _run(mols, precision, monkeypatch, v)
        assert name == v
        assert np.abs(e - e0).max() < 1e-9, (v, e - e0)
        assert np.abs(g - g0).max() < 1e-9, v


def test_only_the_lists_of_the_pick_are_kept(monkeypatch):
    """14,739 atoms: the 32 x 16 tiles are 0.21 million, 3.4 MB; "rows" needs none.  The device's free memory
    counts in steps of 2 MB."""
    import torch

    monkeypatch.setenv("GFNFF_EEQ_SOLVER", "pcg")
    m = 17
    site = 3.1 * np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), axis=-1).reshape(-1, 1, 3)
    X = (site + workloads.water_geometry()[None]).reshape(-1, 3)
    Z = np.tile(np.array([8, 1, 1], dtype=np.int32), m ** 3)
    used = {}
    for variant in ("rows", "rows", "sym32"):   # the first run also loads the kernels
        monkeypatch.setenv("GFNFF_PAIRS_VARIANT", variant)
        free0 = torch.cuda.mem_get_info()[0]
        g = GFNFF(precision=FP64)
        assert g.setMolecule(Z, X), g.getErrorMessage()
        assert g.calculateEnergy(True) != 0.0
        used[variant] = free0 - torch.cuda.mem_get_info()[0]
        g.close()
    assert used["sym32"] - used["rows"] >= 2 << 20, used
