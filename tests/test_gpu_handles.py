"""Several handles in one process: the launch limits of a kernel belong to the process, so a
handle set up later for a smaller system must not take them from an earlier, larger one."""
import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, MIXED, workloads
from tests.oracle_api import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["pipelined", "classic"])
@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_larger_handle_after_smaller_setup(precision, form, monkeypatch):
    monkeypatch.setenv("GFNFF_EEQ_SOLVER", "pcg")
    monkeypatch.setenv("GFNFF_PCG", form)
    Z, X = workloads.water_cluster(150, 5)
    large, small = GFNFF(precision=precision), GFNFF(precision=precision)
    assert large.setMolecule(Z, X), large.getErrorMessage()
    assert small.setMolecule(Z[:30], X[:30]), small.getErrorMessage()
    e = large.calculateEnergy(True)
    assert not large.hasError(), large.getErrorMessage()
    T, G, q, cn = Oracle(Z, X).engrad(X)
    assert abs(e - T["total"]) < 1e-6
    assert np.abs(large.getGradient() - G).max() < 1e-6
