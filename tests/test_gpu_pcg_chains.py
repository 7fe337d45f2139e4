"""Conjugate gradients of large systems of long chains: the preconditioner takes whole fragments (512
unknowns at most), whose rows one grid block owns, and still has to fit into shared memory.

Tolerances: both forms are accepted on their true FP64 residual (1e-12 of the right-hand side; 1e-10), so
energies agree to the FP32 coordination numbers of the mixed form (some 1e-9 of 1 Eh per atom of a
chain; 1e-6 is the mixed form's bar), gradients to 1e-5 (the same)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from curcuma_b200 import FP64, GFNFF, MIXED, workloads
from tests.oracle_api import Oracle

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


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


@pytest.mark.parametrize("nc", [11, 12, 21, 22, 43, 170])   # 34, 37, 64, 67, 130, 511 unknowns
def test_inverse_of_a_whole_chain(nc, monkeypatch):
    """One fragment is one block: its inverse solves the set-up geometry in one product and the check of the
    true residual (two where rounding leaves more than 1e-12 of the right-hand side)."""
    monkeypatch.setenv("GFNFF_EEQ_SOLVER", "pcg")
    Z, X = workloads.alkane(nc, nc)
    g = GFNFF(precision=FP64)
    assert g.setMolecule(Z, X), g.getErrorMessage()
    assert g.eeqSolver() == "pcg"
    e = g.calculateEnergy(True)
    assert not g.hasError(), g.getErrorMessage()
    assert g.eeqIterations() <= 2
    T, G, q, cn = Oracle(Z, X).engrad(X)
    assert abs(e - T["total"]) < 1e-8
    assert np.abs(g.getCharges() - q).max() < 1e-9


def test_setup_of_long_chains_is_not_serial():
    """The inverses of whole chains are formed on the device: on one host thread, where a host
    inversion is at its slowest (2.5e9 multiply-adds here), set-up takes no longer than with blocks of
    128 unknowns, but for noise."""
    code = ("import time; from tests.test_gpu_pcg_chains import rods; from curcuma_b200 import GFNFF\n"
            "Z, X = rods(8)\n"
            "t = []\n"
            "for _ in range(3):\n"
            "    g = GFNFF(); t0 = time.perf_counter(); assert g.setMolecule(Z, X); t.append(time.perf_counter() - t0)\n"
            "    assert g.eeqSolver() == 'pcg'; g.close()\n"
            "print(min(t))")
    t = []
    for block in ("128", "512"):
        env = dict(os.environ, OMP_NUM_THREADS="1", GFNFF_PCG_PREBLK=block, GFNFF_EEQ_SOLVER="pcg")
        p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr
        t.append(float(p.stdout.split()[-1]))
    assert t[1] < 1.3 * t[0] + 0.1, t
