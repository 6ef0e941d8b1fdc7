"""Tensor-core field kernel of the mixed engine at the edges of its tiles.

2 (kz + 1) features are rounded up to 16, 24, 32, 40, 48 or 64, a CTA takes 128
ions and a group of tiles of 32 (16 with dipole forces) mesh rows: kz on both
sides of every rounding, meshes of a few and of many rows (one, two and more
tiles per CTA), ion counts off the tile.  Against the same engine on the
CUDA-core kernels, tolerances as the other tensor-core operator test (the dipole
solve at 1e-10, FP32 sums: 2e-6)."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

from .gpu_util import forces, rms_rel

pytestmark = pytest.mark.gpu


def _run(s, tc, monkeypatch):
    monkeypatch.setenv("MDFF_REC_TC", "1" if tc else "0")
    monkeypatch.setenv("MDFF_FIELD_TC", "1" if tc else "0")
    p = params_copy(s.params)
    p.solver, p.cg_tol, p.precision = _abi.SOLVER_CG, 1e-10, _abi.PREC_MIXED
    with ForceEngine(p, s.cell) as eng:
        r = eng.engforce(*s.soa())
        assert eng.stats()["converged"]
    return r


@pytest.mark.parametrize("mesh", [(2, 2, 1), (1, 3, 7), (4, 4, 8), (3, 5, 11), (4, 3, 12), (3, 3, 15), (5, 4, 16),
                                  (3, 3, 19), (2, 4, 20), (3, 2, 23), (2, 3, 24), (2, 2, 31)])
def test_feature_counts(mesh, monkeypatch):
    s = systems.random_ionic((33, 32), L=14.0, seed=71, kES=mesh, calc=_abi.CALC_OTHER)
    a, b = _run(s, True, monkeypatch), _run(s, False, monkeypatch)
    assert rms_rel(forces(a), forces(b)) <= 2e-6
    assert rms_rel(a["mu"], b["mu"]) <= 2e-6


@pytest.mark.parametrize("ncell,kmax", [(5, 9), (6, 13), (9, 6)])
def test_row_groups(ncell, kmax, monkeypatch):
    s = systems.mgo(ncell=ncell, kmax=kmax, jitter=0.15, rcut=6.0, alpha=0.5, calc=_abi.CALC_OTHER)
    a, b = _run(s, True, monkeypatch), _run(s, False, monkeypatch)
    assert rms_rel(forces(a), forces(b)) <= 2e-6
    assert rms_rel(a["mu"], b["mu"]) <= 2e-6
