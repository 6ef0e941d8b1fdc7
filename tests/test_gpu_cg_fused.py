"""Vector kernels of the CG iteration that take the operator's parts directly.

With MDFF_OVERLAP=0 the mixed engine forms the operator as a field and runs the
general vector kernels; the default takes k_cg_q / k_cg_step / k_cg_next.  Both
solve to 1e-10: dipoles and forces agree to 2e-6 (the FP32 operator and force pass
of the other operator tests).  Boxes with one ion per thread and more, fewer ions than a
block, all ions and some ions polarisable, a surface term, MD (the accumulated
structure factor) and single calls.  FP64: against the SCF solver at 1e-12, the
fixed point is the same, 1e-8."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

from .gpu_util import forces, rms_rel

pytestmark = pytest.mark.gpu


def _boxes():
    return {
        "few": systems.random_ionic((5, 4), L=9.0, seed=5, calc=_abi.CALC_OTHER),
        "some": systems.random_ionic((20, 30, 20), L=13.0, seed=18, q=(-1.5, 2.0, -1.5), pol=(1.1, 0.0, 1.1),
                                     calc=_abi.CALC_OTHER),
        "surface": systems.random_ionic((24, 24), L=13.0, seed=52, lsurf=1, calc=_abi.CALC_OTHER),
        "md": systems.sio2(nsio2=300, seed=10, calc=_abi.CALC_MD),
        "many": systems.mgo(ncell=17, jitter=0.15, rcut=5.0, alpha=0.6, kmax=6, calc=_abi.CALC_OTHER),
    }


def _run(s, precision, solver, tol):
    p = params_copy(s.params)
    p.solver, p.cg_tol, p.conv_tol_ind, p.precision = solver, tol, tol, precision
    p.max_scf_pol_iter = 2000
    with ForceEngine(p, s.cell) as eng:
        r = eng.engforce(*s.soa())
        assert eng.stats()["converged"]
    return r


@pytest.mark.parametrize("name", ["few", "some", "surface", "md", "many"])
def test_mixed_iteration(name, monkeypatch):
    s = _boxes()[name]
    a = _run(s, _abi.PREC_MIXED, _abi.SOLVER_CG, 1e-10)
    monkeypatch.setenv("MDFF_OVERLAP", "0")
    b = _run(s, _abi.PREC_MIXED, _abi.SOLVER_CG, 1e-10)
    assert rms_rel(a["mu"], b["mu"]) <= 2e-6
    assert rms_rel(forces(a), forces(b)) <= 2e-6


@pytest.mark.parametrize("name", ["few", "some", "surface"])
def test_fp64_iteration(name):
    s = _boxes()[name]
    a = _run(s, _abi.PREC_FP64, _abi.SOLVER_CG, 1e-12)
    b = _run(s, _abi.PREC_FP64, _abi.SOLVER_SCF, 1e-12)
    assert rms_rel(a["mu"], b["mu"]) <= 1e-8
    assert rms_rel(forces(a), forces(b)) <= 1e-8
