"""FP64 structure factor over many ion chunks, all ions and a polarisable subset of
other chunk counts, against the CPU oracle.

Silica, O polarisable (two thirds of the ions), 148 SMs: 1188 ions at kmax 10 are 30
chunks and their 792 dipoles 33; kmax 16 has 15 and 15, several stagings each; kmax 22
has 4 and 4 in two passes over nz (summed by the thread-per-k kernel).  Two SCF solves of
the same iteration count 1e-10, two CG solves at 1e-12 1e-9."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

from .gpu_util import compare

pytestmark = pytest.mark.gpu


def _system(kmax, **kw):
    return systems.sio2(nsio2=396, seed=31, rcut=9.0, alpha=0.35, kmax=kmax, calc=_abi.CALC_OTHER, **kw)


@pytest.mark.parametrize("kmax", [10, 16, 22])
def test_scf(oracle, kmax):
    s = _system(kmax)
    o = oracle.Oracle(s.params, s.cell).engforce(*s.soa(), efg=True)
    with ForceEngine(params_copy(s.params), s.cell) as eng:
        for call in range(2):  # the launch-by-launch call, then the whole-step graph
            g = eng.engforce(*s.soa())
            compare(g, o, 1e-10)
            assert eng.stats()["n_pol_iter"] == o["n_scf"]
        e = eng.efg()
    assert np.abs(e - o["efg"]).max() <= 1e-10 * np.abs(o["efg"]).max()


def test_cg(oracle):
    s = _system(10)
    p = params_copy(s.params)
    p.conv_tol_ind = 1e-12
    p.max_scf_pol_iter = 1000
    o = oracle.Oracle(p, s.cell).engforce(*s.soa())
    p.solver = _abi.SOLVER_CG
    p.cg_tol = 1e-12
    with ForceEngine(p, s.cell) as eng:
        compare(eng.engforce(*s.soa()), o, 1e-9)
