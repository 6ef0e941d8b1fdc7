"""A coordinate that is not a number shows in the forces of its batched box and of no
other, with short-range pairs alone (no reciprocal sum that would carry it) and
with charges."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import BatchEngine
from mdff_b200.params import params_copy

from .gpu_util import forces

pytestmark = pytest.mark.gpu

LJ = dict(lcoulomb=0, lbmhft=0, lnmlj=1, trunc=1, epslj={(0, 0): 0.01, (0, 1): 0.02, (1, 1): 0.015},
          sigmalj={(0, 0): 2.0, (0, 1): 2.2, (1, 1): 2.6}, qlj={(0, 0): 12.0, (0, 1): 12.0, (1, 1): 12.0},
          plj={(0, 0): 6.0, (0, 1): 6.0, (1, 1): 6.0})


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("kind", ["bmh", "lj", "charges"])
@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED])
def test_bad_coordinate(kind, bad, precision):
    kw = dict(bmh=dict(lcoulomb=0), lj=LJ, charges={})[kind]
    s = systems.random_ionic((20, 21), L=13.0, seed=3, pol=(0.0, 0.0), **kw)
    psets, configs = [], []
    for k in range(2):
        p = params_copy(s.params)
        p.calc, p.precision, p.solver = _abi.CALC_OTHER, precision, _abi.SOLVER_CG
        psets.append(p)
        configs.append((k, [p.natmi[t] for t in range(p.ntype)], s.cell))
    P = np.concatenate([s.pos, s.pos])
    n = s.natm
    with BatchEngine(psets, configs) as eng:
        good = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
        P[7, 1] = bad
        f = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
    assert np.isnan(f[7]).all()
    assert np.isnan(f[:n]).any(axis=1).all()  # every ion meets it: the pair is within no cutoff and beyond none
    assert np.array_equal(f[n:], good[n:])
