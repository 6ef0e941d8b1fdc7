"""Real-space cutoff of the batched force pass: the exact FP64 decision in both engines.

Two ions at distances within 1e-9 of the cutoff, where the Ewald real-space force is still a
sizeable part of the whole (alpha rc = 0.6): a pair taken or left out by an FP32 distance would
change the force by a tenth.  Forces and energy against the oracle, FP64 1e-10,
mixed the 1e-5 force bar."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import BatchEngine
from mdff_b200.params import params_copy

from .gpu_util import forces, rms_rel

pytestmark = pytest.mark.gpu

RC = 5.0


@pytest.mark.parametrize("precision,tol", [(_abi.PREC_FP64, 1e-10), (_abi.PREC_MIXED, 1e-5)])
def test_pairs_at_the_cutoff(oracle, precision, tol):
    s = systems.random_ionic((1, 1), L=13.0, seed=3, pol=(0.0, 0.0), lbmhft=0, alphaES=0.12, kES=(4, 4, 4),
                             cutlongrange=RC, cutshortrange=RC)
    rng = np.random.default_rng(8)
    psets, configs, pos = [], [], []
    for k in range(60):
        u = rng.standard_normal(3)
        a = rng.uniform(0.0, 13.0, 3)
        d = RC * (1.0 + (1e-9 if k % 2 else -1e-9))
        pos.append(np.array([a, a + d * u / np.linalg.norm(u)]))
        p = params_copy(s.params)
        p.calc, p.precision, p.solver = _abi.CALC_OTHER, precision, _abi.SOLVER_CG
        psets.append(p)
        configs.append((k, [1, 1], s.cell))
    P = np.concatenate(pos)
    with BatchEngine(psets, configs) as eng:
        out = eng.engforce(P[:, 0], P[:, 1], P[:, 2])
    orc = oracle.Oracle(psets[0], s.cell)
    mags = []
    for k, x in enumerate(pos):
        o = orc.engforce(*(np.ascontiguousarray(x[:, c]) for c in range(3)))
        f = {c: out[c][2 * k:2 * k + 2] for c in ("fx", "fy", "fz")}
        assert rms_rel(forces(f), forces(o)) <= tol, k
        mags.append(np.linalg.norm(forces(o)[0]))
    assert min(mags[0::2]) > 1.05 * max(mags[1::2]) or max(mags[0::2]) < 0.95 * min(mags[1::2])
