"""Reciprocal tiles, partner lists and pair cache of the batched engine at the
edges of their ranges, against the CPU oracle.

The structure factor runs on groups of 8 mesh rows by tiles of 4 values of nz
and steps of 4 ions, the field on 16 ions, steps of 2 nz and 4 rows, both from
a staging buffer: meshes from one k vector per row to more row groups than
warps, nz counts on both sides of every tile, ion counts that are not
multiples of a step, a box whose weights do not fit the buffer on one CTA, and
a short-range cutoff beyond half the box.  FP64 tolerance: two dipole solves at
1e-12, 1e-9 as the other batch tests; mixed: the 1e-5 force bar."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import BatchEngine
from mdff_b200.params import params_copy

from .gpu_util import compare, forces, rms_rel

pytestmark = pytest.mark.gpu

MESHES = [(1, 1, 0), (2, 3, 1), (3, 2, 5), (5, 6, 6), (7, 5, 7), (6, 8, 8), (9, 4, 9), (4, 5, 10), (5, 3, 12),
          (16, 18, 3)]


def _evaluate(syslist, precision, shape):
    psets, configs, pos = [], [], []
    for k, s in enumerate(syslist):
        p = params_copy(s.params)
        p.conv_tol_ind = p.cg_tol = 1e-12 if precision == _abi.PREC_FP64 else 1e-9
        p.max_scf_pol_iter = p.cg_max_iter = 2000
        p.calc = _abi.CALC_OTHER
        p.precision = precision
        p.solver = _abi.SOLVER_CG
        psets.append(p)
        configs.append((k, [p.natmi[t] for t in range(p.ntype)], s.cell))
        pos.append(s.pos)
    with BatchEngine(psets, configs) as eng:
        eng.set_shape(*shape)
        P = np.concatenate(pos)
        out = eng.engforce(P[:, 0], P[:, 1], P[:, 2])
        res = []
        for c in range(eng.nconf):
            a, b = eng.offsets[c], eng.offsets[c + 1]
            d = {k: out[k][a:b] for k in ("fx", "fy", "fz", "mu", "ef")}
            d.update(out["conf"][c])
            res.append(d)
    return res


def _oracle(oracle, s):
    p = params_copy(s.params)
    p.conv_tol_ind = 1e-12
    p.max_scf_pol_iter = 2000
    p.calc = _abi.CALC_OTHER
    return oracle.Oracle(p, s.cell).engforce(*s.soa())


@pytest.mark.parametrize("shape", [(1, 256), (4, 512)])
@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED])
def test_mesh_tiles(oracle, shape, precision):
    syslist = [systems.random_ionic((17, 20), L=13.0, seed=40 + k, kES=m, triclinic=k % 2 == 1,
                                    cutshortrange=9.0 if k == 3 else 5.5, lsurf=1 if k == 4 else 0,
                                    dip={(0, 1): 0.3} if k == 5 else None)
               for k, m in enumerate(MESHES)]
    res = _evaluate(syslist, precision, shape)
    for s, r in zip(syslist, res):
        o = _oracle(oracle, s)
        if precision == _abi.PREC_FP64:
            compare(r, o, 1e-9)
        else:
            assert rms_rel(forces(r), forces(o)) < 1e-5


@pytest.mark.parametrize("shape", [(1, 512), (8, 256)])
def test_more_ions_than_the_staging_buffer(oracle, shape):
    s = systems.mgo(ncell=5, jitter=0.15, rcut=7.0, alpha=0.45, kmax=7)  # 1000 ions, 500 polarisable
    res = _evaluate([s], _abi.PREC_FP64, shape)
    compare(res[0], _oracle(oracle, s), 1e-9)
