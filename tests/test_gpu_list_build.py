"""Verlet-list build at the edges of its FP32 decision and its bitmaps.

Rows are decided in FP32 except within the rounding margin of the cutoff and of
an ambiguous image, and read off a bitmap of the ions in ascending order.  Lattices put
whole shells of pairs exactly at the cutoff and exactly half a box apart, coordinates lie
several cells outside the box, ion counts are off the bitmap's words: the half list must
equal the oracle's (the reference's arithmetic) entry by entry."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

pytestmark = pytest.mark.gpu


def _lattice(n, a, shift, tri):
    """n^3 sites of spacing a (simple cubic, optionally sheared), shifted by whole cells"""
    s = systems.random_ionic((n ** 3 // 2, n ** 3 - n ** 3 // 2), L=n * a, seed=1, calc=_abi.CALC_OTHER)
    g = np.arange(n) / n
    f = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    cell = np.array(s.cell, dtype=float).reshape(3, 3).copy()
    if tri:
        cell = cell + n * a * np.array([[0, 0.25, 0], [0, 0, 0.125], [0, 0, 0]])
    rng = np.random.default_rng(3)
    f = f + shift * rng.integers(-3, 4, f.shape)
    return s, cell, f @ cell.T


@pytest.mark.parametrize("n,mult,shift,tri", [(4, 2.0, 0, False), (5, 2.0, 1, False), (6, 2.0, 1, True),
                                              (7, 3.0, 0, False), (9, 2.0, 1, False), (11, 2.5, 1, True)])
def test_shells_at_the_cutoff(oracle, n, mult, shift, tri):
    a = 3.0
    s, cell, pos = _lattice(n, a, shift, tri)
    p = params_copy(s.params)
    p.skindiff = 0.5
    p.cutlongrange = min(mult * a, 0.5 * n * a) - p.skindiff  # list cutoff: on a shell (or half the box)
    p.cutshortrange = p.cutlongrange
    xyz = tuple(np.ascontiguousarray(pos[:, k]) for k in range(3))
    orc = oracle.Oracle(params_copy(p), cell)
    with ForceEngine(p, cell) as eng:
        for which in (0, 1):
            so, po, lo, no = orc.vnlist(*xyz, which=which)
            sg, pg, lg, ng = eng.verlet_half_list(*xyz, which=which)
            assert (so, no) == (sg, ng)
            assert np.array_equal(po, pg)
            assert np.array_equal(lo[:no], lg[:ng])


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED])
def test_handles_with_different_meshes_side_by_side(precision):
    # shared-memory limits belong to the kernels, not to the handle made last
    big = systems.mgo(ncell=3, kmax=16, calc=_abi.CALC_OTHER)
    small = systems.mgo(ncell=2, kmax=3, calc=_abi.CALC_OTHER)

    def eng(s):
        p = params_copy(s.params)
        p.precision, p.solver = precision, _abi.SOLVER_CG
        return ForceEngine(p, s.cell)

    with eng(big) as e:
        want = e.engforce(*big.soa())
    with eng(big) as e, eng(small) as f:
        f.engforce(*small.soa())
        got = e.engforce(*big.soa())
        f.engforce(*small.soa())
    assert np.array_equal(want["fx"], got["fx"])
