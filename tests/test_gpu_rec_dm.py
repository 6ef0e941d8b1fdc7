"""FP64 tensor-core reciprocal sums and the device SCF loop of the single engine at
the edges of their ranges, against the CPU oracle.

k_rho_dm takes 64 mesh rows a block, tiles of 4 values of nz (up to 5 tiles a
pass) and chunks of at least 16 ions; k_field_dm 128 ions a block, steps of 2 nz
(instantiated counts 3-9, 11, 13, 16, none beyond nz = 31) and 4 rows: meshes on
both sides of each, one that needs the smaller staging buffers, and one that
falls back to the recurrence kernels (rows of 600 ny).  Boxes with
polarisable and other ions, triclinic or cubic, with the surface term (host
SCF loop) and without (device loop).  Tolerances: two SCF solves of the same
iteration count 1e-10, two CG solves at 1e-12 1e-9, mixed the 1e-5 force bar."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

from .gpu_util import compare, forces, rms_rel

pytestmark = pytest.mark.gpu

MESHES = [(1, 1, 0), (2, 3, 3), (7, 7, 4), (3, 4, 7), (4, 2, 11), (5, 6, 12), (3, 3, 17), (2, 3, 19), (2, 2, 20),
          (1, 2, 23), (2, 1, 31), (1, 2, 32), (3, 90, 2), (0, 600, 1)]


def _system(k, mesh, **kw):
    # 23 + 37 ions, 37 polarisable; odd meshes in a triclinic box
    return systems.random_ionic((23, 37), L=15.0, seed=60 + k, kES=mesh, triclinic=k % 2 == 1, alphaES=0.35,
                                calc=_abi.CALC_OTHER, **kw)


@pytest.mark.parametrize("k", range(len(MESHES)), ids=[str(m) for m in MESHES])
def test_scf_and_field_gradient(oracle, k):
    s = _system(k, MESHES[k])
    o = oracle.Oracle(s.params, s.cell).engforce(*s.soa(), efg=True)
    with ForceEngine(params_copy(s.params), s.cell) as eng:
        for call in range(2):  # the launch-by-launch call, then the whole-step graph
            g = eng.engforce(*s.soa())
            compare(g, o, 1e-10)
            assert eng.stats()["n_pol_iter"] == o["n_scf"]
        e = eng.efg()
    assert np.abs(e - o["efg"]).max() <= 1e-10 * np.abs(o["efg"]).max()


@pytest.mark.parametrize("k", [2, 5, 8, 11])
@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED])
def test_cg(oracle, k, precision):
    s = _system(k, MESHES[k], lsurf=1 if k == 5 else 0)
    p = params_copy(s.params)
    p.conv_tol_ind = 1e-12
    p.max_scf_pol_iter = 1000
    o = oracle.Oracle(p, s.cell).engforce(*s.soa())
    p.solver = _abi.SOLVER_CG
    p.precision = precision
    p.cg_tol = 1e-12 if precision == _abi.PREC_FP64 else 1e-9
    with ForceEngine(p, s.cell) as eng:
        g = eng.engforce(*s.soa())
    if precision == _abi.PREC_FP64:
        compare(g, o, 1e-9)
    else:
        assert rms_rel(forces(g), forces(o)) < 1e-5


@pytest.mark.parametrize("limits", [(1, 1), (3, 2), (5, 100), (0, 4)])
def test_device_scf_loop_limits(oracle, limits):
    """min / max iterations of the reference's loop, ASPC sequence included."""
    mn, mx = limits
    s = _system(3, (5, 5, 5), extrapolate_order=2)
    s.params.calc = _abi.CALC_MD
    s.params.min_scf_pol_iter, s.params.max_scf_pol_iter = mn, mx
    s.params.conv_tol_ind = 1e-6
    orc = oracle.Oracle(params_copy(s.params), s.cell)
    rng = np.random.default_rng(3)
    pos = s.pos.copy()
    with ForceEngine(params_copy(s.params), s.cell) as eng:
        for t in range(5):
            xyz = [np.ascontiguousarray(pos[:, a]) for a in range(3)]
            g, o = eng.engforce(*xyz, itime=t), orc.engforce(*xyz, itime=t)
            assert eng.stats()["n_pol_iter"] == o["n_scf"]
            compare(g, o, 1e-9)
            pos = pos + rng.normal(0.0, 0.01, pos.shape)
