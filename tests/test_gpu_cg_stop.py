"""CG solves that end at every position of the device loop's body (four iterations).

The iterations after the one that ended the solve leave the dipoles, the counters and
the scalars alone: with a cap of 1..9 iterations the graph's loop gives the dipoles
of the launch-by-launch loop (per-kernel profiling), which runs no iteration too
many.  kz 34 and rows of 600 ny take the recurrence kernels.  The same iterations of the same FP64 operator in other summation orders: 1e-9; mixed,
FP32 sums in other orders: 1e-5 of the dipoles."""
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import ForceEngine
from mdff_b200.params import params_copy

from .gpu_util import rms_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED])
@pytest.mark.parametrize("cap,mesh", [(c, (7, 7, 7)) for c in (1, 2, 3, 4, 5, 8, 9)]
                         + [(c, m) for c in (3, 5) for m in ((2, 2, 34), (0, 600, 1))])
def test_iteration_caps(cap, mesh, precision):
    s = systems.random_ionic((20, 30, 20), L=13.0, seed=18, q=(-1.5, 2.0, -1.5), pol=(1.1, 0.0, 1.1),
                             kES=mesh, calc=_abi.CALC_OTHER)
    p = params_copy(s.params)
    p.solver, p.precision, p.cg_max_iter = _abi.SOLVER_CG, precision, cap
    p.fail_on_nonconvergence = 0
    p.cg_tol = 1e-12 if precision == _abi.PREC_FP64 else 1e-9
    res = []
    for prof in (False, True):
        with ForceEngine(p, s.cell) as eng:
            assert eng._lib.mdff_gpu_profile(eng._h, 1 if prof else 0) == 0
            for call in range(2):  # the loop alone, then within the whole-step graph
                r = eng.engforce(*s.soa())
                assert eng.stats()["n_pol_iter"] == cap
                res.append(r["mu"])
    for mu in res[:2]:
        assert rms_rel(mu, res[2]) <= (1e-9 if precision == _abi.PREC_FP64 else 1e-5)
