"""Batched boxes whose meshes are long in x and y (slabs, rods), beside boxes that leave
the least staging buffer.

A record of kx + ky = 112 is 2 KB: the least buffer (16 KB, which a shape of 256 threads
has beside a box above 853 ions) holds three of them twice, and at kx + ky = 80 four only
with the weights elsewhere.  Forces, energies and fields against the CPU oracle
(two dipole solves at 1e-12: 1e-9); the fit gradient of such a box beside one of 1728 ions
(least buffer at 512 threads) against its gradient alone, two adjoint solves at
1e-12 of the right-hand side: 1e-8 of the largest entry."""
import numpy as np
import pytest

from mdff_b200 import _abi, fit, systems
from mdff_b200.engine import BatchEngine
from mdff_b200.params import params_copy

from .gpu_util import compare

pytestmark = pytest.mark.gpu


def _params(s):
    p = params_copy(s.params)
    p.conv_tol_ind = p.cg_tol = 1e-12
    p.max_scf_pol_iter = p.cg_max_iter = 2000
    p.calc, p.precision, p.solver = _abi.CALC_OTHER, _abi.PREC_FP64, _abi.SOLVER_CG
    return p


def _batch(syslist):
    psets = [_params(s) for s in syslist]
    configs = [(k, [p.natmi[t] for t in range(p.ntype)], s.cell) for k, (p, s) in enumerate(zip(psets, syslist))]
    return psets, configs, np.concatenate([s.pos for s in syslist])


_ref = {}  # oracle results: the same boxes for every launch shape


@pytest.mark.parametrize("mesh", [(56, 56, 4), (40, 40, 12), (64, 48, 1)])
@pytest.mark.parametrize("shape", [(1, 256), (8, 256), (2, 512)])
def test_long_rows(oracle, shape, mesh):
    slab = systems.random_ionic((60, 70), L=16.0, seed=17, kES=mesh, triclinic=True)
    big = systems.mgo(ncell=5, jitter=0.15, rcut=7.0, alpha=0.45, kmax=5)  # 1000 ions
    psets, configs, P = _batch([slab, big])
    with BatchEngine(psets, configs) as eng:
        eng.set_shape(*shape)
        out = eng.engforce(P[:, 0], P[:, 1], P[:, 2])
        for c, s in enumerate((slab, big)):
            a, b = eng.offsets[c], eng.offsets[c + 1]
            r = {k: out[k][a:b] for k in ("fx", "fy", "fz", "mu", "ef")}
            r.update(out["conf"][c])
            key = mesh if c == 0 else "big"
            if key not in _ref:
                _ref[key] = oracle.Oracle(psets[c], s.cell).engforce(*s.soa())
            compare(r, _ref[key], 1e-9)


def test_adjoint_long_rows():
    torch = pytest.importorskip("torch")
    slab = systems.mgo(ncell=3, jitter=0.2, seed=61, rcut=6.0, alpha=0.5, kmax=4)
    slab.params.kES[0], slab.params.kES[1], slab.params.kES[2] = 56, 56, 4
    big = systems.mgo(ncell=6, jitter=0.15, seed=90, rcut=8.0, alpha=0.4, kmax=5)  # 1728 ions
    n = slab.natm
    rng = np.random.default_rng(5)
    wU, wF, wm = 1e-3, rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    grads = []
    for boxes in ([slab], [slab, big]):
        psets, configs, P = _batch(boxes)
        ff = fit.BatchForceField(psets, configs, fit.MGO_FIT)
        x = torch.tensor(np.ascontiguousarray(P.T), dtype=torch.float64, device="cuda")
        th = torch.tensor(ff.theta0.copy(), dtype=torch.float64, requires_grad=True)
        U, F, mu = fit.EngForceFn().apply(th, ff, x)
        (wU * U[0] + (torch.tensor(wF, device="cuda") * F[:n]).sum()
         + (torch.tensor(wm, device="cuda") * mu[:n]).sum()).backward()
        grads.append(th.grad.numpy().copy())
        ff.close()
    assert np.abs(grads[1] - grads[0]).max() <= 1e-8 * np.abs(grads[0]).max()
