"""Reciprocal channels and pair loops of the adjoint at the edges of their tiles.

The structure-factor channels run on groups of 8 mesh rows, tiles of 4 values
of nz and steps of 4 ions, the right-hand side on 16 ions and steps of 2 nz:
meshes with one k per row up to four tiles of nz, and a box whose weights do not
fit the staging buffer.  The gradient of a random linear function of energies,
forces and dipoles against central differences of the same FP64 engine at a
relative step of 1e-5 (truncation ~1e-10, solver noise 1e-13 / 1e-5), to 1e-6 of
the largest scaled entry."""
import numpy as np
import pytest

from mdff_b200 import _abi, fit, systems
from mdff_b200.params import params_copy

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MESHES = [(1, 1, 0), (2, 3, 1), (3, 2, 3), (5, 6, 4), (4, 5, 7), (6, 4, 8), (3, 3, 11), (4, 3, 12)]


def _boxes(name):
    if name == "meshes":
        out = []
        for k, m in enumerate(MESHES):
            s = systems.mgo(ncell=2, jitter=0.2, seed=60 + k, rcut=4.0, alpha=0.6, kmax=4)
            s.params.kES[0], s.params.kES[1], s.params.kES[2] = m
            out.append(s)
        return out
    if name == "many":  # more boxes than clusters of eight: small clusters
        return [systems.mgo(ncell=2, jitter=0.2, seed=80 + k, rcut=4.0, alpha=0.6, kmax=3 + k % 4) for k in range(90)]
    return [systems.mgo(ncell=6, jitter=0.15, seed=90, rcut=8.0, alpha=0.4, kmax=7)]


@pytest.mark.parametrize("name", ["meshes", "many", "large"])
def test_adjoint_channels_vs_fd(name):
    psets, configs, pos = [], [], []
    for k, s in enumerate(_boxes(name)):
        p = params_copy(s.params)
        p.conv_tol_ind = p.cg_tol = 1e-13
        p.max_scf_pol_iter = p.cg_max_iter = 3000
        p.calc, p.precision, p.solver = _abi.CALC_OTHER, _abi.PREC_FP64, _abi.SOLVER_CG
        psets.append(p)
        configs.append((k, [p.natmi[t] for t in range(p.ntype)], s.cell))
        pos.append(s.pos)
    ff = fit.BatchForceField(psets, configs, fit.MGO_FIT)
    x = torch.tensor(np.ascontiguousarray(np.concatenate(pos).T), dtype=torch.float64, device="cuda")
    rng = np.random.default_rng(11)
    wU = torch.tensor(1e-3 * rng.standard_normal(ff.nconf), device="cuda")
    wF = torch.tensor(rng.standard_normal((ff.ntot, 3)), device="cuda")
    wm = torch.tensor(rng.standard_normal((ff.ntot, 3)), device="cuda")
    fn = fit.EngForceFn()

    def j(t):
        U, F, mu = fn.apply(t, ff, x)
        return (wU * U).sum() + (wF * F).sum() + (wm * mu).sum()

    theta = ff.theta0.copy()
    th = torch.tensor(theta, dtype=torch.float64, requires_grad=True)
    j(th).backward()
    g = th.grad.numpy().copy()
    fd = np.zeros(theta.size)
    with torch.no_grad():
        for k in range(theta.size):
            h = 1e-5 * max(abs(theta[k]), 1.0)
            v = []
            for sg in (1, -1):
                t = theta.copy()
                t[k] += sg * h
                v.append(float(j(torch.tensor(t, dtype=torch.float64))))
            fd[k] = (v[0] - v[1]) / (2 * h)
    ff.close()
    sc = np.maximum(np.abs(theta), 1.0)
    err = np.abs(sc * (g - fd)) / np.abs(sc * fd).max()
    assert err.max() <= 1e-6, dict(zip(fit.param_names(fit.MGO_FIT), err))
