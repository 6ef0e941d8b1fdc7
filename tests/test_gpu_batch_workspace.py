"""Device memory of the batched engine's workspaces.

The autotuner tries shapes of up to 148 clusters, each with its own partner lists and pair
cache; afterwards the engine holds what its shape needs and no more (64 MB: allocation
granularity), and gives the same results.  With little memory free the engine runs fewer
clusters at a time instead of failing, with the same results (two solves at 1e-10)."""
import numpy as np
import pytest

from mdff_b200 import _abi, systems
from mdff_b200.engine import BatchEngine
from mdff_b200.params import params_copy

from .gpu_util import forces, rms_rel

pytestmark = pytest.mark.gpu


def _batch(cells):
    """MgO boxes of 8 ncell^3 ions, each with its own displacements."""
    boxes = {c: systems.mgo(ncell=c, jitter=0.15, seed=7, rcut=4.0, alpha=0.7, kmax=3) for c in set(cells)}
    kinds = sorted(boxes)
    psets = []
    for c in kinds:
        p = params_copy(boxes[c].params)
        p.calc, p.precision, p.solver = _abi.CALC_OTHER, _abi.PREC_FP64, _abi.SOLVER_CG
        p.conv_tol_ind = p.cg_tol = 1e-10
        psets.append(p)
    configs = [(kinds.index(c), [psets[kinds.index(c)].natmi[t] for t in range(2)], boxes[c].cell) for c in cells]
    rng = np.random.default_rng(2)
    return psets, configs, np.concatenate([boxes[c].pos + rng.normal(0.0, 0.02, boxes[c].pos.shape) for c in cells])


def _used(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_tune_keeps_one_shape():
    torch = pytest.importorskip("torch")
    # one box of 1728 ions, which wants a large cluster, among 147 of 64: one CTA per box
    # is the shape with the most partner lists
    psets, configs, P = _batch([6] + [2] * 147)
    with BatchEngine(psets, configs) as eng:  # (kernels and stacks resident before memory is compared)
        ref = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
        eng.tune()
    used0 = _used(torch)
    with BatchEngine(psets, configs) as eng:
        eng.engforce(P[:, 0], P[:, 1], P[:, 2])
        cluster, threads, _ = eng.tune()
        f = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
        tuned = _used(torch) - used0
    assert rms_rel(f, ref) <= 1e-8  # two solves at 1e-10
    with BatchEngine(psets, configs) as eng:
        eng.set_shape(cluster, threads)
        eng.engforce(P[:, 0], P[:, 1], P[:, 2])
        fresh = _used(torch) - used0
    assert abs(tuned - fresh) <= 64 << 20, (tuned, fresh)


def test_little_memory_runs_fewer_clusters():
    torch = pytest.importorskip("torch")
    psets, configs, P = _batch([6] * 100)  # 1728 ions: 12 MB of partner lists a cluster
    with BatchEngine(psets, configs) as eng:
        eng.set_shape(2, 512)
        ref = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(max(free - (700 << 20), 0), dtype=torch.uint8, device="cuda")
    try:
        with BatchEngine(psets, configs) as eng:
            eng.set_shape(2, 512)
            f = forces(eng.engforce(P[:, 0], P[:, 1], P[:, 2]))
    finally:
        del held
        torch.cuda.empty_cache()
    assert rms_rel(f, ref) <= 1e-8
