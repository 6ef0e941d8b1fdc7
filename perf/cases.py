"""Timed cases: what programs have this framework do, through its public entry points.

A case is a dict of plain values.  ``listed()`` are the cases that are always
timed, ``draw(rng)`` gives another one of the same ranges, ``prepare`` makes
the inputs and the engine a program keeps, ``run`` is one pass, ``work`` the
bytes and operations of a pass, ``exact`` the same outputs in plain FP64 torch.

Kinds of pass:
  call     one engforce on device arrays (a snapshot, an optimiser's step)
  host     one engforce on host arrays (the Fortran host's call)
  md       velocity-Verlet steps on device-resident state
  host_md  velocity-Verlet steps of a host integrator around engforce
  batch    one evaluation of many independent boxes
  fit      forward and backward of a force-matching loss

Systems: rock-salt NaCl (Tosi-Fumi, not polarisable) and MgO (Lewis-Catlow,
polarisable O with Tang-Toennies damping), and silica as beta-cristobalite
(BKS with an r^-24 wall, polarisable O, damped), jittered off their lattice
sites, some formula units left out so that ion counts are ragged, the cell
sheared where a case says so.

The mixed-precision engine computes pairs and phases in FP32 and its forces are
good to single precision (its bar is 1e-5 relative): its results are handed on
as float32 arrays, as the programs that choose it keep them (trajectory frames,
training targets).  Results of the FP64 engine stay float64.
"""
import math

import numpy as np
import torch

from mdff_b200 import _abi, fit
from mdff_b200.engine import BatchEngine, ForceEngine
from mdff_b200.params import make_params

COUL = 14.3996441494161            # e^2/(4 pi eps0), eV A
PRESS = 0.00624150964712042        # GPa -> eV/A^3
RHO = 1.660538782                  # g/cm^3 -> amu/A^3
TIME = 98.2269514139276            # ps -> internal time
BOLTZ = 8.61734229648141e-05       # eV/K
SHEAR = np.array([[1.0, 0.15, 0.1], [0.0, 0.95, -0.08], [0.0, 0.0, 1.05]])


def _tosi_fumi():
    j = 1.0 / 1.602176487e-19
    sig, cpa = (1.170, 1.585), {(0, 0): 1.25, (0, 1): 1.0, (1, 1): 0.75}
    c = {(0, 0): 1.68, (0, 1): 11.2, (1, 1): 116.0}
    d = {(0, 0): 0.8, (0, 1): 13.9, (1, 1): 233.0}
    return {k: dict(A=cpa[k] * 0.338e-19 * j * math.exp((sig[k[0]] + sig[k[1]]) / 0.317), B=1.0 / 0.317,
                    C=c[k] * 1e-19 * j, D=d[k] * 1e-19 * j) for k in cpa}


# pair: A exp(-B r) - C/r^6 - D/r^8 + wall/r^24; tt: (dipole type, charge type) -> b, c
# (order 4); ratio: ions of each type per formula unit
MODELS = {
    "nacl": dict(q=(1.0, -1.0), mass=(22.98977, 35.453), ratio=(1, 1), units=4, density=1.55, temp=1200.0,
                 jitter=0.3, rcut=12.0, alpha=0.3, kmax=10, cells=6, pol={}, tt={}, pair=_tosi_fumi()),
    "mgo": dict(q=(2.0, -2.0), mass=(24.305, 15.9994), ratio=(1, 1), units=4, density=3.58, temp=2000.0,
                jitter=0.2, rcut=10.0, alpha=0.35, kmax=16, cells=10, pol={1: 1.6}, tt={(1, 0): (3.0, 1.0)},
                pair={(0, 1): dict(A=1428.5, B=1.0 / 0.2945, C=0.0, D=0.0),
                      (1, 1): dict(A=22764.0, B=1.0 / 0.149, C=27.88, D=0.0)}),
    "sio2": dict(q=(2.4, -1.2), mass=(28.0855, 15.9994), ratio=(1, 2), units=8, density=2.2, temp=300.0,
                 jitter=0.1, rcut=10.0, alpha=0.3, kmax=12, cells=8, pol={1: 1.3},
                 tt={(1, 1): (5.58406251008641721012, 2.8904937083), (1, 0): (3.66418041600447487325, 1.446)},
                 pair={(0, 1): dict(A=18003.7572, B=4.87318, C=133.5381, D=0.0, wall=1.2 ** 24),
                       (1, 1): dict(A=1388.7730, B=2.76, C=175.0, D=0.0, wall=1.9 ** 24),
                       (0, 0): dict(A=0.0, B=0.0, C=0.0, D=0.0, wall=2.4 ** 24)}),
}
EPSW = 1e-6      # accuracy of the Ewald rule where the box is smaller than the cutoff
SCALARS = ("u_bmhft", "vir_bmhft", "u_coul", "u_pol", "pvirial_coul")


# --------------------------------------------------------------------------
# cases

def listed():
    return [
        # the smallest call: a box of the size of the reference's own example decks, default engine
        dict(name="mgo216_fp64_scf_host", kind="host", system="mgo", cells=3, vacant=0, precision="fp64",
             solver="scf", shear=False, steps=1, efg=False),
        # the plain molten-salt run: the Fortran host integrates, engforce is called every step
        dict(name="nacl1728_fp64_host_md", kind="host_md", system="nacl", cells=6, vacant=0, precision="fp64",
             solver="cg", shear=False, steps=10, efg=False),
        # a large molten salt, ragged count, device-resident run in mixed precision
        dict(name="nacl13700_mixed_md", kind="md", system="nacl", cells=12, vacant=62, precision="mixed",
             solver="cg", shear=False, steps=4, efg=False),
        # polarisable MD with the reference's own settings: FP64, SCF from the ASPC predictor
        dict(name="sio2_3000_fp64_scf_md", kind="md", system="sio2", cells=5, vacant=0, precision="fp64",
             solver="scf", shear=False, steps=4, efg=False),
        # a snapshot solved from scratch by the default engine at the size of the MgO workload
        dict(name="mgo8000_fp64_scf_call", kind="call", system="mgo", cells=10, vacant=0, precision="fp64",
             solver="scf", shear=False, steps=1, efg=False),
        # a snapshot with its electric field gradients (the NMR / EFG analysis), FP64 CG
        dict(name="sio2_5100_fp64_cg_efg", kind="call", system="sio2", cells=6, vacant=27, precision="fp64",
             solver="cg", shear=False, steps=1, efg=True),
        # the two large polarisable MD workloads in mixed precision
        dict(name="sio2_12288_mixed_md", kind="md", system="sio2", cells=8, vacant=0, precision="mixed",
             solver="cg", shear=False, steps=5, efg=False),
        dict(name="mgo8000_mixed_md", kind="md", system="mgo", cells=10, vacant=0, precision="mixed",
             solver="cg", shear=False, steps=5, efg=False),
        # a triclinic snapshot of ragged size from host arrays, mixed precision from scratch
        dict(name="sio2_8100_tri_mixed_host", kind="host", system="sio2", cells=7, vacant=41, precision="mixed",
             solver="cg", shear=True, steps=1, efg=False),
        # the batched evaluation: 256 boxes of 64 to 1000 ions of both salts
        dict(name="batch256_mixed", kind="batch", boxes=256, nmin=64, nmax=1000, precision="mixed", host=False),
        # a small batch from host arrays (a few candidate structures at a time), FP64
        dict(name="batch24_fp64_host", kind="batch", boxes=24, nmin=64, nmax=300, precision="fp64", host=True),
        # a step of force-field fitting over 64 boxes
        dict(name="fit64", kind="fit", boxes=64, nmin=216, nmax=512),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "host", "md", "md", "host_md", "call", "batch", "batch", "fit"])
    if kind == "fit":
        nmin = rng.randrange(64, 217)
        return dict(kind=kind, boxes=logint(8, 64), nmin=nmin, nmax=rng.randrange(nmin + 40, 513))
    if kind == "batch":
        nmin = rng.randrange(64, 200)
        return dict(kind=kind, boxes=logint(8, 256), nmin=nmin, nmax=rng.randrange(nmin + 40, 1001),
                    precision=rng.choice(["mixed", "mixed", "fp64"]), host=rng.random() < 0.5)
    system = rng.choice(["nacl", "mgo", "sio2"])
    cells = logint(*{"nacl": (4, 12), "mgo": (3, 10), "sio2": (3, 8)}[system])
    precision = rng.choice(["fp64", "mixed"])
    solver = "cg" if precision == "mixed" or system == "nacl" else rng.choice(["scf", "cg"])
    md = kind in ("md", "host_md")
    units = MODELS[system]["units"] * cells ** 3
    ions = units * sum(MODELS[system]["ratio"])
    steps = max(1, min(20, (12000 if solver == "scf" else 50000) // ions)) if md else 1
    return dict(kind=kind, system=system, cells=cells, vacant=rng.randrange(0, max(2, int(units * (0.01 if md else 0.05)))),
                precision=precision, solver=solver, shear=not md and rng.random() < 0.3, steps=steps,
                efg=kind == "call" and precision == "fp64" and rng.random() < 0.3)


# --------------------------------------------------------------------------
# systems

def _lattice(system, m):
    """Cation and anion sites of m^3 conventional cells, in cell units of the box."""
    fcc = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    if system == "sio2":
        tet = np.array([[-1, -1, -1], [-1, 1, 1], [1, -1, 1], [1, 1, -1]]) / 8.0
        cat = np.concatenate([fcc, fcc + 0.25])
        ani = ((fcc + 0.25)[:, None] + tet[None]).reshape(-1, 3)
    else:
        cat, ani = fcc, fcc + np.array([0.5, 0, 0])
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return [(g[:, None] + b[None]).reshape(-1, 3) / m for b in (cat, ani)]


def _ewald_rule(L, cut):
    """alpha and kmax of ewald_param at EPSW for a cubic box of edge L."""
    tol = math.sqrt(abs(math.log(EPSW * cut)))
    alpha = math.sqrt(abs(math.log(EPSW * cut * tol))) / cut
    tol1 = math.sqrt(-math.log(EPSW * cut * (2.0 * tol * alpha) ** 2))
    return alpha, int(math.floor(0.25 + L * alpha * tol1 / math.pi + 0.5))


def _box(rng, system, m, vacant, density=1.0, shear=False):
    """One box: dict of the model, the cell, positions, ions per type, cutoffs, alpha and kmax."""
    M = MODELS[system]
    units = M["units"] * m ** 3
    mass = sum(r * w for r, w in zip(M["ratio"], M["mass"]))
    L = (units * mass * RHO / (M["density"] * density)) ** (1.0 / 3.0)
    cell = L * (SHEAR if shear else np.eye(3))
    natmi = [r * (units - vacant) for r in M["ratio"]]
    frac = np.concatenate([s[np.sort(rng.choice(len(s), n, replace=False))]
                           for s, n in zip(_lattice(system, m), natmi)])
    pos = frac @ cell.T + rng.uniform(-M["jitter"], M["jitter"], frac.shape)
    inv = np.linalg.inv(cell)
    half = 0.5 * min(1.0 / np.linalg.norm(inv, axis=1))
    rc = min(M["rcut"], half)
    alpha, kmax = M["alpha"], [int(round(M["kmax"] * m / M["cells"]))] * 3
    if rc < M["rcut"]:
        alpha, k = _ewald_rule(np.linalg.norm(cell, axis=0).max(), rc)
        kmax = [k] * 3
    typ = np.repeat([0, 1], natmi)
    return dict(model=M, cell=cell, pos=pos, natmi=natmi, typ=typ, rs=rc, rl=rc, alpha=alpha, kmax=kmax,
                q=np.array(M["q"])[typ], pol=np.array([M["pol"].get(t, 0.0) for t in (0, 1)])[typ])


def _params(box, precision, **kw):
    M = box["model"]
    tab = {n: {k: p[n] for k, p in M["pair"].items() if p.get(n)} for n in ("A", "B", "C", "D", "wall")}
    tt = {(a, min(a, b), max(a, b)): v for (a, b), v in M["tt"].items()}
    base = dict(lcoulomb=1, lbmhft=1, cutshortrange=box["rs"], cutlongrange=box["rl"], skindiff=1.0,
                qch=list(M["q"]), Abmhftd=tab["A"], Bbmhftd=tab["B"], Cbmhftd=tab["C"], Dbmhftd=tab["D"],
                wall24=tab["wall"], alphaES=box["alpha"], kES=box["kmax"],
                ldip_polar=[1 if t in M["pol"] else 0 for t in (0, 1)], poldip_iso=M["pol"],
                ldip_damping={k: 1 for k in tt}, pol_damp_b={k: v[0] for k, v in tt.items()},
                pol_damp_c={k: v[1] for k, v in tt.items()}, pol_damp_k={k: 4 for k in tt},
                conv_tol_ind=1e-8, extrapolate_order=4,
                precision=_abi.PREC_MIXED if precision == "mixed" else _abi.PREC_FP64)
    base.update(kw)
    return make_params(box["natmi"], **base)


def _single(case, seed):
    rng = np.random.default_rng(seed)
    box = _box(rng, case["system"], case["cells"], case["vacant"], shear=case["shear"])
    mass = np.array(box["model"]["mass"])[box["typ"]]
    v = rng.standard_normal(box["pos"].shape) * np.sqrt(BOLTZ * box["model"]["temp"] / mass)[:, None]
    box["vel"] = v - (v * mass[:, None]).sum(0) / mass.sum()
    box["mass"] = mass
    box["dt"] = 0.001 * TIME
    return box


def _boxes(case, seed):
    """The boxes of a batch: both salts (MgO alone for the fit), densities within
    10 %.  Kinds, sizes and densities belong to the case, the sites that are
    filled and the positions come from the seed."""
    plan, rng = np.random.default_rng(case["boxes"] * 1000003 + case["nmin"] * 1009 + case["nmax"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["boxes"]):
        system = "mgo" if case["kind"] == "fit" or plan.random() < 0.5 else "nacl"
        half = int(plan.integers(case["nmin"] // 2, case["nmax"] // 2 + 1))
        m = 1
        while 4 * m ** 3 < half:
            m += 1
        b = _box(rng, system, m, 4 * m ** 3 - half, density=plan.uniform(0.9, 1.1))
        L = b["cell"][0, 0]
        b["set"] = 0 if system == "nacl" else 1
        b["rs"], b["rl"] = (6.0, 4.0)[b["set"]], min(12.0, 0.5 * L)
        b["alpha"], k = _ewald_rule(L, b["rl"])
        b["kmax"] = [k] * 3
        out.append(b)
    return out


def _psets(precision, tol, maxit):
    sets = []
    for system, rs in (("nacl", 6.0), ("mgo", 4.0)):
        box = dict(model=MODELS[system], rs=rs, rl=12.0, alpha=1.0, kmax=[1] * 3, natmi=[1, 1])
        sets.append(_params(box, precision, lautoES=1, epsw=EPSW, solver=_abi.SOLVER_CG, cg_tol=tol,
                            cg_max_iter=maxit, conv_tol_ind=tol, calc=_abi.CALC_OTHER))
    return sets


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _soa(pos):
    return np.ascontiguousarray(pos.T)


THETA0 = np.array([1428.5, 0.2945, 0.0, 22764.0, 0.149, 27.88, 1.6, 3.0, 1.0, 1.0])


def _theta_true(seed):
    return THETA0 * (1.0 + 0.05 * np.random.default_rng(seed + 1).standard_normal(THETA0.size))


# --------------------------------------------------------------------------
# one pass

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        boxes = _boxes(case, seed)
        eng = BatchEngine(_psets(case["precision"], 1e-8, 200), [(b["set"], b["natmi"], b["cell"]) for b in boxes])
        pos = _soa(np.concatenate([b["pos"] for b in boxes]))
        st = dict(case=case, eng=eng, pos=pos)
        if not case["host"]:
            st.update(pos=_dev(pos), force=torch.zeros(pos.shape, dtype=torch.float64, device="cuda"),
                      mu=torch.zeros(pos.T.shape, dtype=torch.float64, device="cuda"),
                      ef=torch.zeros(pos.T.shape, dtype=torch.float64, device="cuda"))
        return st
    if kind == "fit":
        boxes = _boxes(case, seed)
        ff = fit.BatchForceField(_psets("fp64", 1e-11, 1000), [(b["set"], b["natmi"], b["cell"]) for b in boxes],
                                 fit.MGO_FIT)
        pos = _dev(_soa(np.concatenate([b["pos"] for b in boxes])))
        fn = fit.EngForceFn()
        with torch.no_grad():
            target = fn.apply(torch.tensor(_theta_true(seed)), ff, pos)[1]
        return dict(case=case, ff=ff, pos=pos, fn=fn, target=target,
                    theta=torch.tensor(ff.theta0, dtype=torch.float64, requires_grad=True))
    box = _single(case, seed)
    md = kind in ("md", "host_md")
    eng = ForceEngine(_params(box, case["precision"], calc=_abi.CALC_MD if md else _abi.CALC_OTHER,
                              solver=_abi.SOLVER_CG if case["solver"] == "cg" else _abi.SOLVER_SCF, cg_tol=1e-8),
                      box["cell"])
    pos, vel, n = _soa(box["pos"]), _soa(box["vel"]), len(box["mass"])
    st = dict(case=case, eng=eng, dt=box["dt"], t=0, pos=pos, vel=vel, invm=1.0 / box["mass"], force=None)
    if kind in ("call", "md"):
        st.update(pos=_dev(pos), vel=_dev(vel), invm=_dev(st["invm"]))
    if kind == "call":
        st.update({k: torch.zeros(s, dtype=torch.float64, device="cuda")
                   for k, s in (("force", (3, n)), ("mu", (n, 3)), ("ef", (n, 3)))})
    return st


def _thermo(r):
    return np.concatenate([[r[k] for k in SCALARS], np.ravel(r["tau"])])


def _as(case, out):
    """Results as the program keeps them: float32 from the mixed engine."""
    if case.get("precision") != "mixed":
        return out
    return {k: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32) for k, v in out.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fit":
        theta = state["theta"]
        theta.grad = None
        U, F, mu = state["fn"].apply(theta, state["ff"], state["pos"])
        loss = ((F - state["target"]) ** 2).sum()
        loss.backward()
        return {"loss": loss.detach(), "grad": theta.grad, "U": U.detach(), "F": F.detach(), "mu": mu.detach()}
    eng = state["eng"]
    if kind in ("host", "host_md"):
        return _as(case, _host(state, eng) if kind == "host" else _host_md(state, eng))
    if kind == "batch" and case["host"]:
        r = eng.engforce(*state["pos"])
        return _as(case, {"force": np.stack([r["fx"], r["fy"], r["fz"]]), "mu": r["mu"], "ef": r["ef"],
                          "thermo": np.stack([_thermo(c) for c in r["conf"]])})
    # the engine runs on its own streams: what torch has in flight on these tensors ends first
    torch.cuda.current_stream().synchronize()
    if kind == "md":
        e = eng.md_nve(state["pos"].data_ptr(), state["vel"].data_ptr(), state["invm"].data_ptr(), state["dt"],
                       case["steps"], itime0=state["t"])
        state["t"] += case["steps"]
        return _as(case, {"pos": state["pos"], "vel": state["vel"], "energy": e})
    ptr = [state[k].data_ptr() for k in ("pos", "force", "mu", "ef")]
    r = eng.engforce_device(*ptr)
    out = {k: state[k] for k in ("force", "mu", "ef")}
    out["thermo"] = np.stack([_thermo(c) for c in r]) if kind == "batch" else _thermo(r)
    if case.get("efg"):
        out["efg"] = eng.efg()
    return _as(case, out)


def _host(state, eng):
    r = eng.engforce(*state["pos"])
    return {"force": np.stack([r["fx"], r["fy"], r["fz"]]), "mu": r["mu"], "ef": r["ef"], "thermo": _thermo(r)}


def _host_md(state, eng):
    pos, vel, invm, dt = state["pos"], state["vel"], state["invm"], state["dt"]
    f = state["force"]
    energy = np.zeros((state["case"]["steps"], 2))
    for k in range(state["case"]["steps"]):
        if f is None:
            r = eng.engforce(*pos, itime=state["t"])
            f = np.stack([r["fx"], r["fy"], r["fz"]])
        vel += 0.5 * dt * f * invm
        pos += dt * vel
        state["t"] += 1
        r = eng.engforce(*pos, itime=state["t"])
        f = np.stack([r["fx"], r["fy"], r["fz"]])
        vel += 0.5 * dt * f * invm
        energy[k] = (0.5 * (vel * vel / invm).sum(), r["u_lj"] + r["u_bmhft"] + r["u_coul"])
    state["force"] = f
    return {"pos": pos, "vel": vel, "energy": energy, "force": f}


# --------------------------------------------------------------------------
# the work of a pass: pairs within the cutoffs and (k, ion) terms, each once per
# evaluation and per operator application that a solve to the tolerance needs

def work(case):
    def box_work(n, vol, rl, rs, nk, npol, applications, adjoint=False):
        near_l, near_s = n * n / vol * 4.19 * rl ** 3, n * n / vol * 4.19 * rs ** 3
        pp = near_l * (npol / n) ** 2
        f = near_s * 89 + near_l * 229 + nk * n * 52.0
        if npol:
            f += near_l * npol / n * 60 + nk * n * 31.0 + applications * (pp * 21 + nk * npol * 36.0)
        return f * (2.0 if adjoint else 1.0)

    if case["kind"] in ("batch", "fit"):
        flops = ions = 0.0
        for b in _boxes(case, 1):
            n, k = len(b["typ"]), b["kmax"][0]
            ions += n
            flops += box_work(n, abs(np.linalg.det(b["cell"])), b["rl"], b["rs"], ((2 * k + 1) ** 3 - 1) // 2,
                              int((b["pol"] > 0).sum()), 10, case["kind"] == "fit")
        return dict(bytes=ions * 8 * (3 + 9 if case["kind"] == "batch" else 3 + 9 + 6), flops=flops)
    M = MODELS[case["system"]]
    units = M["units"] * case["cells"] ** 3
    n = (units - case["vacant"]) * sum(M["ratio"])
    vol = units * sum(r * w for r, w in zip(M["ratio"], M["mass"])) * RHO / M["density"]
    L = vol ** (1.0 / 3.0)
    rc = min(M["rcut"], 0.5 * L)
    kmax = _ewald_rule(L, rc)[1] if rc < M["rcut"] else round(M["kmax"] * case["cells"] / M["cells"])
    npol = n * M["ratio"][1] / sum(M["ratio"]) if M["pol"] else 0
    md = case["kind"] in ("md", "host_md")
    per = {"scf": (8, 20), "cg": (6, 10)}[case["solver"]][0 if md else 1]
    nk = ((2 * kmax + 1) ** 3 - 1) // 2
    flops = case["steps"] * box_work(n, vol, rc, rc, nk, npol, per)
    if case["efg"]:
        flops += nk * n * 30.0
    per_ion = 8 * (12 if case["kind"] == "host_md" else 14 if md else 12 + (9 if case["efg"] else 0))
    return dict(bytes=n * per_ion * (case["steps"] if case["kind"] == "host_md" else 1), flops=flops)


# --------------------------------------------------------------------------
# the same outputs in plain FP64 torch: the Ewald multipole sum with the
# Numerical Recipes erfc, Tang-Toennies damping and dipoles solved to rounding

def _erfc(x):
    t = 1.0 / (1.0 + 0.5 * x)
    p = torch.full_like(t, 0.17087277)
    for c in (-.82215223, 1.48851587, -1.13520398, .27886807, -.18628806, .09678418, .37409196, 1.00002368):
        p = p * t + c
    return t * torch.exp(-x * x - 1.26551223 + t * p)


class _Solve(torch.autograd.Function):
    """x = H^-1 b for a symmetric operator given as a solver."""

    @staticmethod
    def forward(ctx, b, solve):
        ctx.solve = solve
        return solve(b)

    @staticmethod
    def backward(ctx, g):
        return ctx.solve(g), None


def _pairs(s, A, rmax):
    """Ordered pairs (i, j, r_i - r_j, r^2) within rmax by the minimum image."""
    ii, jj, rr = [], [], []
    n = len(s)
    for a in range(0, n, 512):
        d = s[a:a + 512, None] - s[None]
        d = (d - torch.round(d)) @ A.T
        r2 = (d * d).sum(-1)
        near = r2 <= rmax * rmax
        near[torch.arange(len(d), device=s.device), torch.arange(a, a + len(d), device=s.device)] = False
        i, j = torch.nonzero(near, as_tuple=True)
        ii.append(i + a)
        jj.append(j)
        rr.append(d[i, j])
    i, j, r = torch.cat(ii), torch.cat(jj), torch.cat(rr)
    return i, j, r, (r * r).sum(1)


def _exact_box(box, pos, theta=None, efg=False, device="cuda"):
    """Forces, dipoles, field and thermodynamics of one box; theta: the fit
    parameters as a tensor (differentiable), else the model's own values."""
    M, n = box["model"], len(box["typ"])
    t64 = dict(dtype=torch.float64, device=device)
    A = torch.tensor(box["cell"], **t64)
    Binv = torch.linalg.inv(A)
    vol = float(torch.linalg.det(A))
    typ = torch.tensor(box["typ"], device=device)
    al, kmax = box["alpha"], box["kmax"]
    tab = torch.zeros((5, 2, 2), **t64)
    for (a, b), p in M["pair"].items():
        for c, name in enumerate(("A", "B", "C", "D", "wall")):
            tab[c, a, b] = tab[c, b, a] = p.get(name, 0.0)
    A_, B_, C_, D_, W_ = tab
    tb, tc = torch.zeros((2, 2), **t64), torch.zeros((2, 2), **t64)
    for (a, b), (vb, vc) in M["tt"].items():
        tb[a, b], tc[a, b] = vb, vc
    qs = torch.tensor(M["q"], **t64)
    alpha_o = M["pol"].get(1, 0.0)
    if theta is not None:
        e01 = torch.tensor([[0.0, 1.0], [1.0, 0.0]], **t64)
        e11 = torch.tensor([[0.0, 0.0], [0.0, 1.0]], **t64)
        e10 = torch.tensor([[0.0, 0.0], [1.0, 0.0]], **t64)
        A_ = theta[0] * e01 + theta[3] * e11
        B_ = e01 / theta[1] + e11 / theta[4]
        C_ = theta[2] * e01 + theta[5] * e11
        alpha_o, tb, tc, qs = theta[6], theta[7] * e10, theta[8] * e10, qs * theta[9]
    q = qs[typ]
    s = pos @ Binv.T
    i, j, r, r2 = _pairs(s, A, max(box["rs"], box["rl"]))
    ti, tj = typ[i], typ[j]
    zero3 = torch.zeros((n, 3), **t64)
    eye = torch.eye(3, **t64)

    def tau6(rr, f):
        t = rr.T @ f
        return 0.5 * (t + t.T) * 0.5 / vol

    # short range
    near = (r2 < box["rs"] ** 2) & ((A_[ti, tj] != 0) | (W_[ti, tj] != 0))
    ri, d = r[near], torch.sqrt(r2[near])
    a, b = ti[near], tj[near]
    on = (A_[a, b] != 0).to(torch.float64)
    er, c6 = A_[a, b] * torch.exp(-B_[a, b] * d), on * C_[a, b] / d ** 6
    d8, wl = on * D_[a, b] / d ** 8, W_[a, b] / d ** 24
    f = ((B_[a, b] * er - 6 * c6 / d - 8 * d8 / d + 24 * wl / d) / d)[:, None] * ri
    F = zero3.index_add(0, i[near], f)
    u_sr = 0.5 * (er - c6 - d8 + wl).sum()
    vir_sr = 0.5 * (ri * f).sum() / 3.0
    tau = tau6(ri, f) / PRESS

    # real-space Ewald
    keep = r2 <= box["rl"] ** 2
    i, j, r, r2, ti, tj = i[keep], j[keep], r[keep], r2[keep], ti[keep], tj[keep]
    d = torch.sqrt(r2)
    ex = torch.exp(-al * al * r2) / math.sqrt(math.pi)
    F0 = _erfc(al * d)
    F1 = F0 + 2 * al * d * ex
    F2 = F1 + 4.0 / 3.0 * (al * d) ** 3 * ex
    F3 = F2 + 8.0 / 15.0 * (al * d) ** 5 * ex
    B0, B1, B2, B3 = F0 / d, F1 / d ** 3, 3 * F2 / d ** 5, 15 * F3 / d ** 7

    def damped(a, b):  # radial functions of the charge of type b on the dipole of type a
        x = tb[a, b] * d
        e = tc[a, b] * torch.exp(-x)
        f1 = e * (1 + x + x ** 2 / 2 + x ** 3 / 6 + x ** 4 / 24)
        f2 = f1 + d / 3 * tb[a, b] * e * x ** 4 / 24
        return B1 - f1 / d ** 3, B2 - 3 * f2 / d ** 5

    C1i, C2i = damped(ti, tj)
    C1j, C2j = damped(tj, ti)
    qi, qj = q[i], q[j]

    # reciprocal space
    kx, ky, kz = (torch.arange(-k, k + 1, **t64) for k in kmax)
    N = torch.stack(torch.meshgrid(kx, ky, kz, indexing="ij"), -1).reshape(-1, 3)
    N = N[(N[:, 0] > 0) | ((N[:, 0] == 0) & ((N[:, 1] > 0) | ((N[:, 1] == 0) & (N[:, 2] > 0))))]
    K = 2 * math.pi * N @ Binv
    kk = (K * K).sum(1)
    Ak = torch.exp(-kk / (4 * al * al)) / kk
    ph = 2 * math.pi * N @ s.T
    P = torch.polar(torch.ones_like(ph), ph)
    del ph
    tpi_V = 2 * math.pi / vol
    selfa, selfa2 = al / math.sqrt(math.pi), 2 * al ** 3 / (3 * math.sqrt(math.pi))

    def rho(qv, mu):  # sum_i (q_i + i k.mu_i) e^{i k.r_i}
        out = P @ qv.to(torch.complex128) if qv is not None else 0
        if mu is not None:
            out = out + 1j * (K.to(torch.complex128) * (P @ mu.to(torch.complex128))).sum(1)
        return out

    def rec_field(rh):  # -sum_k k A Im(rho conj(e))
        g = (P.conj().T @ ((Ak * 1.0)[:, None] * K * rh[:, None])).imag
        return -4 * tpi_V * g

    mu = zero3
    polar = bool(M["pol"])
    u_pol = torch.zeros((), **t64)
    if polar:
        ispol = torch.tensor(box["pol"] > 0, device=device)
        pm = ispol.to(torch.float64)[:, None]
        pp = (ispol[i] & ispol[j])
        ip, jp, rp, b1p, b2p = i[pp], j[pp], r[pp], B1[pp].detach(), B2[pp].detach()

        def T(m):
            mj = m[jp]
            e = b2p[:, None] * rp * (rp * mj).sum(1, keepdim=True) - b1p[:, None] * mj
            return (zero3.index_add(0, ip, e) + rec_field(rho(None, m)) + 2 * selfa2 * m) * pm

        Es = (zero3.index_add(0, i, (qj * C1i)[:, None] * r) + rec_field(rho(q, None))) * pm
        a0 = float(alpha_o)

        def solve(b):
            x = torch.zeros_like(b)
            res = b * pm
            p, rz, stop = res.clone(), float((res * res).sum()), 0.0
            stop = rz * 1e-28
            for _ in range(400):
                if rz <= stop:
                    break
                w = p / a0 - T(p)
                step = rz / float((p * w).sum())
                x, res = x + step * p, res - step * w
                new = float((res * res).sum())
                p, rz = res + new / rz * p, new
            return x

        with torch.no_grad():
            mu0 = solve(Es.detach())
        mu = mu0 + _Solve.apply(Es - mu0 / alpha_o + T(mu0), solve)
        u_pol = 0.5 * (mu * mu).sum() / alpha_o

    mi, mj = mu[i], mu[j]
    rmi, rmj = (r * mi).sum(1), (r * mj).sum(1)
    both = ((box_pol := torch.tensor(box["pol"] > 0, device=device))[i] & box_pol[j]).to(torch.float64)
    mij = (mi * mj).sum(1)
    u = qi * qj * B0 - both * (B2 * rmi * rmj - B1 * mij) + qi * C1j * rmj - qj * C1i * rmi
    fr = qi * qj * B1 + both * (B2 * mij - B3 * rmi * rmj) + qi * C2j * rmj - qj * C2i * rmi
    f = (fr[:, None] * r + (both * B2 * rmj + qj * C1i)[:, None] * mi
         + (both * B2 * rmi - qi * C1j)[:, None] * mj)
    e = (qj * C1i + both * B2 * rmj)[:, None] * r - (both * B1)[:, None] * mj
    rh = rho(q, mu)
    st = Ak * (rh.real ** 2 + rh.imag ** 2)
    Er = rec_field(rh)
    kmu = K @ mu.T
    H = 4 * tpi_V * ((P.conj() * (Ak * rh)[:, None]).real * kmu).T @ K if polar else 0.0
    F = F + COUL * (zero3.index_add(0, i, f) + q[:, None] * Er + H)
    ef = zero3.index_add(0, i, e) + Er + 2 * selfa2 * mu
    u_coul = COUL * (0.5 * u.sum() + 2 * tpi_V * st.sum() - selfa * (q * q).sum() - selfa2 * (mu * mu).sum() + u_pol)
    kc = 2 * (1 / kk + 1 / (4 * al * al))
    trec = 2 * tpi_V / vol * (eye * st.sum() - (K * (kc * st)[:, None]).T @ K)
    tau_c = (tau6(r, f) + trec) * COUL / PRESS
    out = dict(F=F, mu=mu, ef=ef, U=u_sr + u_coul,
               thermo=torch.cat([torch.stack([u_sr, vir_sr, u_coul, u_pol, torch.trace(tau_c) / 3 * PRESS]),
                                 (tau + 2 * tau_c).reshape(-1)]))
    if efg:
        g = -qj[:, None, None] * (B2[:, None, None] * r[:, :, None] * r[:, None] - B1[:, None, None] * eye)
        rm = r[:, :, None] * mj[:, None]
        g = g + both[:, None, None] * (-(B3 * rmj)[:, None, None] * r[:, :, None] * r[:, None]
                                       + B2[:, None, None] * (rmj[:, None, None] * eye + rm + rm.transpose(1, 2)))
        g = torch.zeros((n, 3, 3), **t64).index_add(0, i, g)
        amp = (P.conj() * (Ak * rh)[:, None]).real
        kab = (K[:, :, None] * K[:, None] * torch.triu(torch.ones((3, 3), **t64))).reshape(-1, 9)
        g = g + 4 * tpi_V * (amp.T @ kab).reshape(n, 3, 3) - 2 * selfa2 * q[:, None, None] * eye
        out["efg"] = g * COUL
    return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = dict(dtype=torch.float64, device=dev)
    kind = case["kind"]
    if kind == "batch":
        got = [_exact_box(b, torch.tensor(b["pos"], **t64), device=dev) for b in _boxes(case, seed)]
        return {"force": torch.cat([g["F"] for g in got]).T.contiguous(), "mu": torch.cat([g["mu"] for g in got]),
                "ef": torch.cat([g["ef"] for g in got]), "thermo": torch.stack([g["thermo"] for g in got])}
    if kind == "fit":
        theta = torch.tensor(THETA0, requires_grad=True, **t64)
        true = torch.tensor(_theta_true(seed), **t64)
        loss, U, F, mu = 0.0, [], [], []
        for b in _boxes(case, seed):
            pos = torch.tensor(b["pos"], **t64)
            with torch.no_grad():
                target = _exact_box(b, pos, true, device=dev)["F"]
            g = _exact_box(b, pos, theta, device=dev)
            part = ((g["F"] - target) ** 2).sum()
            part.backward()
            loss += part.detach()
            U.append(g["U"].detach())
            F.append(g["F"].detach())
            mu.append(g["mu"].detach())
        return {"loss": loss, "grad": theta.grad.cpu(), "U": torch.stack(U), "F": torch.cat(F), "mu": torch.cat(mu)}
    box = _single(case, seed)
    pos = torch.tensor(box["pos"], **t64)
    if kind in ("call", "host"):
        g = _exact_box(box, pos, efg=case["efg"], device=dev)
        out = {"force": g["F"].T.contiguous(), "mu": g["mu"], "ef": g["ef"], "thermo": g["thermo"]}
        if case["efg"]:
            out["efg"] = g["efg"]
        return out
    vel, dt = torch.tensor(box["vel"], **t64), box["dt"]
    invm = torch.tensor(1.0 / box["mass"], **t64)[:, None]
    g, energy = _exact_box(box, pos, device=dev), []
    for _ in range(case["steps"]):
        vel = vel + 0.5 * dt * g["F"] * invm
        pos = pos + dt * vel
        g = _exact_box(box, pos, device=dev)
        vel = vel + 0.5 * dt * g["F"] * invm
        energy.append(torch.stack([0.5 * (vel * vel / invm).sum(), g["U"]]))
    out = {"pos": pos.T.contiguous(), "vel": vel.T.contiguous(), "energy": torch.stack(energy)}
    if kind == "host_md":
        out["force"] = g["F"].T.contiguous()
    return out
