"""Cases of the propagation workloads: what they are, their inputs, one pass, and their exact values.

A case names a network, how many source-parameter points share one call, the
redshift range and the job:

* ``forward``   -- one solve through the solver API (one point: the single-RHS
  solver; several: the multi-RHS solver), states back on the host;
* ``gradient``  -- the differentiable solve, a chi-square of the z = 0
  all-particle flux against a fixed spectrum, and its gradient with respect to
  the source parameters of every point (and the photon-density scale);
* ``em_build``  -- the cascade transfer and the Bethe-Heitler pair shape of a
  list of rate windows, as a solve with a new photon field or step builds them.

A network (its grids, species, fold kernel) is built once per process, as a
program that scans sources keeps it; the points come from the seed.
"""

import math

import numpy as np
import torch

from prince_b200 import adjoint, cr_sources, photonfields, synth
from prince_b200.em_cascade import KineticCascadeModel
from prince_b200.operators import run_fd_loss_operator
from prince_b200.run import PriNCeRun
from prince_b200.schedule import make_schedule, z_grid
from prince_b200.solvers import MultiRHSPropagationSolverETD2, UHECRPropagationSolverETD2

DZ = 1e-3
CKPT = 32
INJECTED = (2212, 1000020040, 1000070140, 1000140280, 1000260560)  # H, He, N, Si, Fe

# name -> (max mass, species, log10 E range and bins per decade, model seed)
NETWORKS = {
    "light": (4, 6, (6, 14, 8), 1),          # 384 states: the light-nuclei run
    "mid": (16, 60, (5, 14, 96 / 9), 5),     # 5,760 states: up to oxygen
    "a56": (56, 350, (5, 14, 96 / 9), 2),    # 33,600 states: up to iron
}
EM_GRID = (-3, 14, 128 / 17)                 # 128 bins for gamma, e-, e+


def listed():
    return [
        # a first look at one source nearby: the smallest call, all launches and host work
        {"name": "light one near", "job": "forward", "network": "light", "points": 1, "z_lo": 0.1, "z_hi": 0.1},
        # the light-nuclei run over its whole range
        {"name": "light one", "job": "forward", "network": "light", "points": 1, "z_lo": 1.0, "z_hi": 1.0},
        # a scan of an odd number of points on the light network
        {"name": "light scan", "job": "forward", "network": "light", "points": 37, "z_lo": 0.5, "z_hi": 1.0},
        # one spectrum through the full network: what a fit without batching calls
        {"name": "full one", "job": "forward", "network": "a56", "points": 1, "z_lo": 1.0, "z_hi": 1.0},
        # a few walkers of a sampler
        {"name": "full few", "job": "forward", "network": "a56", "points": 7, "z_lo": 0.2, "z_hi": 0.4},
        # a ragged batch on a medium network
        {"name": "mid batch", "job": "forward", "network": "mid", "points": 203, "z_lo": 0.1, "z_hi": 0.8},
        # a ragged batch on the full network
        {"name": "full batch", "job": "forward", "network": "a56", "points": 100, "z_lo": 0.1, "z_hi": 0.5},
        # the headline batch: 512 points with uneven redshift ranges
        {"name": "full headline", "job": "forward", "network": "a56", "points": 512, "z_lo": 0.5, "z_hi": 1.0},
        # one optimiser step over source parameters and the photon-density scale
        {"name": "gradient scale", "job": "gradient", "network": "a56", "points": 128, "z_lo": 0.2, "z_hi": 0.4,
         "scale": True},
        # one optimiser step over source parameters alone
        {"name": "gradient sources", "job": "gradient", "network": "a56", "points": 250, "z_lo": 0.2, "z_hi": 0.4,
         "scale": False},
        # the co-evolved electromagnetic cascade
        {"name": "cascade batch", "job": "forward", "network": "a56", "points": 300, "z_lo": 0.1, "z_hi": 0.5,
         "em": True},
        # the cascade's matrices for the windows of a solve from z = 1
        {"name": "cascade build", "job": "em_build", "network": "a56", "windows": 100, "z_hi": 1.0, "em": True},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    job = rng.choice(["forward"] * 5 + ["gradient"] * 2 + ["cascade", "em_build"])
    network = rng.choice(["light", "mid", "a56", "a56"])
    if job == "em_build":
        return {"job": "em_build", "network": "a56", "windows": int(_log_uniform(rng, 3, 200)),
                "z_hi": round(_log_uniform(rng, 0.1, 2.0), 3), "em": True}
    if job == "cascade":
        z_hi = round(_log_uniform(rng, 0.05, 0.6), 3)
        return {"job": "forward", "network": rng.choice(["mid", "a56"]), "points": int(_log_uniform(rng, 2, 300)),
                "z_lo": round(z_hi * rng.uniform(0.2, 1.0), 3), "z_hi": z_hi, "em": True}
    if job == "gradient":
        z_hi = round(_log_uniform(rng, 0.05, 0.4), 3)
        return {"job": "gradient", "network": network, "points": int(_log_uniform(rng, 2, 200)),
                "z_lo": round(z_hi * rng.uniform(0.2, 1.0), 3), "z_hi": z_hi, "scale": rng.random() < 0.5}
    z_hi = round(_log_uniform(rng, 0.05, 1.0), 3)
    points = 1 if rng.random() < 0.2 else int(_log_uniform(rng, 2, 380))
    return {"job": "forward", "network": network, "points": points,
            "z_lo": round(z_hi * rng.uniform(0.2, 1.0), 3), "z_hi": z_hi}


_RUNS = {}


def _run(case):
    key = (case["network"], bool(case.get("em")))
    if key not in _RUNS:
        mass, count, grid, seed = NETWORKS[case["network"]]
        if case["network"] == "light":
            species, cut = synth.light_network_species(), {}
            field = photonfields.CMBPhotonSpectrum()
        else:
            species, cut = synth.full_network_species(mass, n_species=count), {"x_cut_proton": 1e-4}
            field = photonfields.CombinedPhotonField(
                [photonfields.CMBPhotonSpectrum(), photonfields.ModifiedBlackBodyCIB()])
        em = {"enable_em_cascade": True, "enable_em_decoupled_grid": True, "em_grid": EM_GRID} if key[1] else {}
        run = PriNCeRun(synth.SyntheticPhotoNuclear(species, seed=seed, **cut), field, cosmic_ray_grid=grid,
                        photon_grid=(-15, -6, grid[2]), **em)
        if key[1]:
            run.em_cascade_model = KineticCascadeModel(run, DZ)
        _RUNS[key] = run
    return _RUNS[key]


def _points(run, case, seed):
    """Seeded source-parameter points: spectral index, log10 rigidity cutoff, fractions, evolution, z_max."""
    rng = np.random.default_rng(seed)
    k = case["points"]
    species = [p for p in INJECTED if p in run.spec_man.pdgid2sref]
    return species, {
        "gamma": rng.uniform(-1.5, 2.5, k),
        "lg_rmax": rng.uniform(9.0, 11.0, k),
        "frac": rng.dirichlet(np.ones(len(species)), k),
        "m": rng.uniform(-3.0, 5.0, k),
        "z_max": rng.uniform(case["z_lo"], case["z_hi"], k) if case["z_lo"] < case["z_hi"] else np.full(k, case["z_hi"]),
    }


def _source(run, species, pt, k):
    params = {p: (pt["gamma"][k], 10 ** pt["lg_rmax"][k], float(f)) for p, f in zip(species, pt["frac"][k])}
    return cr_sources.RigdityCutoffSource(run, norm=1.0, params=params, m=("simple", float(pt["m"][k])),
                                          z_max=float(pt["z_max"][k]))


_TARGETS = {}


def _target(run, case):
    """The spectrum a fit compares with: the all-particle flux of one fixed point (device tensor)."""
    key = (case["network"], bool(case.get("em")), case["z_hi"])
    if key not in _TARGETS:
        species = [p for p in INJECTED if p in run.spec_man.pdgid2sref]
        pt = {"gamma": [1.0], "lg_rmax": [10.2], "frac": [np.full(len(species), 1.0 / len(species))], "m": [1.0],
              "z_max": [case["z_hi"]]}
        s = UHECRPropagationSolverETD2(initial_z=case["z_hi"], final_z=0.0, prince_run=run)
        s.add_source_class(_source(run, species, pt, 0))
        s.solve(dz=DZ)
        x = torch.as_tensor(s.state[:, None], device="cuda")
        egrid, flux = adjoint.group_flux(run, x)
        _TARGETS[key] = (egrid > 10 ** 9.5, flux[:, :1])
    return _TARGETS[key]


def prepare(case, seed):
    run = _run(case)
    if case["job"] == "em_build":
        rng = np.random.default_rng(seed)
        zs = np.sort(rng.uniform(0.0, case["z_hi"], case["windows"]))[::-1]
        return {"job": "em_build", "run": run, "zs": [float(z) for z in zs]}
    species, pt = _points(run, case, seed)
    if case["job"] == "forward":
        kw = dict(initial_z=case["z_hi"], final_z=0.0, prince_run=run)
        if case["points"] == 1:
            solver = UHECRPropagationSolverETD2(**kw)
            solver.add_source_class(_source(run, species, pt, 0))
        else:
            solver = MultiRHSPropagationSolverETD2(K=case["points"], **kw)
            for k in range(case["points"]):
                solver[k].add_source_class(_source(run, species, pt, k))
        if case.get("em"):
            sched = make_schedule(z_grid(case["z_hi"], 0.0, DZ), solver.recomp_z_threshold)
            run.em_cascade_model.prefetch([float(z) for z in sched.z_window])
        return {"job": "forward", "solver": solver}
    batch = adjoint.SourceBatch(run, species, z_max=pt["z_max"], initial_z=case["z_hi"], dz=DZ)
    par = {n: torch.tensor(pt[n], requires_grad=True) for n in ("gamma", "lg_rmax", "frac", "m")}
    scale = torch.tensor(1.0, dtype=torch.float64, requires_grad=bool(case["scale"]))
    return {"job": "gradient", "run": run, "batch": batch, "plan": batch.plan(case["z_hi"], dz=DZ, ckpt_every=CKPT),
            "par": par, "scale": scale, "target": _target(run, case)}


def run(state):
    if state["job"] == "forward":
        state["solver"].solve(dz=DZ)
        return state["solver"].state
    if state["job"] == "em_build":
        model = KineticCascadeModel(state["run"], DZ)
        model.prefetch(state["zs"])
        parts = [model(z) for z in state["zs"]]
        return [np.stack([p[i] for p in parts]) for i in range(3)]
    p, batch, scale = state["par"], state["batch"], state["scale"]
    x = adjoint.PropagateFunction.apply(batch.grids(p["gamma"], p["lg_rmax"], p["frac"]), batch.coefficients(p["m"]),
                                        scale, state["plan"])
    sel, target = state["target"]
    flux = adjoint.group_flux(state["run"], x)[1][sel]
    t = target[sel]
    chi2 = (((flux - t) / (0.1 * t + 1e-3 * t.max())) ** 2).sum(dim=0)
    wrt = list(p.values()) + ([scale] if scale.requires_grad else [])
    grads = torch.autograd.grad(chi2.sum(), wrt)
    return {"states": x.detach(), "chi2": chi2.detach(), "gradients": list(grads)}


def work(case):
    """Operations and bytes one pass cannot do without.

    Per step and active column the two stages multiply the off-diagonal
    coupling entries and the loss stencil; per rate window every coupling entry
    is folded with the photon field.  The operator's kernel is read once, the
    states written once; where the state, the stage state and F(x) exceed the
    126 MB L2 they also pass through memory once per stage (48 bytes a value and
    step).  A gradient needs the transposed products too, and reads as much.
    """
    if case["job"] == "em_build":
        n, ne, ncr, nz = 128, 400, 96, case["windows"]
        build = 2.0 * nz * (2 * n * n * ne + n * 400 * ne)     # contractions with the photon stacks
        passes = 2.0 * nz * n ** 3 * 5                         # one pass of the scattering and the lepton transfer
        return {"bytes": 8.0 * nz * (2 * n * n + n * ncr), "flops": build + passes}
    run = _run(case)
    n, entries = run.dim_states, run.int_rates.coupling_mat.nnz
    photon = run.ph_grid.d
    steps = z_grid(case["z_hi"], 0.0, DZ).size - 1
    windows = int(math.ceil(case["z_hi"] / 0.01))
    share = 1.0 - 0.5 * (1.0 - case["z_lo"] / case["z_hi"])   # mean active part of the range
    columns = case["points"] * steps * share
    flops = 2.0 * entries * photon * windows + columns * (2 * 2.0 * entries + 2 * 8.0 * n + 12.0 * n)
    data = 8.0 * entries * photon + 8.0 * n * case["points"]
    if 3 * 8.0 * n * case["points"] > 126e6:
        data += 48.0 * n * columns
    if case.get("em"):
        flops += columns * 2.0 * (2 * 128 * 128 + 128 * run.cr_grid.d)
    if case["job"] == "gradient":
        flops, data = 2.0 * flops, 2.0 * data
    return {"bytes": data, "flops": flops}


def _phi(w):
    """exp(w), (e^w - 1)/w and (e^w - 1 - w)/w^2 for w <= 0, by series near zero."""
    s = np.where(np.abs(w) < 0.5, w, 0.0)
    p1 = np.zeros_like(s)
    p2 = np.zeros_like(s)
    for q in range(16, -1, -1):
        p1 = p1 * s + 1.0 / math.factorial(q + 1)
        p2 = p2 * s + 1.0 / math.factorial(q + 2)
    big = np.where(np.abs(w) < 0.5, 1.0, w)
    e = np.exp(w)
    near = np.abs(w) < 0.5
    return e, np.where(near, p1, (e - 1.0) / big), np.where(near, p2, (e - 1.0 - big) / (big * big))


def exact(case, seed):
    """The light network's forward solves, stepped in numpy with dense matrices; None for the larger ones."""
    if case["job"] != "forward" or case["network"] != "light" or case.get("em"):
        return None
    run = _run(case)
    n, rates, pair = run.dim_states, run.int_rates, run.pair_loss_rates_grid
    field, egrid = run.photon_field, run.ph_grid.grid
    kernel, indptr, cols = rates._batch_matrix, rates.coupling_mat.indptr, rates.coupling_mat.indices
    rows = np.repeat(np.arange(n), np.diff(indptr))
    loss = run_fd_loss_operator(run).toarray()
    loss_diag = np.diag(loss).copy()
    loss_off = loss - np.diag(loss_diag)
    species, pt = _points(run, case, seed)
    k = case["points"]
    sources = [_source(run, species, pt, j) for j in range(k)]
    inject = np.stack([s.injection_grid for s in sources], axis=1)
    z = case["z_hi"] + np.arange(int(math.floor(case["z_hi"] / DZ)) + 1) * -DZ
    if abs(z[-1]) > 1e-12:
        z = np.append(z, 0.0)
    sched = make_schedule(z, run.backend.update_rates_z_threshold)   # step sizes, dl/dz and H(z) of the run's cosmology
    x = np.zeros((n, k))
    window = -1
    for i in range(z.size - 1):
        if sched.window[i] != window:
            window = sched.window[i]
            zw = sched.z_window[window]
            coupling = np.zeros((n, n))
            coupling[rows, cols] = kernel @ _cmb(egrid, zw, field)
            diag = np.diag(coupling).copy()
            coupling[np.arange(n), np.arange(n)] = 0.0
            dens = _cmb(pair.photon_grid, zw, field) * pair.phi_xi2
            rate = ((dens[:, 1:] + dens[:, :-1]) * np.diff(pair.xi) / 2.0).sum(axis=1)
            kappa_pair = pair.scale_vec * np.tile(rate, n // rate.size)
        h, dl = sched.h[i], sched.dldz[i]
        kappa = sched.hc[i] * run.adia_loss_rates_grid.energy_vector + kappa_pair
        e, p1, p2 = _phi(h * dl * (diag + kappa * loss_diag))
        evolve = np.where(z[i] <= pt["z_max"], (1.0 + z[i]) ** pt["m"], 0.0)
        b = sched.finj[i] * inject * evolve

        def rest(v):
            return dl * (coupling @ v + loss_off @ (kappa[:, None] * v)) + b

        f = rest(x)
        a = e[:, None] * x + h * p1[:, None] * f
        x = a + h * p2[:, None] * (rest(a) - f)
    return x[:, 0] if k == 1 else x


def _cmb(energy, z, field):
    """The black-body density (1+z)^2 n0(E / (1+z)) with the field's constants."""
    (_, pref, kt, _), = field.device_components()
    red = energy / (1.0 + z)
    ratio = np.minimum(red / kt, 709.0)
    return np.where(red / kt < 709.0, pref * (1.0 + z) ** 2 * red ** 2 / np.expm1(ratio), 0.0)
