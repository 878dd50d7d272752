"""A state that is not finite reaches what couples to it and nothing else (needs a B200).

The bin-local rows, and the sweep's loss term, are multiplied as 8 x 4 tiles whose zeros stand for pairs that do not
couple; zero times infinity is a NaN.  One such value is put into one column: species that the coupling cannot carry
it to have to stay finite and equal to the row kernels', and the other columns too.
"""

import numpy as np
import pytest
import torch

from prince_b200 import _lib
from prince_b200 import adjoint as AD
from prince_b200.schedule import make_schedule, z_grid

pytestmark = pytest.mark.gpu
K, COL = 9, 4
FLAGS = _lib.PB_ADIABATIC | _lib.PB_PAIRPROD | _lib.PB_PHOTOHAD | _lib.PB_PARTIAL_DIFF


@pytest.fixture(scope="module")
def medium():
    from workloads import network_run
    return network_run(max_mass=16, n_species=60, seed=5)


def _species(run):
    """(bins, daughters of each species as a matrix [daughter, mother], species with rows that leave their bin)."""
    n = run.dim_states
    d = n // run.spec_man.nspec
    M = run.int_rates.coupling_mat.tocoo()
    off = M.row != M.col
    r, c = M.row[off], M.col[off]
    links = np.zeros((n // d, n // d), dtype=bool)
    links[r // d, c // d] = True
    band = np.unique((r // d)[r % d != c % d])
    return d, links, band


def _reach(links, start, levels):
    hit = np.zeros(links.shape[0], dtype=bool)
    hit[start] = True
    for _ in range(levels):
        hit |= links[:, hit].any(axis=1)
    return hit


def _solve(run, state, n_steps, mode, tma=1):
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    m = MultiRHSPropagationSolverETD2(initial_z=n_steps * 1e-3, final_z=0.0, prince_run=run, K=state.shape[1])
    ctx = m._dev.ctx
    m._set_field(ctx)
    sched = make_schedule(z_grid(n_steps * 1e-3, 0.0, 1e-3), run.backend.update_rates_z_threshold)
    x = state.copy()
    try:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, tma)
        ctx.solve(sched, FLAGS, x.shape[1], None, np.full(sched.n_steps, x.shape[1], dtype=np.int32), x, init_state=True)
    finally:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, 1)
    return x


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("tma", [1, 0])
def test_forward_tiles(medium, value, tma):
    run = medium
    d, links, band = _species(run)
    local = np.setdiff1d(np.arange(links.shape[0]), band)
    # a mother with daughters that leaves the most bin-local species out of its reach over one step's two stages
    free = {s: np.setdiff1d(np.flatnonzero(~_reach(links, s, 2)), band) for s in local if links[local, s].any()}
    mother = max(free, key=lambda s: free[s].size)
    assert free[mother].size >= 8
    state = np.random.default_rng(1).uniform(1.0, 2.0, (run.dim_states, K))
    state[mother * d + d // 2, COL] = value
    got, ref = _solve(run, state, 1, 1, tma), _solve(run, state, 1, 0)
    rows = (free[mother][:, None] * d + np.arange(d)).ravel()
    assert np.isfinite(ref[rows]).all()
    assert np.isfinite(got[rows]).all()
    np.testing.assert_allclose(got[rows], ref[rows], rtol=1e-12)
    others = np.delete(np.arange(K), COL)
    assert np.isfinite(got[:, others]).all()


@pytest.mark.parametrize("tma", [1, 0])
def test_adjoint_tiles(medium, tma):
    """The sweep of two steps: its tiles carry a daughter's value to its mothers only, and the loss term inside the
    band kernel to the stencil's bins (three to a side and stage) only."""
    run = medium
    d, links, band = _species(run)
    n, e0 = run.dim_states, d // 2
    local = np.setdiff1d(np.arange(links.shape[0]), band)
    up = links.T
    free = {s: np.flatnonzero(~_reach(up, s, 3)) for s in local if up[local, s].any()}
    daughter = max(free, key=lambda s: free[s].size)
    assert free[daughter].size >= 8
    plan = AD.Plan(run, 2e-3, K, np.arange(n), np.arange(K), np.zeros(K, dtype=np.int64))
    coeff = torch.ones((plan.sched.n_steps, K), dtype=torch.float64)
    seed = torch.tensor(np.random.default_rng(2).uniform(1.0, 2.0, (n, K)), device="cuda:0")
    seed[daughter * d + e0, COL] = float("inf")
    grads = {}
    ctx = plan.dev.ctx
    try:
        for name, mode, stage in (("tiles", 1, tma), ("rows", 0, 1)):
            ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
            ctx.set_option(_lib.PB_OPT_TMA_STAGING, stage)
            G = torch.zeros((n, K), dtype=torch.float64, requires_grad=True)
            X = AD.PropagateFunction.apply(G, coeff, torch.tensor(1.0, dtype=torch.float64), plan)
            assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == mode
            X.backward(seed)
            grads[name] = G.grad.numpy().copy()
    finally:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, 1)
    got, ref = grads["tiles"], grads["rows"]
    far = np.flatnonzero(np.abs(np.arange(d) - e0) > 3 * 3)
    rows = np.concatenate([(free[daughter][:, None] * d + np.arange(d)).ravel(), daughter * d + far])
    assert np.isfinite(ref[rows]).all()
    assert np.isfinite(got[rows]).all()
    np.testing.assert_allclose(got[rows], ref[rows], rtol=1e-9, atol=1e-12 * np.abs(ref[rows]).max())
    assert np.isfinite(got[:, np.delete(np.arange(K), COL)]).all()
