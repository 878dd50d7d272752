"""Captured runs of steps: what is kept, what is replayed, and the same bits wherever a step falls (needs a B200)."""

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _bare_context(n):
    """A context with ``n`` states that only lose energy: no coupling entries, no stencil neighbours."""
    from prince_b200 import _lib
    ctx = _lib.Context(0)
    empty = sp.csr_matrix((n, n))
    ctx.set_coupling(n, empty.indptr, empty.indices)
    ctx.set_photon_grid(np.logspace(-15, -6, 8))
    ctx.set_photon_field([(0, 1.0, 1e-13, 0.0)])
    ctx.set_fd_operator(empty, np.ones(n))
    ctx.set_losses(np.ones(n), np.zeros(n), np.full(n, -1), np.linspace(1.0, 2.0, 4), np.ones(4), np.ones((1, 4)))
    return ctx


class _Sched:
    def __init__(self, n_steps):
        self.n_steps = n_steps
        self.z_window = np.array([0.5])
        self.window = np.zeros(n_steps, dtype=np.int32)
        self.h = np.full(n_steps, -1e-3)
        self.dldz = np.full(n_steps, -1.0)
        self.hc = np.full(n_steps, 1.0)
        self.finj = np.zeros(n_steps)


def test_run_with_a_refused_launch_is_not_kept():
    """More columns than a grid has column tiles: the launch is refused on the host.  Every solve has to say so, the
    second as the first: a run kept without its kernels would return the initial state as the answer."""
    from prince_b200 import _lib
    ctx = _bare_context(2)
    K = 65535 * 32 + 1
    sched = _Sched(16)
    state = np.ones((2, K))
    n_active = np.full(16, K, dtype=np.int32)
    for _ in range(2):
        with pytest.raises(RuntimeError):
            ctx.solve(sched, _lib.PB_ADIABATIC | _lib.PB_PARTIAL_DIFF, K, None, n_active, state, init_state=True)
    # the context still solves what fits
    K = 4
    state = np.ones((2, K))
    ctx.solve(sched, _lib.PB_ADIABATIC | _lib.PB_PARTIAL_DIFF, K, None, np.full(16, K, dtype=np.int32), state,
              init_state=True)
    np.testing.assert_allclose(state, np.exp(16e-3), rtol=1e-12)


@pytest.mark.parametrize("n", [600, 1500])
def test_one_column_sits_out_the_steps_without_active_columns(n):
    """Steps without active columns leave the state alone, inside a captured run (n above the small networks') as
    in one launch of all steps and step by step: sixteen steps of which twelve are taken, then two more."""
    from prince_b200 import _lib
    ctx = _bare_context(n)
    active = np.ones(18, dtype=np.int32)
    active[[3, 4, 9, 15]] = 0
    state = np.ones((n, 1))
    ctx.solve(_Sched(18), _lib.PB_ADIABATIC | _lib.PB_PARTIAL_DIFF, 1, None, active, state, init_state=True)
    np.testing.assert_allclose(state, np.exp(14e-3), rtol=1e-12)


@pytest.fixture(scope="module")
def medium_run():
    from workloads import network_run
    return network_run(max_mass=16, n_species=60, seed=5)


@pytest.mark.parametrize("K,band_warps", [(20, 8), (70, 8), (203, 8), (203, 4)])
def test_states_do_not_depend_on_the_checkpoints(medium_run, K, band_warps):
    """Columns that switch on step by step, across multiples of 64: with checkpoints every step, every five (all
    steps launched alone), every 32 and none (runs at other places), the states are the same bits."""
    import torch
    from prince_b200 import _lib
    from prince_b200 import adjoint as AD
    run = medium_run
    rng = np.random.default_rng(K)
    species = [2212, 1000020040, 1000070140]
    sb = AD.SourceBatch(run, species, z_max=list(rng.uniform(0.005, 0.08, K)), initial_z=0.08)
    G = sb.grids(torch.tensor(rng.uniform(0.5, 2.2, K)), torch.tensor(rng.uniform(9.3, 10.5, K)),
                 torch.tensor(rng.dirichlet(np.ones(3), K)))
    coeff = sb.coefficients(torch.tensor(rng.uniform(-2, 4, K)))
    out = []
    for every in (1, 5, 32, 0):
        plan = sb.plan(0.08, ckpt_every=every)
        ctx = plan.dev.ctx
        ctx.set_option(_lib.PB_OPT_BAND_WARPS, band_warps)
        try:
            X = AD.PropagateFunction.apply(G, coeff, torch.tensor(1.0, dtype=torch.float64), plan)
        finally:
            ctx.set_option(_lib.PB_OPT_BAND_WARPS, 8)
        assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == 1
        out.append(X.cpu().numpy())
    for other in out[1:]:
        assert np.array_equal(out[0], other)


def _batch(run, K, z_range, initial_z, seed):
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    m = MultiRHSPropagationSolverETD2(initial_z=initial_z, final_z=0.0, prince_run=run, K=K)
    for k, p in enumerate(draw_points(run, K, seed=seed, z_range=z_range)):
        m[k].add_source_class(point_source(run, p))
    return m


def test_wide_ragged_batch_captures_once(medium_run):
    """2,048 columns that switch on over 800 steps: every column count of the launches is captured by the first
    solve and found by the second."""
    from prince_b200 import _lib
    m = _batch(medium_run, 2048, (0.01, 0.4), 0.4, seed=1)
    m.solve(dz=5e-4)
    ctx = m._dev.ctx
    first, state = ctx.info(_lib.PB_INFO_STEP_CAPTURES), m.state.copy()
    m.solve(dz=5e-4)
    assert ctx.info(_lib.PB_INFO_STEP_CAPTURES) == first
    assert np.array_equal(m.state, state)


def test_runs_are_dropped_and_captured_again(medium_run):
    """More batch sizes than runs are kept: the first size's run has gone when it is solved again, with another
    schedule and then the first one, and the states are the same bits as before, and as with the other staging."""
    from prince_b200 import _lib
    run = medium_run
    first = _batch(run, 9, (0.01, 0.04), 0.04, seed=2)
    ctx = first._dev.ctx
    first.solve(dz=1e-3)
    state = first.state.copy()
    for K in range(10, 40):
        _batch(run, K, (0.01, 0.02), 0.02, seed=K).solve(dz=1e-3)
    before = ctx.info(_lib.PB_INFO_STEP_CAPTURES)
    other = _batch(run, 9, (0.01, 0.03), 0.03, seed=3)
    other.solve(dz=1e-3)
    assert ctx.info(_lib.PB_INFO_STEP_CAPTURES) == before + 1
    first.solve(dz=1e-3)
    assert ctx.info(_lib.PB_INFO_STEP_CAPTURES) == before + 1   # the same run, for another schedule
    assert np.array_equal(first.state, state)
    again = other.state.copy()
    ctx.set_option(_lib.PB_OPT_TMA_STAGING, 0)                  # other kernels, the same sums
    try:
        other.solve(dz=1e-3)
    finally:
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, 1)
    assert np.array_equal(other.state, again)
