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
