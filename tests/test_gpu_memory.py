"""Memory kept between calls is bounded and given back (needs a B200)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
GIB = 1 << 30


@pytest.fixture(scope="module")
def em_run():
    from workloads import em_network_run
    return em_network_run(max_mass=16, n_species=60, seed=5)


def _build(run, windows):
    from prince_b200.em_cascade import kinetic_transfer
    from prince_b200.solvers import DeviceRun
    ctx = DeviceRun.of(run, 0).ctx
    Tg, Te, _ = kinetic_transfer(ctx, run.photon_field, run.em_grid.grid, np.linspace(0.0, 1.0, windows), 1e-3)
    return Tg, Te


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_cascade_temporaries_kept_are_bounded(em_run):
    """Builds of 1,500 windows take more than 3 GB of temporaries; at most 2 GiB stay, and the results are the same
    bits with all, some and none of the temporaries in the kept memory."""
    _build(em_run, 3)
    before = _free()
    out = [_build(em_run, 1500) for _ in range(3)]
    kept = before - _free()
    assert 0 < kept <= 2 * GIB + (64 << 20), kept
    for Tg, Te in out[1:]:
        assert np.array_equal(Tg, out[0][0]) and np.array_equal(Te, out[0][1])


def test_solve_takes_the_idle_temporaries_when_memory_runs_out(em_run):
    """With the rest of the device taken, a solve whose buffers fit only where the cascade's temporaries lie."""
    from prince_b200 import _lib
    from prince_b200.schedule import make_schedule, z_grid
    from prince_b200.solvers import DeviceRun
    ctx = DeviceRun.of(em_run, 0).ctx
    for _ in range(2):
        _build(em_run, 400)
    n, K = em_run.dim_states, 5120
    x = np.ones((n, K))
    sched = make_schedule(z_grid(2e-3, 0.0, 1e-3), em_run.backend.update_rates_z_threshold)
    hog = torch.empty(_free() - (512 << 20), dtype=torch.uint8, device="cuda")
    ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 0)
    try:  # three arrays of 0.25 GB and more: over 512 MB, within 512 MB and the kept 2 GiB
        assert 3 * x.nbytes > 640 << 20
        ctx.solve(sched, _lib.PB_ADIABATIC | _lib.PB_PARTIAL_DIFF, K, None, np.full(sched.n_steps, K, dtype=np.int32), x,
                  init_state=True)
    finally:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
        del hog
    assert np.isfinite(x).all() and (x != 1.0).any()
    _build(em_run, 3)


def test_page_locked_cascade_results_are_bounded(em_run):
    """Results that are kept are page-locked up to a bound and plain beyond it, the same values; one window kept
    counts as its block, and what is released counts no more."""
    from prince_b200 import _lib

    def locked(a):
        return torch.from_numpy(a).is_pinned()

    Tg, Te = _build(em_run, 100)
    assert locked(Tg) and locked(Te)
    kept, total = [], 0
    while total <= 2 * _lib._LOCKED_MAX:
        g, e = _build(em_run, 100)
        kept.append(g[0])   # views: each keeps its build's block alive
        kept.append(e[0])
        total += g.nbytes + e.nbytes
        assert np.array_equal(g, Tg) and np.array_equal(e, Te)
    assert sum(Tg.nbytes for a in kept if locked(a)) <= _lib._LOCKED_MAX
    assert not locked(kept[-1])
    del kept, g, e
    assert all(locked(a) for a in _build(em_run, 100))


def test_band_partial_sums_take_the_launches_size():
    """2,048 columns: a solve allocates its states (four arrays), its operator, and partial sums of the groups that
    its launches take: a group has a species at least, so no more than 60 groups of the 192 band rows (189 MB), not
    the 148 of the largest launch (466 MB)."""
    from prince_b200 import _lib
    from prince_b200.photonfields import device_components, device_table
    from prince_b200.schedule import make_schedule, z_grid
    from prince_b200.solvers import DeviceRun
    from workloads import network_run
    run = network_run(max_mass=16, n_species=60, seed=5)
    ctx = DeviceRun.of(run, 0).ctx
    ctx.set_photon_field(device_components(run.photon_field), table=device_table(run.photon_field))
    n, K = run.dim_states, 2048
    sched = make_schedule(z_grid(2e-3, 0.0, 1e-3), run.backend.update_rates_z_threshold)
    x = np.ones((n, K))

    def solve(cols):
        ctx.solve(sched, _lib.PB_ADIABATIC | _lib.PB_PARTIAL_DIFF, cols, None,
                  np.full(sched.n_steps, cols, dtype=np.int32), np.ascontiguousarray(x[:, :cols]), init_state=True)

    solve(2)
    before = _free()
    solve(K)
    assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == 1
    taken = before - _free()
    partial = run.spec_man.nspec * 192 * K * 8
    assert taken <= 4 * x.nbytes + partial + (64 << 20), (taken, x.nbytes)
