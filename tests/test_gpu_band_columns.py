"""Band tiles at the edges of their launch choices (needs a B200).

The TMA-staged band kernel covers 8 columns per CTA when there are no more and
64 otherwise, and skips the warps without active columns; the mother species
are split over as many groups as give the shortest schedule, and the rows'
partial sums are added by one warp or eight.  At the edges of these choices
the states must equal those of the cp.async staging bit for bit (the same
partial sums), and match the general row kernels at the parity tolerance with
every bin within 1e-13 of its local magnitude, as the two kernel families do
elsewhere.
"""

import numpy as np
import pytest

from golden_io import local_scale_check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def medium_run():
    from workloads import network_run
    return network_run(max_mass=16, n_species=60, seed=5)


@pytest.mark.parametrize("K", [2, 8, 9, 16, 64, 65, 129])
def test_band_columns_against_both_references(medium_run, K):
    from prince_b200 import _lib
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    run = medium_run
    m = MultiRHSPropagationSolverETD2(initial_z=0.03, final_z=0.0, prince_run=run, K=K)
    for k, p in enumerate(draw_points(run, K, seed=K, z_range=(0.01, 0.04))):
        m[k].add_source_class(point_source(run, p))
    ctx = m._dev.ctx
    out = {}
    try:
        for name, mode, tma in (("tma", 1, 1), ("cp.async", 1, 0), ("rows", 0, 1)):
            ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
            ctx.set_option(_lib.PB_OPT_TMA_STAGING, tma)
            m.solve(dz=1e-3)
            assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == mode
            out[name] = m.state.copy()
    finally:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, 1)
    assert np.array_equal(out["tma"], out["cp.async"])
    worst, _, _ = local_scale_check(out["tma"], out["rows"], [s.sl for s in run.spec_man.species_refs], tol=1e-10)
    assert worst < 1e-13, worst
