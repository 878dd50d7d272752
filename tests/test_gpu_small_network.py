"""Small networks: all steps of a solve in one launch (needs a B200).

The light network (384 states) runs ``k_small`` for every batch that fits one
wave of clusters: one or two columns per cluster of one to eight CTAs.  The
batch sizes below are the edges of those choices, with columns switching on at
different redshifts.  As for the full network's short-range batches, every bin
must match the CPU oracle to 1e-10 of its local magnitude, and at most 1e-4 of
the support may miss the strict per-bin 1e-10: bins at the zero crossings of
the loss stencil's oscillations, which a relative 1e-15 of the oracle's own
operator values moves by as much.
"""

import pytest

from golden_io import local_scale_check
from oracle import etd2_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope="module")
def light():
    from workloads import light_run
    return light_run()


@pytest.mark.parametrize("K", [2, 17, 19, 38, 75, 149, 297])
def test_small_network_batches_match_the_oracle(light, K):
    from prince_b200 import _lib
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    run = light
    srcs = [point_source(run, p) for p in draw_points(run, K, seed=K, z_range=(0.01, 0.06))]
    m = MultiRHSPropagationSolverETD2(initial_z=0.05, final_z=0.0, prince_run=run, K=K)
    for k, s in enumerate(srcs):
        m[k].add_source_class(s)
    m.solve(dz=1e-3)
    # up to two columns per CTA fit one wave of 148; beyond that the bin-blocked kernels run
    assert m._dev.ctx.info(_lib.PB_INFO_LAST_BLOCKED) == (1 if K > 2 * 148 else 0)
    ref = O.OracleSolver(run, 0.05, 0.0, K=K, exp="cr").solve([[s] for s in srcs], dz=1e-3)
    worst, above, total = local_scale_check(m.state, ref, [s.sl for s in run.spec_man.species_refs], tol=TOL)
    assert worst <= TOL, (worst, above, total)
    assert above <= 1e-4 * total, (above, total)


@pytest.mark.parametrize("K", [1, 3])
def test_small_network_with_more_than_512_rows(K):
    """576 states (96 bins): the 1024-thread CTAs, one and three columns."""
    from prince_b200 import photonfields as pf, synth
    from prince_b200.run import PriNCeRun
    from prince_b200.solvers import MultiRHSPropagationSolverETD2, UHECRPropagationSolverETD2
    from workloads import A56_GRID, A56_PHOTON, draw_points, point_source
    model = synth.SyntheticPhotoNuclear(synth.light_network_species(), seed=1)
    run = PriNCeRun(model, pf.CMBPhotonSpectrum(), cosmic_ray_grid=A56_GRID, photon_grid=A56_PHOTON)
    assert run.dim_states == 576
    srcs = [point_source(run, p) for p in draw_points(run, K, seed=K, z_range=(0.03, 0.05))]
    if K == 1:
        m = UHECRPropagationSolverETD2(initial_z=0.05, final_z=0.0, prince_run=run)
        m.add_source_class(srcs[0])
    else:
        m = MultiRHSPropagationSolverETD2(initial_z=0.05, final_z=0.0, prince_run=run, K=K)
        for k, s in enumerate(srcs):
            m[k].add_source_class(s)
    m.solve(dz=1e-3)
    ref = O.OracleSolver(run, 0.05, 0.0, K=K, exp="cr").solve([[s] for s in srcs], dz=1e-3).reshape(576, K)
    worst, above, total = local_scale_check(m.state.reshape(576, K), ref, [s.sl for s in run.spec_man.species_refs],
                                            tol=TOL)
    assert worst <= TOL, (worst, above, total)
    assert above <= 1e-4 * total, (above, total)



def test_stage_profile_after_a_solve_in_one_launch(light):
    """The bin-blocked kernels of a small network's batch can be timed after a solve that ran in one launch, as
    after one that ran them; the states that the solve left are those of before, and the next solve's too."""
    import numpy as np
    from prince_b200 import _lib
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    m = MultiRHSPropagationSolverETD2(initial_z=0.05, final_z=0.0, prince_run=light, K=19)
    for k, p in enumerate(draw_points(light, 19, seed=19, z_range=(0.05, 0.06))):
        m[k].add_source_class(point_source(light, p))
    m.solve(dz=1e-3)
    ctx, state = m._dev.ctx, m.state.copy()
    assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == 0
    for stage in (1, 2):
        times = ctx.profile_stage(10, stage, reps=2)
        assert all(t > 0.0 for t in times), times
    m.solve(dz=1e-3)
    assert np.array_equal(m.state, state)


def _small_batch(run, K):
    """A batch of K points over 50 steps: (solver after the solve, columns and CTAs of a cluster, sources)."""
    from prince_b200 import _lib
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    srcs = [point_source(run, p) for p in draw_points(run, K, seed=K, z_range=(0.01, 0.06))]
    m = MultiRHSPropagationSolverETD2(initial_z=0.05, final_z=0.0, prince_run=run, K=K)
    for k, s in enumerate(srcs):
        m[k].add_source_class(s)
    m.solve(dz=1e-3)
    return m, divmod(m._dev.ctx.info(_lib.PB_INFO_LAST_SMALL), 256), srcs


@pytest.mark.parametrize("K,columns", [(2, 1), (17, 1), (75, 1), (149, 2), (296, 2), (297, 0)])
def test_small_network_batches_take_one_launch(light, K, columns):
    """The batch sizes of the oracle test above run the kernel that they are there for: a column per cluster up to
    the SMs, then two, and beyond one wave the bin-blocked kernels."""
    _, (cc, cs), _ = _small_batch(light, K)
    assert cc == columns and (cs >= 1) == (columns > 0), (cc, cs)
    if K == 2:
        assert cs == 8


def test_four_columns_per_cluster_match_the_oracle():
    """576 states: 75 columns do not fit a CTA each, and take four per cluster of several CTAs."""
    from prince_b200 import photonfields as pf, synth
    from prince_b200.run import PriNCeRun
    from workloads import A56_GRID, A56_PHOTON
    model = synth.SyntheticPhotoNuclear(synth.light_network_species(), seed=1)
    run = PriNCeRun(model, pf.CMBPhotonSpectrum(), cosmic_ray_grid=A56_GRID, photon_grid=A56_PHOTON)
    m, (cc, cs), srcs = _small_batch(run, 75)
    assert cc == 4 and cs > 1, (cc, cs)
    ref = O.OracleSolver(run, 0.05, 0.0, K=75, exp="cr").solve([[s] for s in srcs], dz=1e-3)
    worst, above, total = local_scale_check(m.state, ref, [s.sl for s in run.spec_man.species_refs], tol=TOL)
    assert worst <= TOL, (worst, above, total)
    assert above <= 1e-4 * total, (above, total)
