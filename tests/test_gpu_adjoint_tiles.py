"""The adjoint sweep's tiles at the edges of their sizes (needs a B200).

The sweep's band kernel multiplies 64 columns per CTA and, where its shared
memory fits (up to 96 bins here, not 99), starts its sums from the loss term;
its bin-local kernel multiplies groups of eight mother rows as 8 x 4 tiles of 16
columns.  At column counts around those sizes, for bins that fill their row tiles
or not, with and without the photon scale, the loss term and the photohadronic
term, the gradients must equal those of the cp.async staging bit for bit (the
same sums), and match the row kernels' within 1e-9 relative, or 1e-12 of the
largest gradient of their kind where the terms cancel: the criterion of the two
kernel families' other comparison.
"""

import numpy as np
import pytest
import torch

from prince_b200 import _lib, synth
from prince_b200 import adjoint as AD
from prince_b200.run import PriNCeRun
from workloads import A56_PHOTON, cib_field

pytestmark = pytest.mark.gpu
SPECIES = [2212, 1000020040, 1000070140]
_RUNS = {}


def _run(bins):
    if bins not in _RUNS:
        species = synth.full_network_species(16, n_species=60)
        model = synth.SyntheticPhotoNuclear(species, seed=5, x_cut_proton=1e-4)
        _RUNS[bins] = PriNCeRun(model, cib_field(), cosmic_ray_grid=(5, 5 + bins * 9 / 96, 96 / 9),
                                photon_grid=A56_PHOTON)
    return _RUNS[bins]


@pytest.mark.parametrize("bins,K,off", [(96, 2, 0), (96, 8, 0), (96, 9, 0), (96, 16, 0), (96, 17, 0), (96, 64, 0), (96, 65, 0),
                                        (96, 129, 0), (64, 7, 0), (64, 66, 0), (99, 5, 0), (99, 65, 0),
                                        (96, 19, _lib.PB_PARTIAL_DIFF), (96, 19, _lib.PB_PHOTOHAD)])
@pytest.mark.parametrize("with_scale", [True, False])
def test_sweep_tiles_against_cp_async_and_row_kernels(bins, K, off, with_scale):
    run = _run(bins)
    rng = np.random.default_rng(K)
    sb = AD.SourceBatch(run, SPECIES, z_max=list(rng.uniform(0.01, 0.02, K)), initial_z=0.02)
    plan = sb.plan(0.02, ckpt_every=8)
    plan.flags &= ~off
    ctx = plan.dev.ctx
    assert ctx.info(_lib.PB_INFO_BLOCKED_LAYOUT) == 1
    seed = torch.tensor(rng.uniform(0.5, 1.5, (run.dim_states, K)), device="cuda:0")
    par = dict(gamma=rng.uniform(0.5, 2.2, K), lg_rmax=rng.uniform(9.3, 10.5, K),
               frac=rng.dirichlet(np.ones(len(SPECIES)), K), m=rng.uniform(-2, 4, K))
    out = {}
    try:
        for name, mode, tma in (("tma", 1, 1), ("cp.async", 1, 0), ("rows", 0, 1)):
            ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
            ctx.set_option(_lib.PB_OPT_TMA_STAGING, tma)
            t = {k: torch.tensor(v, dtype=torch.float64, requires_grad=True) for k, v in par.items()}
            scale = torch.tensor(1.0, dtype=torch.float64, requires_grad=with_scale)
            G = sb.grids(t["gamma"], t["lg_rmax"], t["frac"])
            X = AD.PropagateFunction.apply(G, sb.coefficients(t["m"]), scale, plan)
            assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == mode
            (seed * X).sum().backward()
            out[name] = [t[k].grad.numpy().copy() for k in t] + ([scale.grad.numpy().copy()] if with_scale else [])
    finally:
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, 1)
    for a, b, c in zip(out["tma"], out["cp.async"], out["rows"]):
        assert np.array_equal(a, b)
        np.testing.assert_allclose(a, c, rtol=1e-9, atol=1e-12 * np.abs(c).max())
