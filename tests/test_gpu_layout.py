"""Layouts at the C ABI: what they turn down and what a changed one leaves behind (needs a B200)."""

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# Sizes at which a write past the species' tables leaves the heap's own padding, in a child process: the library
# must turn the layout down, not the C library's heap checks.
_TAIL_COLUMN = """
import scipy.sparse as sp
from prince_b200 import _lib
ctx = _lib.Context(0)
for n, d, blocks, row, col in ((10, 4, 8, 1, 9), (8008, 4, 8, 1, 8001), (8008, 4, 8, 0, 8004), (8008, 4, 8, 2, 8003)):
    M = sp.csr_matrix(([1.0], ([row], [col])), shape=(n, n))   # a block row that couples to a tail row
    ctx.set_coupling(n, M.indptr, M.indices)
    ctx.set_layout(d, blocks)
    assert ctx.info(_lib.PB_INFO_BLOCKED_LAYOUT) == 0
ctx.close()
print("turned down")
"""


def test_block_row_that_couples_to_a_tail_row_keeps_the_row_kernels():
    """In the same bin (the column's remainder is the row's) and in another one."""
    res = subprocess.run([sys.executable, "-c", _TAIL_COLUMN], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "turned down" in res.stdout, res.stderr[-2000:]


def _network(n_species, bins):
    from prince_b200 import synth
    from prince_b200.run import PriNCeRun
    from workloads import A56_PHOTON, cib_field
    model = synth.SyntheticPhotoNuclear(synth.full_network_species(16, n_species=n_species), seed=5, x_cut_proton=1e-4)
    return PriNCeRun(model, cib_field(), cosmic_ray_grid=(5, 5 + bins * 9 / 96, 96 / 9), photon_grid=A56_PHOTON)


def _states(run, K, mode, seed=3):
    """A batch's states and the gradient of their sum with respect to the injection grids."""
    import numpy as np
    import torch
    from prince_b200 import _lib
    from prince_b200 import adjoint as AD
    from prince_b200.solvers import MultiRHSPropagationSolverETD2
    from workloads import draw_points, point_source
    m = MultiRHSPropagationSolverETD2(initial_z=0.02, final_z=0.0, prince_run=run, K=K)
    for k, p in enumerate(draw_points(run, K, seed=seed, z_range=(0.01, 0.03))):
        m[k].add_source_class(point_source(run, p))
    ctx = m._dev.ctx
    ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
    m.solve(dz=1e-3)
    assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == mode and ctx.info(_lib.PB_INFO_LAST_TMA) == mode
    species = [2212, 1000020040]
    sb = AD.SourceBatch(run, species, z_max=[0.02] * K, initial_z=0.02)
    plan = sb.plan(0.02, ckpt_every=8)
    G = sb.grids(torch.full((K,), 1.5, dtype=torch.float64), torch.full((K,), 10.0, dtype=torch.float64),
                 torch.full((K, 2), 0.5, dtype=torch.float64)).detach().requires_grad_(True)
    X = AD.PropagateFunction.apply(G, sb.coefficients(torch.zeros(K, dtype=torch.float64)),
                                   torch.tensor(1.0, dtype=torch.float64), plan)
    X.sum().backward()
    ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, 1)
    return m.state.copy(), G.grad.cpu().numpy().copy(), np.asarray(X.detach().cpu())


def test_second_network_on_a_context_gets_its_own_tensor_maps(monkeypatch):
    """A smaller network with other bins, set on the context that a larger one used: its states fit the same
    buffers, so only its layout tells its tensor maps from the first network's.  Against its row kernels on a
    context of its own: states within 1e-13 of their local magnitude, gradients within 1e-9 relative or 1e-12 of
    the largest, as the two kernel families elsewhere."""
    import numpy as np
    from golden_io import local_scale_check
    from prince_b200 import _lib
    from prince_b200.solvers import DeviceRun
    K = 9
    first, second, alone = _network(60, 96), _network(40, 64), _network(40, 64)
    _states(first, K, 1)
    shared = DeviceRun.of(first, 0).ctx
    with monkeypatch.context() as mp:
        mp.setattr(_lib, "Context", lambda device=0: shared)
        second._b200_device_runs = {0: DeviceRun(second, 0)}
    got = _states(second, K, 1)
    ref = _states(alone, K, 0)
    sls = [s.sl for s in second.spec_man.species_refs]
    for i in (0, 2):
        worst, _, _ = local_scale_check(got[i], ref[i], sls, tol=1e-10)
        assert worst < 1e-13, worst
    np.testing.assert_allclose(got[1], ref[1], rtol=1e-9, atol=1e-12 * np.abs(ref[1]).max())
