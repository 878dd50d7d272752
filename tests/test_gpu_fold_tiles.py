"""The fold's tiles at the edges of their choices (needs a B200).

The fold multiplies the kernel (entries x photon bins) by the photon vectors of
all rate windows.  Its tile depends on the windows (1 to 8 warps of 16, then
blocks) and on the photon bins (two buffers of kernel rows or one, 16-byte or
8-byte copies when the bin count is odd).  A random kernel on a random pattern
is folded for window counts and photon bins at those edges and compared with
the host product: relative 1e-13 of the sum of absolute terms, the rounding of
at most 200 FP64 products in any order with two ulps of the densities.
"""

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dph,W", [(72, 1), (95, 16), (96, 17), (96, 49), (97, 128), (104, 129), (199, 63), (200, 130)])
def test_fold_values_against_the_host_product(dph, W):
    from prince_b200 import _lib
    from prince_b200.photonfields import CMBPhotonSpectrum, device_components
    from prince_b200.schedule import make_schedule
    rng = np.random.default_rng(100 * dph + W)
    n, d = 24, 8
    M = sp.random(n, n, density=0.35, random_state=3, format="csr")
    M = (M + sp.identity(n)).tocsr()
    M.sort_indices()
    R = M.nnz
    kernel = rng.uniform(0.5, 1.5, (R, dph)) * rng.choice([-1.0, 1.0], (R, dph))
    eph = np.logspace(-14, -10, dph)
    ctx = _lib.Context(0)
    ctx.set_coupling(n, M.indptr, M.indices)
    ctx.set_layout(d)
    ctx.set_fold_kernel(kernel)
    ctx.set_photon_grid(eph)
    field = CMBPhotonSpectrum()
    ctx.set_photon_field(device_components(field))
    ctx.set_fd_operator(sp.csr_matrix((n, n)), np.zeros(n))
    xi = np.linspace(3.0, 4.0, 3)
    ctx.set_losses(np.ones(n), np.zeros(n), np.full(n, -1), xi, np.ones(3), np.full((d, 3), 1e-12))
    zg = np.linspace(1.0, 0.9, W + 1)
    sched = make_schedule(zg, 0.0)
    assert len(sched.z_window) == W
    state = np.zeros((n, 1))
    ctx.solve(sched, _lib.PB_PHOTOHAD, 1, None, np.ones(W, dtype=np.int32), state)
    ip, ix = ctx.operator_pattern(n)
    rows = np.repeat(np.arange(n), np.diff(M.indptr))
    off = rows != M.indices
    assert np.array_equal(ix, M.indices[off])
    for w in {0, W // 2, W - 1}:
        dens = field.get_photon_density(eph, sched.z_window[w])
        ref, scale = kernel @ dens, np.abs(kernel) @ dens
        vals, diag, _ = ctx.window_values(w, n, ix.size)
        assert np.max(np.abs(vals - ref[off]) / scale[off]) < 1e-13
        assert np.max(np.abs(diag[rows[~off]] - ref[~off]) / scale[~off]) < 1e-13
