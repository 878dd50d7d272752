"""Bin-local rows that share few mothers: gathered row groups beside tiled ones (needs a B200).

The groups of eight rows whose mothers are many are summed entry by entry, the others as 8 x 4 tiles.  Patterns with
random mothers (one entry a row, up to the most that are gathered, and mixtures with rows without entries and with
shared mothers) must give the row kernels' states, within 1e-13 of their local magnitude, and gradients, within 1e-9
relative or 1e-12 of the largest, as the two kernel families elsewhere, with both stagings the same bits.
"""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from golden_io import local_scale_check
from prince_b200 import _lib
from prince_b200 import adjoint as AD
from prince_b200.operators import run_fd_loss_operator, split_diagonal
from prince_b200.solvers import DeviceRun
from test_gpu_layout import _network

pytestmark = pytest.mark.gpu
NSP, D, DPH = 40, 64, 8


def _mothers(rng, kind):
    """Mother species of each species by kind of pattern."""
    def some(s, k):
        return rng.choice(np.delete(np.arange(NSP), s), k, replace=False)
    if kind == "one":
        return [some(s, 1) for s in range(NSP)]
    if kind == "five":
        return [some(s, 5) for s in range(NSP)]
    if kind == "uneven":   # none to 30 a row: passes end at each row's own count
        return [some(s, int(k)) for s, k in enumerate(rng.integers(0, 31, NSP))]
    shared = some(0, 12)   # half the rows share twelve mothers (tiles), the others are random (gathered)
    return [np.setdiff1d(shared, [s]) if s % 2 else some(s, 3) for s in range(NSP)]


def _device(run, rng, kind):
    """The run's device state with the coupling replaced: bin-local rows of the kind and two band rows a bin."""
    dev = DeviceRun(run, 0)
    n = run.dim_states
    assert n == NSP * D
    e = np.arange(D)
    rows, cols = [], []
    for s, m in enumerate(_mothers(rng, kind)):
        rows.append(np.repeat(s * D + e, len(m)))
        cols.append((e[:, None] + D * np.asarray(m, dtype=np.int64)[None, :]).ravel())
    for b in (0, 1):
        for m in range(0, NSP, 3):
            for off in (1, 7):
                rows.append(b * D + e[: D - off])
                cols.append(m * D + e[off:])
    r, c = np.concatenate(rows), np.concatenate(cols)
    M = sp.csr_matrix((np.ones(r.size), (r, c)), shape=(n, n))
    M.sum_duplicates()
    M.sort_indices()
    ctx = dev.ctx
    ctx.set_coupling(n, M.indptr, M.indices)
    ctx.set_layout(D)
    assert ctx.info(_lib.PB_INFO_BLOCKED_LAYOUT) == 0   # the loss operator comes next
    ctx.set_photon_grid(np.logspace(-15, -6, DPH))
    ctx.set_fold_kernel(rng.uniform(0.0, 1e-43, (M.nnz, DPH)))   # rates of about one per unit of z an entry
    diag, off = split_diagonal(sp.csr_matrix(run_fd_loss_operator(run)))
    ctx.set_fd_operator(off, diag)
    pl = run.pair_loss_rates_grid
    pair_bin = np.tile(np.arange(D), NSP).astype(np.int32)
    ctx.set_losses(run.adia_loss_rates_grid.energy_vector, pl.scale_vec, pair_bin, pl.xi, pl.phi_xi2, pl.photon_grid)
    assert ctx.info(_lib.PB_INFO_BLOCKED_LAYOUT) == 1
    run._b200_device_runs = {0: dev}
    return dev


@pytest.mark.parametrize("kind", ["one", "five", "uneven", "mixed"])
@pytest.mark.parametrize("K", [9, 70])
def test_gathered_groups_against_the_row_kernels(kind, K):
    run = _network(NSP, D)
    rng = np.random.default_rng(K)
    ctx = _device(run, rng, kind).ctx
    species = [2212, 1000020040, 1000070140]
    sb = AD.SourceBatch(run, species, z_max=list(rng.uniform(0.01, 0.02, K)), initial_z=0.02)
    plan = sb.plan(0.02, ckpt_every=8)
    seed = torch.tensor(rng.uniform(0.5, 1.5, (run.dim_states, K)), device="cuda:0")
    par = dict(gamma=rng.uniform(0.5, 2.2, K), lg_rmax=rng.uniform(9.3, 10.5, K), frac=rng.dirichlet(np.ones(3), K),
               m=rng.uniform(-2, 4, K))
    states, grads = {}, {}
    for name, mode, tma in (("tma", 1, 1), ("cp.async", 1, 0), ("rows", 0, 1)):
        ctx.set_option(_lib.PB_OPT_BATCHED_KERNELS, mode)
        ctx.set_option(_lib.PB_OPT_TMA_STAGING, tma)
        t = {k: torch.tensor(v, dtype=torch.float64, requires_grad=True) for k, v in par.items()}
        scale = torch.tensor(1.0, dtype=torch.float64, requires_grad=True)
        X = AD.PropagateFunction.apply(sb.grids(t["gamma"], t["lg_rmax"], t["frac"]), sb.coefficients(t["m"]), scale, plan)
        assert ctx.info(_lib.PB_INFO_LAST_BLOCKED) == mode
        (seed * X).sum().backward()
        states[name] = X.detach().cpu().numpy()
        grads[name] = [t[k].grad.numpy().copy() for k in t] + [scale.grad.numpy().copy()]
    assert np.array_equal(states["tma"], states["cp.async"])
    worst, _, _ = local_scale_check(states["tma"], states["rows"], [s.sl for s in run.spec_man.species_refs], tol=1e-10)
    assert worst < 1e-13, worst
    for a, b, c in zip(grads["tma"], grads["cp.async"], grads["rows"]):
        assert np.array_equal(a, b)
        np.testing.assert_allclose(a, c, rtol=1e-9, atol=1e-12 * np.abs(c).max())
