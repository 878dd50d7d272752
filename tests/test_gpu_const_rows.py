"""Constant operators of short and long rows (needs a B200).

Up to four entries a row on average a thread sums a row, beyond that four lanes do.  Around that line, without
entries, with rows of very different lengths, for an odd and an even number of steps (the row factors of two steps
take turns) and for steps of different lengths, the state must match a float64 ETD2 loop on the host to 1e-12 relative
(sums of positive terms; 60 steps of a few roundings each), through both entry points.
"""

import numpy as np
import pytest
import scipy.sparse as sp

from prince_b200 import _lib

pytestmark = pytest.mark.gpu


def _reference(d, L, zg, x):
    x = x.copy()
    for h in np.diff(zg):
        w = h * d
        e = np.exp(w)
        f1 = np.expm1(w) / w
        f2 = (np.expm1(w) - w) / (w * w)   # |w| >= 0.02: ten digits cancel at most four
        F = L @ x
        a = e * x + h * f1 * F
        x = a + h * f2 * (L @ a - F)
    return x


@pytest.mark.parametrize("steps", [1, 2, 59, 60])
@pytest.mark.parametrize("n,entries,kind", [(1, 0, "even"), (257, 0, "even"), (300, 4, "even"), (300, 5, "even"),
                                            (1000, 4, "uneven"), (1000, 3, "uneven"), (4097, 1, "even")])
def test_rows_against_the_host(n, entries, kind, steps):
    import torch
    rng = np.random.default_rng(n + entries)
    nnz = n * entries
    rows = np.repeat(np.arange(n), entries) if kind == "even" else np.sort(rng.integers(0, n, nnz) ** 2 // n)
    L = sp.csr_matrix((rng.uniform(0.1, 1.0, nnz) / max(entries, 1), (rows, rng.integers(0, n, nnz))), shape=(n, n))
    L.sum_duplicates()
    L.sort_indices()
    d = rng.uniform(2.0, 4.0, n)
    zg = np.concatenate([[0.0], np.cumsum(rng.uniform(0.01, 0.02, steps))])
    x0 = rng.uniform(0.5, 1.5, n)
    ref = _reference(d, L, zg, x0)
    ctx = _lib.Context(0)
    np.testing.assert_allclose(ctx.integrate_const(d, L, zg, x0), ref, rtol=1e-12)

    def dev(a, dtype):
        return torch.tensor(np.ascontiguousarray(a if a.size else np.zeros(1), dtype=dtype), device="cuda:0")

    t = [dev(d, np.float64), dev(L.indptr, np.int64), dev(L.indices, np.int32), dev(L.data, np.float64),
         dev(zg, np.float64), dev(x0, np.float64)]
    ctx.integrate_const_noalloc(n, t[0].data_ptr(), L.nnz, t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), steps,
                                t[4].data_ptr(), t[5].data_ptr())
    np.testing.assert_allclose(t[5].cpu().numpy(), ref, rtol=1e-12)
