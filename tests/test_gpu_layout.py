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
