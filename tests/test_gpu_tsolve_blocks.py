"""Which kernel a transpose solve of many blocks takes: many uncoupled ones the
grid's (which takes the blocks together), few or coupled ones the step program.
Their orders of additions differ, so the results tell: bit for bit the grid
solve's on one side of the rule, not on the other. (The reference's pivots leave
dense blocks like these with small pivots; the results themselves are held to
the oracle's factors in test_solve_program.py and test_gpu_adjoint.py.)"""
import numpy as np
import pytest
import scipy.sparse as sp

from rustspice_gb300 import native as N
from rustspice_gb300.solver import GpuKluSolver

pytestmark = pytest.mark.gpu

# (blocks, rows of a block, coupled to the next block, over the grid):
# rows times blocks of 3.6 million is the line
CASES = [(2000, 8, False, True), (671, 8, False, True), (670, 8, False, False),
         (3000, 1, False, True), (400, 8, False, False), (2000, 8, True, False),
         (30, 12, True, False)]


@pytest.mark.parametrize("blocks,size,coupled,grid", CASES)
def test_blocks(blocks, size, coupled, grid, monkeypatch):
    rng = np.random.default_rng(blocks + size)
    A = sp.block_diag([sp.csc_matrix(rng.uniform(-1, 1, (size, size)) + 4 * size * np.eye(size))
                       for _ in range(blocks)])
    n = blocks * size
    if coupled:
        r = np.arange(blocks - 1) * size
        A = A + sp.csr_matrix((np.full(blocks - 1, 0.5), (r, r + size)), shape=(n, n))
    A = A.tocsc()
    A.sort_indices()
    ap, ai, ax = A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    b = rng.standard_normal(n)
    got = []
    for steps in ("1", "0"):
        monkeypatch.setenv("GPUKLU_SOLVE_STEPS", steps)
        g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
        g.factor(ap, ai, ax)
        y = b.copy()
        g.tsolve(y)
        assert np.all(np.isfinite(y))
        assert (g.stats()["noffdiag"] > 0) == coupled
        got.append(y)
        g.close()
    if size > 1 and not coupled and blocks > 1:
        assert np.array_equal(got[0], got[1]) == grid
