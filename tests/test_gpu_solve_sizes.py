"""The step-program solve at the sizes where its chunks change: the last rows
count with chunks of 1024, 512, ... slots beside the solution in one block's 227
KB, and the ones around it. Against the grid solve (which other tests hold to the
oracle) bit for bit; the transpose against SciPy."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from rustspice_gb300 import native as N
from rustspice_gb300.solver import GpuKluSolver

pytestmark = pytest.mark.gpu


def last_rows(chunk):
    """Rows of the largest system whose solution (an even number of entries,
    one of them spare) leaves room for two chunks and their segments."""
    return (227 * 1024 - 48 * chunk - 2 * 65 * 8) // 8 // 2 * 2 - 1


SIZES = sorted({last_rows(ch) + d for ch in (1024, 512, 256, 128, 64, 32)
                for d in (-9, -3, -1, 0, 1)})


@pytest.mark.parametrize("staged", [False, True], ids=["loaded", "copied"])
@pytest.mark.parametrize("n", SIZES)
def test_sizes(n, staged, monkeypatch):
    if staged:  # the form of large programs: slots copied in bulk
        monkeypatch.setenv("GPUKLU_SOLVE_STAGED", "0")
    rng = np.random.default_rng(n)
    e = rng.uniform(-1.0, 1.0, (2, n - 1))
    e[:, 1::2] = 0.0  # 2 x 2 blocks
    A = sp.diags([e[0], rng.uniform(3.0, 4.0, n), e[1]], [-1, 0, 1]).tocsc()
    A.eliminate_zeros()
    A.sort_indices()
    ap, ai, ax = A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    b = rng.standard_normal(n)
    with monkeypatch.context() as m:
        m.setenv("GPUKLU_ONE_BLOCK", "0")
        r = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
        r.factor(ap, ai, ax)
        want = b.copy()
        r.solve(want)
        r.close()
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    g.factor(ap, ai, ax)
    x = b.copy()
    g.solve(x)
    assert np.array_equal(x, want), np.max(np.abs(x - want))
    y = b.copy()
    g.tsolve(y)
    ref = sla.spsolve(A.T.tocsc(), b)
    assert np.max(np.abs(y - ref)) <= 1e-12 * np.max(np.abs(ref))
    g.close()
