"""The step-program solve at the edges of its layout: rows of one operation
up to several thread rows, chains (a row with many more updates than steps),
chunk sizes from the largest to the smallest (set by the system's size), and
sizes beyond one block. Forward against the oracle bit for bit, the transpose
against SciPy (diagonally dominant systems: 1e-12 relative)."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from oracle import pyoracle as po
from rustspice_gb300 import native as N
from rustspice_gb300.solver import GpuKluSolver

pytestmark = pytest.mark.gpu


def _arrow(n, rng, band=0):
    """Dense last row and column, `band` off-diagonals."""
    A = sp.diags([rng.uniform(0.1, 1.0, n - k) for k in range(band + 1)], range(band + 1)).tolil()
    A = (A + A.T).tolil()
    A[n - 1, :] = rng.uniform(-1.0, 1.0, n)
    A[:, n - 1] = rng.uniform(-1.0, 1.0, (n, 1))
    A.setdiag(rng.uniform(4.0, 5.0, n) + 2 * band)
    A[n - 1, n - 1] = 2.0 * n
    return A.tocsc()


def _pairs(k, rng):
    """k independent 2 x 2 blocks behind one shared last unknown."""
    n = 2 * k + 1
    A = sp.lil_matrix((n, n))
    for i in range(k):
        A[2 * i, 2 * i + 1], A[2 * i + 1, 2 * i] = rng.uniform(-1, 1, 2)
        A[2 * i + 1, n - 1], A[n - 1, 2 * i] = rng.uniform(-1, 1, 2)
    A.setdiag(rng.uniform(3.0, 4.0, n))
    A[n - 1, n - 1] = 2.0 * n
    return A.tocsc()


def _ladder(n, rng):
    e = rng.uniform(-1.0, 1.0, n - 1)
    return sp.diags([e, rng.uniform(3.0, 4.0, n), e], [-1, 0, 1]).tocsc()


CASES = ([("arrow", n, b) for n, b in ((2, 0), (33, 0), (40, 1), (300, 2), (3000, 1))]
         + [("pairs", k, 0) for k in (1, 31, 32, 33, 127, 128, 129, 700)]
         + [("ladder", n, 0) for n in (22000, 26500, 28000, 28600, 30000)])


@pytest.mark.parametrize("kind,size,band", CASES, ids=[f"{c[0]}{c[1]}b{c[2]}" for c in CASES])
def test_step_program_edges(kind, size, band):
    rng = np.random.default_rng(size + band)
    A = {"arrow": lambda: _arrow(size, rng, band), "pairs": lambda: _pairs(size, rng),
         "ladder": lambda: _ladder(size, rng)}[kind]()
    A.sort_indices()
    n = A.shape[0]
    ap, ai, ax = A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    b = rng.standard_normal(n)
    o = po.Solver("nativeklu_exact", n)
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    for scale in (1.0, 1.5):  # a first factorization, then a refactorization
        o.prepare(n)
        assert o.analyze(ap, ai) == 0 and o.factor(ap, ai, ax * scale) == 0
        st, want = o.solve(b)
        assert st == 0
        g.factor(ap, ai, ax * scale)
        x = b.copy()
        g.solve(x)
        assert np.array_equal(x, want), np.max(np.abs(x - want))
        if g.stats()["noffdiag"] == 0:
            y = b.copy()
            g.tsolve(y)
            ref = sla.spsolve((A * scale).T.tocsc(), b)
            assert np.max(np.abs(y - ref)) <= 1e-12 * np.max(np.abs(ref))
    g.close()


@pytest.mark.parametrize("kind,size,band", [("arrow", 2, 0), ("arrow", 300, 2), ("pairs", 33, 0),
                                            ("pairs", 700, 0), ("ladder", 22000, 0),
                                            ("ladder", 28600, 0)])
def test_slots_laid_out_ahead(kind, size, band, monkeypatch):
    """The form of large programs (slots laid out by the grid, copied in bulk) at
    every chunk size: the same bits."""
    monkeypatch.setenv("GPUKLU_SOLVE_STAGED", "0")
    test_step_program_edges(kind, size, band)
