"""The solve of systems whose solution leaves no room for chunks of 128 slots
beside it in one block's shared memory (k_solve_list), at the edges of its
range: from 28,149 rows, the last with such chunks, over 29,054, the last whose
solution fits, to the grid solve beyond; the transpose has chunks of 64 and 32
to 28,725 rows, then the grid. Forward against the grid solve, and the oracle
at two sizes, bit for bit, the transpose against SciPy; the Newton loop, whose last iterations are launched
ahead and skipped, against the grid solve's bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, newton_dc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,arrow", [(n, False) for n in (28148, 28149, 28150, 28151, 28601, 28725,
                                                          28726, 29053, 29054, 29055)]
                         + [(28150, True), (29054, True)])
def test_edges(n, arrow, monkeypatch):
    rng = np.random.default_rng(n)
    e = rng.uniform(-1.0, 1.0, n - 1)
    A = sp.diags([e, rng.uniform(3.0, 4.0, n), e], [-1, 0, 1])
    if arrow:  # a row with far more updates than the others
        at = np.arange(0, n - 2, 7)
        A = A + sp.csr_matrix((rng.uniform(-1e-3, 1e-3, len(at)), (np.full(len(at), n - 1), at)),
                              shape=(n, n))
    A = A.tocsc()
    A.sort_indices()
    ap, ai, ax = A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    b = rng.standard_normal(n)
    got = []
    for one_block in ("1", "0"):  # 0: the grid solve
        monkeypatch.setenv("GPUKLU_ONE_BLOCK", one_block)
        g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
        for scale in (1.0, 1.5):
            g.factor(ap, ai, ax * scale)
            x = b.copy()
            g.solve(x)
            got.append(x)
            if one_block == "1":
                y = b.copy()
                g.tsolve(y)
                ref = sla.spsolve((A * scale).T.tocsc(), b)
                assert np.max(np.abs(y - ref)) <= 1e-12 * np.max(np.abs(ref))
        g.close()
    assert np.array_equal(got[0], got[2]) and np.array_equal(got[1], got[3])


@pytest.mark.parametrize("n", [28150, 29054])
def test_against_the_oracle(n):
    rng = np.random.default_rng(n)
    e = rng.uniform(-1.0, 1.0, n - 1)
    A = sp.diags([e, rng.uniform(3.0, 4.0, n), e], [-1, 0, 1]).tocsc()
    A.sort_indices()
    ap, ai, ax = A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    x = rng.standard_normal(n)
    o = po.Solver("nativeklu_exact", n)
    o.prepare(n)
    assert o.analyze(ap, ai) == 0 and o.factor(ap, ai, ax) == 0
    st, want = o.solve(x)
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    g.factor(ap, ai, ax)
    g.solve(x)
    assert st == 0 and np.array_equal(x, want)
    g.close()


def test_newton(monkeypatch):
    c = cz.mesh_dc(169, 300)
    cfg = N.newton_config(**wl.TIGHT)
    got = []
    for steps in ("1", "0"):
        monkeypatch.setenv("GPUKLU_SOLVE_STEPS", steps)
        g = GpuKluSolver(1, pivot_mode=N.PIVOT_EXACT)
        dc = DeviceCircuit(c)
        newton_dc(g, dc, cfg)  # the second run refactors from the first iteration on
        got.append(newton_dc(g, dc, cfg))
        g.close()
    assert got[0].converged and got[0].iterations == got[1].iterations
    assert np.array_equal(got[0].x, got[1].x)
