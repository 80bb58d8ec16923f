"""The bordered solver's sparse triangular solves, level sweeps and Schur
assembly at their edges: blocks of symmetric and of unsymmetric pattern (the
reach is a chain of first members, or the closure), blocks whose vector needs
the global scratch and whose solve is left to the plain kernels (30,000 and
12,000 rows), border sizes around a group of 32 rows and a panel of the dense
solve, border rows and columns that touch no block, and repeated entries.
Against SciPy; the systems are diagonally dominant, so the solutions agree to
1e-12 of their largest entry."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from rustspice_gb300.solver import BbdSolver

pytestmark = pytest.mark.gpu


def _block(kind, n, rng):
    if kind == "ladder":
        e = rng.uniform(-1.0, 1.0, (2, n - 1))
        A = sp.diags([e[0], np.zeros(n), e[1]], [-1, 0, 1])
    else:
        A = sp.random(n, n, density=min(1.0, 3.0 / n), random_state=rng,
                      data_rvs=lambda k: rng.uniform(-1.0, 1.0, k))
        if kind == "sym":
            A = A + A.T
    return sp.csc_matrix(A)


def _system(kind, sizes, border, rng):
    nm = sum(sizes)
    A = sp.block_diag([_block(kind, s, rng) for s in sizes], format="coo")
    rows, cols, vals = list(A.row), list(A.col), list(A.data)
    for j in range(border):
        for _ in range(rng.integers(0, 5)):  # some border columns and rows touch no block
            rows.append(int(rng.integers(nm)))
            cols.append(nm + j)
            vals.append(rng.uniform(-1.0, 1.0))
        for _ in range(rng.integers(0, 5)):
            rows.append(nm + j)
            cols.append(int(rng.integers(nm)))
            vals.append(rng.uniform(-1.0, 1.0))
    for _ in range(2 * border):
        rows.append(nm + int(rng.integers(border)))
        cols.append(nm + int(rng.integers(border)))
        vals.append(rng.uniform(-1.0, 1.0))
    for i in range(0, nm, max(1, nm // 40)):  # the last border row and column touch every block
        rows += [i, nm + border - 1]
        cols += [nm + border - 1, i]
        vals += list(rng.uniform(-1.0, 1.0, 2))
    n = nm + border
    S = sp.coo_matrix((vals, (rows, cols)), shape=(n, n)).tocsc()
    S.sum_duplicates()
    d = np.asarray(abs(S).sum(axis=0)).ravel() + np.asarray(abs(S).sum(axis=1)).ravel() + 1.0
    S = (S + sp.diags([d], [0])).tocsc()
    S.sort_indices()
    asg = np.concatenate([np.repeat(np.arange(len(sizes)), sizes), np.full(border, -1)])
    return S, asg.astype(np.int64)


CASES = [("sym", (40, 7, 90), 1), ("sym", (200, 150, 60, 33), 31), ("sym", (64, 65, 300), 33),
         ("unsym", (40, 7, 90), 32), ("unsym", (250, 120, 31), 70), ("unsym", (500, 400), 130),
         ("ladder", (12000, 100), 40), ("ladder", (30000, 2000), 20)]


@pytest.mark.parametrize("kind,sizes,border", CASES,
                         ids=[f"{k}{max(s)}b{b}" for k, s, b in CASES])
def test_bordered_systems(kind, sizes, border):
    rng = np.random.default_rng(border)
    A, asg = _system(kind, sizes, border, rng)
    g = BbdSolver(A.indptr.astype(np.int64), A.indices.astype(np.int64), asg, len(sizes))
    assert not g.info()["fallback"]
    b = rng.standard_normal(A.shape[0])
    for scale in (1.0, 1.25):  # a first factorization, then a refactorization
        B = A.copy()
        B.data = A.data * scale
        g.factor(B.data)
        x = b.copy()
        g.solve(x)
        ref = sla.spsolve(B, b)
        assert np.max(np.abs(x - ref)) <= 1e-12 * np.max(np.abs(ref))
