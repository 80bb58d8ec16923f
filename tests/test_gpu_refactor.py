"""The refactorization kernels at the edges of their layout: columns whose L
part ends just before, at and behind a row of lanes and a piece of 64 slots,
hubs with hundreds of entries, a column longer than shared memory holds, sizes
on both sides of the one-block rule, and values (zeros, exact quotients, scales
up to 1e+-140) on both sides of the fixed-point division's range. Factor and
solve bit for bit against the oracle: the operations and their order are its
own."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import GpuKluSolver

pytestmark = pytest.mark.gpu


def _dense(n, rng):
    return sp.csc_matrix(rng.uniform(-1.0, 1.0, (n, n)) + np.diag(np.full(n, 2.0 * n)))


def _arrow(n, rng):
    A = sp.diags([rng.uniform(1.0, 2.0, n)], [0]).tolil()
    A[n - 1, :] = rng.uniform(-1.0, 1.0, n)
    A[:, n - 1] = rng.uniform(-1.0, 1.0, (n, 1))
    A[n - 1, n - 1] = 2.0 * n
    return A.tocsc()


def _blocks(k, rng):
    """Dense blocks of unequal size under one hub row and column."""
    sizes = [1 + (7 * i) % k for i in range(40)]
    A = sp.block_diag([_dense(s, rng) for s in sizes] + [sp.csc_matrix([[4.0]])]).tolil()
    n = A.shape[0]
    cols = rng.permutation(n - 1)[: n // 2]
    A[n - 1, cols] = rng.uniform(-1.0, 1.0, len(cols))
    A[cols, n - 1] = rng.uniform(-1.0, 1.0, (len(cols), 1))
    A[n - 1, n - 1] = 4.0 * n
    return A.tocsc()


def _integers(n, rng):
    """Small integers: zeros and exact quotients among the L values."""
    A = rng.integers(-1, 2, (n, n)).astype(float)
    A[rng.uniform(size=(n, n)) < 0.7] = 0.0
    return sp.csc_matrix(A + np.diag(np.full(n, 8.0)))


def _scaled(n, rng, e):
    A = _dense(n, rng)
    d = 10.0 ** rng.uniform(-e, e, n)
    return sp.csc_matrix(sp.diags([d], [0]) @ A @ sp.diags([1.0 / d], [0])
                         if e < 100 else sp.diags([d], [0]) @ A)


CASES = ([("dense", n) for n in (1, 2, 8, 9, 31, 32, 33, 34, 63, 64, 65, 66, 97, 130, 200)]
         + [("arrow", n) for n in (3, 64, 65, 300, 5000)]
         + [("blocks", k) for k in (3, 33, 70)] + [("integers", n) for n in (12, 40, 90)]
         + [("scaled", e) for e in (20, 60, 140)])


@pytest.mark.parametrize("one_block", ["", "0"], ids=["rule", "grid"])
@pytest.mark.parametrize("kind,size", CASES, ids=[f"{k}{s}" for k, s in CASES])
def test_refactor_edges(kind, size, one_block, monkeypatch):
    if one_block:
        monkeypatch.setenv("GPUKLU_ONE_BLOCK", one_block)
    rng = np.random.default_rng(size)
    A = {"dense": lambda: _dense(size, rng), "arrow": lambda: _arrow(size, rng),
         "blocks": lambda: _blocks(size, rng), "integers": lambda: _integers(size, rng),
         "scaled": lambda: _scaled(70, rng, size)}[kind]()
    A.sort_indices()
    n = A.shape[0]
    ap, ai = A.indptr.astype(np.int64), A.indices.astype(np.int64)
    b = rng.standard_normal(n)
    o = po.Solver("nativeklu_exact", n)
    o.prepare(n)
    o.analyze(ap, ai)
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    for ax in (A.data.copy(), A.data * rng.uniform(0.9, 1.1, A.nnz)):
        o.factor(ap, ai, ax)
        g.factor(ap, ai, ax)
        x = b.copy()
        g.solve(x)
        assert np.array_equal(x, o.solve(b)[1], equal_nan=True)


@pytest.mark.parametrize("stages", [3, 9, 10, 11, 12, 30, 61])
@pytest.mark.parametrize("mode", ["nativeklu", "nativeklu_exact"])
def test_pivot_pass_rule(stages, mode, monkeypatch):
    """Pivots found as refactorizations (from 16 rows on) and by the sequential
    kernel: the same factors, the oracle's."""
    c = cz.inverter_chain(stages, 0.55)
    n, ap, ai, ax, rhs = po.mna(c, wl.chain_nodeset(stages, 0.55))
    o = po.Solver(mode, n)
    o.prepare(n)
    o.analyze(ap, ai)
    o.factor(ap, ai, ax)
    want = o.solve(rhs)[1]
    for env in ("", "sequential"):
        if env:
            monkeypatch.setenv("GPUKLU_PIVOT_PASS", env)
        g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT if mode.endswith("exact")
                         else N.PIVOT_REFERENCE)
        g.factor(ap, ai, ax)
        x = rhs.copy()
        g.solve(x)
        assert np.array_equal(x, want)
        if env or n < 16:
            assert g.pivot_passes() == 0
