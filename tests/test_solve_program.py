"""The program the single-system solve runs (gpuklu_plan_solve_program: rows of
slots, chains, segments, chunks), forward and transpose, interpreted on the CPU
as the kernel runs it: what stands between two barriers reads the values from
before it and is checked not to touch what another operation there writes.
Forward, bit for bit the device solve (the row-oriented emulation that the
plan-parity tests pin to the oracle); transpose, bit for bit the column sweeps
of the factors' transpose, and in the exact mode a dense solve to 1e-9."""
import numpy as np
import pytest
import scipy.sparse as sp

from plan_emulator import EmulatedSolver, first_factor, solve
from rustspice_gb300 import native as N
from test_step_program import STEP_SYSTEMS

SOLO, WIDE, CHAIN = 0, 1, 2


def _csc(A, rng):
    A = sp.csc_matrix(A)
    A.sort_indices()
    return (A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy(),
            rng.standard_normal(A.shape[0]))


def _arrow(n, band, seed):
    """Dense last row and column and `band` off-diagonals (none: a chain)."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for k in range(1, band + 1):
        A += np.diag(rng.uniform(0.1, 1.0, n - k), k) + np.diag(rng.uniform(0.1, 1.0, n - k), -k)
    A[n - 1, :] = rng.uniform(-1, 1, n)
    A[:, n - 1] = rng.uniform(-1, 1, n)
    A[np.arange(n), np.arange(n)] = rng.uniform(4.0, 5.0, n) + 2 * band
    A[n - 1, n - 1] = 2.0 * n
    return _csc(A, rng)


def _coupled(blocks, size, upper, seed):
    """Diagonal blocks with coupling entries on one side, rows and columns
    shuffled: several BTF blocks."""
    rng = np.random.default_rng(seed)
    n = blocks * size
    A = np.kron(np.eye(blocks), np.ones((size, size))) * rng.uniform(-1, 1, (n, n))
    C = rng.uniform(-1, 1, (n, n)) * (rng.random((n, n)) < 0.05)
    A += (np.triu if upper else np.tril)(C, size if upper else -size)
    A[np.arange(n), np.arange(n)] = rng.uniform(4.0, 5.0, n) + size
    return _csc(A[rng.permutation(n)][:, rng.permutation(n)], rng)


SYSTEMS = STEP_SYSTEMS + [
    ("arrow40", *_arrow(40, 1, 1)), ("arrow300", *_arrow(300, 0, 2)), ("arrow2", *_arrow(2, 0, 3)),
    ("upper", *_coupled(25, 4, True, 4)), ("lower", *_coupled(25, 4, False, 5)),
    ("diagonal", *_csc(np.diag(np.random.default_rng(6).uniform(1, 2, 300)),
                       np.random.default_rng(6)))]


def _together(T, ops, lu, ax):
    """The operations between two barriers, each on the values from before."""
    dst = [o[0] for o in ops]
    assert len(set(dst)) == len(dst)
    for d, s, v, k in ops:
        assert s == d or s not in dst
    new = [T[d] / lu[v] if k == 1 else T[d] - (ax[v] if k == 2 else lu[v]) * T[s]
           for d, s, v, k in ops]
    for d, v in zip(dst, new):
        T[d] = v


def run_program(pr, T, lu, ax):
    chunk, width = (int(v) for v in pr["info"][0])
    ops, segs = pr["ops"].tolist(), pr["segs"].tolist()
    n_ops, n_seg, wide = 0, 0, []
    for s0, ns, g0, ng in pr["chunks"].tolist():
        assert s0 == n_ops and g0 == n_seg and ns <= chunk and 0 < ng <= 64
        at = s0
        for x, first in segs[g0:g0 + ng]:
            kind, cnt = x & 3, x >> 2
            assert kind == WIDE or not wide  # a step's wide rows end before anything else
            if kind == CHAIN:
                chains = pr["chains"][first:first + cnt].tolist()
                rows = {c[0] for c in chains}
                assert len(rows) == cnt
                new = []
                for d, t0, nt, _ in chains:
                    v = T[d]
                    for src, z in pr["terms"][t0:t0 + nt].tolist():
                        assert src not in rows
                        v = v - (ax[~z] if z < 0 else lu[z]) * T[src]
                    new.append(v)
                for c, v in zip(chains, new):
                    T[c[0]] = v
                continue
            w = 32 if kind == SOLO else width
            for _ in range(cnt):
                row = ops[at:at + w]
                at += w
                assert len({o[3] >> 2 for o in row}) == 1
                live = [(d, s, v, k & 3) for d, s, v, k in row if k & 3 != 3]
                assert bool(row[0][3] & 4) == any(o[3] == 1 for o in live)
                assert all(o[0] == o[1] for o in live if o[3] == 1)
                wide += live
                if kind == SOLO or row[0][3] & 8:
                    _together(T, wide, lu, ax)
                    wide = []
        assert at == s0 + ns
        n_ops, n_seg = s0 + ns, g0 + ng
    assert n_ops == len(ops) and n_seg == len(segs) and not wide
    return T


def _transpose_sweeps(P, ax, lu, g):
    T = np.zeros(P.n)
    T[P.out_pos] = g
    blocks = range(P.nblocks)
    for b in (reversed(blocks) if P.offd_lower else blocks):
        b0, b1 = int(P.block_ptr[b]), int(P.block_ptr[b + 1])
        for k in range(b0, b1):
            for i in range(P.n):
                for e in range(P.offd_ptr[i], P.offd_ptr[i + 1]):
                    if P.offd_col[e] == k:
                        T[k] = T[k] - ax[P.offd_raw[e]] * T[i]
            for q in range(P.col_ptr[k], P.dslot[k]):
                T[k] = T[k] - lu[q] * T[P.slot_row[q]]
            T[k] = T[k] / lu[P.dslot[k]]
        for k in range(b1 - 1, b0 - 1, -1):
            for e in range(P.lrow_ptr[k], P.lrow_ptr[k + 1]):
                c = P.lrow_col[e]
                T[c] = T[c] - lu[P.lrow_slot[e]] * T[k]
    return T[P.in_pos]


@pytest.mark.parametrize("mode", [N.PIVOT_REFERENCE, N.PIVOT_EXACT], ids=["reference", "exact"])
@pytest.mark.parametrize("sysm", SYSTEMS, ids=[s[0] for s in SYSTEMS])
def test_the_uploaded_program(sysm, mode):
    name, ap, ai, ax, rhs = sysm
    n = len(ap) - 1
    ax, rhs = np.asarray(ax, np.float64), np.asarray(rhs, np.float64)
    es = EmulatedSolver(mode)
    es.factor(n, ap, ai, ax)
    P, lu = es.plan, es.lu
    _, rperm = first_factor(N.Plan(n, ap, ai, mode), ax)
    a = np.zeros((n, n))
    for j in range(n):
        for t in range(ap[j], ap[j + 1]):
            a[ai[t], j] += ax[t]
    for transpose in (False, True):
        pr = N.solve_program(n, ap, ai, transpose, mode, rperm)
        plain = pr["ops"][(pr["ops"][:, 3] & 3) != 3]
        assert np.sum((plain[:, 3] & 3) == 1) == n  # one pivot division per row
        T = np.zeros(n + 1)
        T[(P.out_pos if transpose else P.in_pos)] = rhs
        got = run_program(pr, T, lu, ax)[(P.in_pos if transpose else P.out_pos)]
        want = _transpose_sweeps(P, ax, lu, rhs) if transpose else solve(P, ax, lu, rhs)
        assert np.array_equal(got, want), (name, transpose, np.max(np.abs(got - want)))
        # (the reference's mode drops what its row swaps move outside the pattern)
        if mode == N.PIVOT_EXACT and name in ("arrow300", "upper", "lower", "arrow40"):
            ref = np.linalg.solve(a.T if transpose else a, rhs)
            assert np.max(np.abs(got - ref)) <= 1e-9 * np.max(np.abs(ref))
        if name == "arrow300":
            assert len(pr["chains"]) > 0
        if mode == N.PIVOT_EXACT and name in ("upper", "lower"):
            assert P.noffdiag > 0


@pytest.mark.parametrize("n,chunk", [(22000, 1024), (26500, 256), (28000, 128), (28600, 32),
                                     (28900, 0)])
def test_chunks_by_size(n, chunk):
    ap, ai = np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int64)
    pr = N.solve_program(n, ap, ai)
    assert (pr is None) if chunk == 0 else int(pr["info"][0, 0]) == chunk
