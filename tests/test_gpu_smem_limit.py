"""A kernel's dynamic shared-memory limit belongs to the process: handles of
other sizes on other threads, a newer batch of smaller circuits and a circuit
refused for its size leave the launches of the others as they were."""
import os
import subprocess
import sys

import numpy as np
import pytest

from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import waveforms as wf
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import ATranBatch, BbdSolver, DeviceCircuit, TranBatch
from test_gpu_launch_errors import solvers_on_threads

pytestmark = pytest.mark.gpu

CFG = dict(wl.TIGHT)


@pytest.mark.parametrize("sides,rounds", [((2, 3, 4, 6), 12000), ((2, 8, 16, 32), 6000)])
def test_handles_on_threads_do_not_lower_each_others_limit(sides, rounds):
    wrong, errors = solvers_on_threads(sides, rounds)
    assert not wrong and not errors, (len(wrong), len(errors), errors[:2])


def _tran(stages):
    cs = [cz.ring_oscillator(stages, seed=5, ring_id=i) for i in range(2)]
    xs = [wl.ring_initial_state(c) for c in cs]
    return TranBatch(cs, np.concatenate(xs), np.array([0, len(xs[0])]), wl.RING_DT, 8, 4,
                     wl.RING_PROBE, wl.RING_TARGET)


def _atran(stages):
    c = cz.inverter_chain(stages, 0.0, seed=13)
    return ATranBatch([c], [{1: wf.pulse(**wl.ATRAN_PULSE)}], [wl.chain_nodeset(stages, 0.0)],
                      np.array([c.node_count - 1]))


@pytest.mark.parametrize("small", [5, 101])
def test_an_older_larger_transient_runs_after_a_smaller_one(small):
    cfg = N.newton_config(**CFG)
    big = _tran(401)  # above a kernel's own 48 KB
    want = big.forward(cfg)
    grad, _ = big.backward(cfg)
    little = _tran(small)
    got = big.forward(cfg)
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[2], got[2])
    assert np.array_equal(np.concatenate(grad), np.concatenate(big.backward(cfg)[0]))
    little.forward(cfg)


@pytest.mark.parametrize("small", [5, 64])
def test_an_older_larger_adaptive_transient_runs_after_a_smaller_one(small):
    cfg = N.newton_config(max_iters=100, abs_tol=1e-9, rel_tol=1e-6, gmin=1e-12)
    run = dict(lte_abs=1e-6, lte_rel=1e-3, max_points=64)
    big = _atran(400)
    want = big.run(cfg, wl.ATRAN_TSTEP, 2e-11, **run)
    little = _atran(small)
    got = big.run(cfg, wl.ATRAN_TSTEP, 2e-11, **run)
    assert np.array_equal(want.x[0], got.x[0]) and want.npoints[0] == got.npoints[0]
    little.run(cfg, wl.ATRAN_TSTEP, 2e-11, **run)


REFUSED = """
import numpy as np
from rustspice_gb300 import circuits as cz, native as N, workloads as wl
from rustspice_gb300.solver import Batch
try:
    Batch([cz.mesh_dc(64, 64)], np.zeros(1, np.int64))
    raise SystemExit("accepted")
except RuntimeError:
    pass
b = Batch([cz.inverter_chain(256, 0.0, seed=3)], np.zeros(1, np.int64), np.ones(1, np.int64),
          np.zeros(1), wl.chain_nodeset(256, 0.0), np.zeros(1, np.int64))
b.run(N.newton_config(**wl.TIGHT))
assert b.results()[2][0] == 0
"""


def test_a_circuit_refused_for_its_size_leaves_the_next_batch_its_memory():
    """In a process of its own: no earlier batch has raised the limit."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", REFUSED], cwd=root, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


RISING = """
import numpy as np, scipy.sparse as sp
from rustspice_gb300.solver import GpuKluSolver

def check(a):
    a = sp.csc_matrix(a)
    a.sort_indices()
    n = a.shape[0]
    g, x = GpuKluSolver(n), np.ones(n)
    g.factor(a.indptr.astype(np.int64), a.indices.astype(np.int64), a.data)
    g.solve(x)
    assert np.abs(a @ x - 1.0).max() < 1e-10, n

for n in range(%d, %d):
    if %d:  # the last column holds n values
        a = sp.lil_matrix(sp.diags([4.0 * n], shape=(n, n)))
        a[n - 1, :n - 1] = -1.0
        a[:n - 1, n - 1] = -1.0
    else:
        a = sp.diags([-1.0, 4.0, -1.0], [-1, 0, 1], shape=(n, n))
    check(a)
"""


@pytest.mark.parametrize("lo,hi,arrow", [(690, 732, 1), (16, 515, 0)])
def test_sizes_that_rise_through_a_kernels_own_limit(lo, hi, arrow):
    """A kernel's own limit is 48 KB less its declared shared memory. Sizes
    that rise by a row at a time pass every one of the bytes between (columns
    of 704 to 720 slots in the grid refactorization), each in a launch that is
    the largest so far. Diagonally dominant systems: the residual is rounding,
    some 1e-13 at the most."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RISING % (lo, hi, arrow)], cwd=root,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_bordered_solvers_of_two_sizes():
    cfg = N.newton_config(**CFG)
    work = []
    for blocks, border, side in ((3, 900, 40), (3, 24, 8)):
        c, asg, nb = cz.bordered_meshes(blocks, border, side, side, 4)
        dc = DeviceCircuit(c)
        ap, ai = dc.pattern()
        work.append((BbdSolver(ap, ai, asg, nb), dc, wl.bordered_nodeset(c)))
    first = [b.newton_dc(dc, cfg, x0=x0).x for b, dc, x0 in work]
    again = [b.newton_dc(dc, cfg, x0=x0).x for b, dc, x0 in work]
    assert all(np.array_equal(p, q) for p, q in zip(first, again))
