"""Calls of the CUDA runtime that it refuses: a call whose kernel was not
launched reports it, and a call is not failed by what an earlier one was
refused. Nothing here runs a kernel that faults."""
import ctypes
import threading

import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import (BbdSolver, DeviceCircuit, GpuKluSolver, SolverError, TranBatch,
                                    dc_backward, newton_dc)

pytestmark = pytest.mark.gpu


def solvers_on_threads(sides, rounds):
    """One solver per mesh side, each factoring and solving in a loop on a
    thread of its own. Returns (results other than the handle's own when it
    runs alone, errors raised)."""
    work = []
    for side in sides:
        c = cz.mesh_dc(side, side)
        n, ap, ai, ax, rhs = po.mna(c, np.zeros(c.node_count))
        g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
        want = []
        for k in range(4):  # the second factorization on refactors
            g.factor(ap, ai, ax * (1 + k % 2))
            x = rhs.copy()
            (g.tsolve if k % 4 == 3 else g.solve)(x)
            want.append(x)
        want[0] = want[2]
        work.append((g, ap, ai, ax, rhs, want))
    wrong, errors = [], []
    start = threading.Barrier(len(sides))

    def loop(g, ap, ai, ax, rhs, want):
        start.wait()
        for k in range(rounds):
            try:
                g.factor(ap, ai, ax * (1 + k % 2))
                x = rhs.copy()
                (g.tsolve if k % 4 == 3 else g.solve)(x)
                if not np.array_equal(x, want[k % 4]):
                    wrong.append((len(rhs), k))
            except SolverError as e:
                errors.append(str(e))

    ts = [threading.Thread(target=loop, args=w) for w in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for w in work:
        w[0].close()
    return wrong, errors


@pytest.mark.parametrize("sides,rounds", [((2, 3, 4, 6), 12000), ((2, 8, 16, 32), 6000)])
def test_a_refused_launch_is_reported(sides, rounds):
    """Handles of different sizes on several threads: a call has the handle's
    own result, or it raises."""
    wrong, _ = solvers_on_threads(sides, rounds)
    assert not wrong, (len(wrong), wrong[:5])


def test_a_refused_allocation_does_not_fail_the_next_call():
    """A transient whose checkpoints no device holds (400 GB) is refused at its
    allocation; a factorization, a solve and an operating point on the same
    thread, each after such a refusal, run."""
    r = cz.ring_oscillator(3, seed=5, ring_id=0)
    x0 = wl.ring_initial_state(r)
    c = cz.mesh_dc(8, 8)
    n, ap, ai, ax, rhs = po.mna(c, np.zeros(c.node_count))
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    g.factor(ap, ai, ax)
    want = rhs.copy()
    g.solve(want)
    h, dc = GpuKluSolver(1, pivot_mode=N.PIVOT_EXACT), DeviceCircuit(c)

    def refused():
        with pytest.raises(RuntimeError):
            TranBatch([r], x0, np.zeros(1, np.int64), wl.RING_DT, 10 ** 10, 1, wl.RING_PROBE,
                      wl.RING_TARGET)

    refused()
    g.factor(ap, ai, ax)
    refused()
    x = rhs.copy()
    g.solve(x)
    assert np.array_equal(x, want)
    refused()
    assert newton_dc(h, dc, N.newton_config(**wl.TIGHT)).converged


def test_an_error_left_by_other_code_does_not_fail_a_call():
    """The thread's last error as another user of the CUDA runtime leaves it (a
    device number that does not exist) before each call."""
    rt = ctypes.CDLL("libcudart.so.13")
    c = cz.mesh_dc(8, 8)
    n, ap, ai, ax, rhs = po.mna(c, np.zeros(c.node_count))
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    h, dc = GpuKluSolver(1, pivot_mode=N.PIVOT_EXACT), DeviceCircuit(c)
    cb, asg, nb = cz.bordered_meshes(3, 24, 8, 8, 4)
    dcb = DeviceCircuit(cb)
    b = BbdSolver(*dcb.pattern(), asg, nb)
    cfg = N.newton_config(**wl.TIGHT)
    out = {}

    def solve(f):
        x = rhs.copy()
        f(x)
        return x

    calls = {"factor": lambda: g.factor(ap, ai, ax), "refactor": lambda: g.factor(ap, ai, ax),
             "solve": lambda: solve(g.solve), "tsolve": lambda: solve(g.tsolve),
             "newton": lambda: newton_dc(h, dc, cfg).x,
             "adjoint": lambda: dc_backward(h, dc, out["newton"], np.ones(dc.n))[0],
             "bordered": lambda: b.newton_dc(dcb, cfg, x0=wl.bordered_nodeset(cb)).x}
    for name, call in calls.items():
        assert rt.cudaSetDevice(4096) != 0 and rt.cudaPeekAtLastError() != 0
        out[name] = call()
        assert rt.cudaPeekAtLastError() == 0, name
        again = call()
        assert out[name] is None or np.array_equal(out[name], again), name
