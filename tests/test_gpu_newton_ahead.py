"""The Newton loop launches an iteration before the one ahead of it is known to
end the loop; such an iteration must do nothing. The iterate, the reason and the
factorization counts of a loop with room for more iterations are those of a loop
that stops exactly there, for systems on both sides of the update over the grid
(4096 unknowns) and of the one-block refactorization, with and without gmin
steps, and for a loop ended by a non-finite iterate."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, newton_dc

pytestmark = pytest.mark.gpu


def _run(c, max_iters, gmin_steps):
    g = GpuKluSolver(1)
    r = newton_dc(g, DeviceCircuit(c), N.newton_config(**dict(wl.TIGHT, max_iters=max_iters,
                                                               gmin_steps=gmin_steps)))
    s = g.stats()
    return r, (s["factor_count"], s["refactor_count"])


@pytest.mark.parametrize("side,gmin_steps", [(3, 0), (4, 3), (16, 0), (20, 4), (66, 0)])
def test_room_for_more_iterations_changes_nothing(side, gmin_steps):
    c = cz.mesh_dc(side, max(1, side * side // 16))
    r, counts = _run(c, 100, gmin_steps)
    assert sum(counts) == r.iterations_total
    if gmin_steps:
        return
    reason, its, _ = po.dc_op(c, "nativeklu", **{k: wl.TIGHT[k] for k in (
        "max_iters", "abs_tol", "rel_tol", "gmin", "gmin_steps")})
    assert (r.reason, r.iterations) == (reason, its)
    if not r.converged:  # (the 3 x 3 mesh runs to the cap, in the oracle as well)
        return
    exact, counts_exact = _run(c, r.iterations, gmin_steps)
    assert exact.converged and counts_exact == counts
    assert np.array_equal(exact.x, r.x)
    short, counts_short = _run(c, r.iterations - 1, gmin_steps)
    assert not short.converged and sum(counts_short) == r.iterations - 1
    assert np.array_equal(_run(c, r.iterations - 1, gmin_steps)[0].x, short.x)


@pytest.mark.parametrize("side", [4, 66])
def test_a_non_finite_stop_leaves_the_iterate(side):
    c = cz.mesh_dc(side, 4)
    c.p[0, 0] = np.nan

    def run(max_iters):
        g = GpuKluSolver(1)
        g.set_stop_on_nonfinite(True)
        dc = DeviceCircuit(c)
        cfg = N.newton_config(**dict(wl.TIGHT, max_iters=max_iters))
        x, it = np.zeros(dc.n), C.c_int64()
        st = N.lib().gpuklu_newton_dc(g.handle, dc.handle, C.byref(cfg), None, N.ptr(x), dc.n,
                                      None, C.byref(it), None, None)
        return x, st, it.value, g.stats()["refactor_count"]

    (xa, sta, ita, ra), (xb, stb, itb, rb) = run(1), run(50)
    assert sta == stb == N.NONFINITE and ita == itb == 1 and ra == rb
    assert np.array_equal(xa, xb, equal_nan=True)


@pytest.mark.parametrize("diodes", [1, 9, 10, 11, 60])
def test_stamping_in_one_block(diodes):
    """Circuits of 1015 to 1074 devices, on both sides of the 1024 that one block
    stamps: the oracle's iterations and its solution at the DC bar (1e-10)."""
    c = cz.mesh_dc(23, diodes, seed=3)
    r, _ = _run(c, 100, 0)
    reason, its, x = po.dc_op(c, "nativeklu", **{k: wl.TIGHT[k] for k in (
        "max_iters", "abs_tol", "rel_tol", "gmin", "gmin_steps")})
    assert (r.reason, r.iterations) == (reason, its)
    assert np.max(np.abs(r.x - x)) <= 1e-10 * np.max(np.abs(x))
