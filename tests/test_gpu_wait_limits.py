"""Waits of a block's warps on one another that run out (the refactorization's
loader and computing warps, the step-program solve's copying and compute
warps): the call reports DEVICE_TIMEOUT, never a result that was not finished,
and the kernel ends. A short limit of polls makes the
waits run out; with the default limit the same handle factors as before."""
import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, SolverError, newton_dc

pytestmark = pytest.mark.gpu


def _system(kind):
    if kind == "diagonal":  # no column waits for another: the pairs' waits alone
        n = 4000
        rng = np.random.default_rng(3)
        return (n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int64),
                rng.uniform(1.0, 2.0, n), rng.standard_normal(n))
    c = cz.mesh_dc(32, 64)
    return po.mna(c, np.zeros(c.node_count))


@pytest.mark.parametrize("kind", ["diagonal", "mesh"])
@pytest.mark.parametrize("polls", [1, 4, 64])
def test_a_pair_that_gives_up_is_reported(kind, polls, monkeypatch):
    monkeypatch.setenv("GPUKLU_ONE_BLOCK", "0")
    n, ap, ai, ax, rhs = _system(kind)
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    for _ in range(2):
        g.factor(ap, ai, ax)
    want = rhs.copy()
    g.solve(want)
    monkeypatch.setenv("GPUKLU_PAIR_POLLS", str(polls))
    g.set_spin_limit(0)  # takes the limits
    gave_up = 0
    for k in range(12):
        monkeypatch.setenv("GPUKLU_PAIR_POLLS", str(polls))
        g.set_spin_limit(0)
        try:
            g.factor(ap, ai, ax * 2.0)
        except SolverError as e:
            assert e.status == N.DEVICE_TIMEOUT, e
            gave_up += 1
            continue
        x = rhs * 2.0
        g.solve(x)
        assert np.array_equal(x, want)
    if polls == 1:
        assert gave_up > 0, "no wait ran out at one poll"
    monkeypatch.delenv("GPUKLU_PAIR_POLLS")
    g.set_spin_limit(0)
    g.factor(ap, ai, ax)
    x = rhs.copy()
    g.solve(x)
    assert np.array_equal(x, want)
    g.close()


def test_the_newton_loop_ends_on_it(monkeypatch):
    monkeypatch.setenv("GPUKLU_ONE_BLOCK", "0")
    cfg = N.newton_config(**dict(wl.TIGHT, gmin_steps=4))
    g, dc = GpuKluSolver(1), DeviceCircuit(cz.mesh_dc())
    ok = newton_dc(g, dc, cfg)
    monkeypatch.setenv("GPUKLU_PAIR_POLLS", "1")
    g.set_spin_limit(0)
    with pytest.raises(SolverError) as e:
        newton_dc(g, dc, cfg)
    assert e.value.status == N.DEVICE_TIMEOUT
    monkeypatch.delenv("GPUKLU_PAIR_POLLS")
    g.set_spin_limit(0)
    again = newton_dc(g, dc, cfg)
    assert again.iterations == ok.iterations and np.array_equal(again.x, ok.x)


@pytest.mark.parametrize("polls", [1, 4, 64, 4096])
def test_a_staged_solve_that_gives_up_is_reported(polls, monkeypatch):
    """The step program with its slots copied in bulk: the compute warps wait
    for a chunk, the copying warp for a free half."""
    monkeypatch.setenv("GPUKLU_SOLVE_STAGED", "0")
    n, ap, ai, ax, rhs = _system("mesh")
    g = GpuKluSolver(n, pivot_mode=N.PIVOT_EXACT)
    g.factor(ap, ai, ax)
    want = {}
    for t in (False, True):
        want[t] = rhs.copy()
        (g.tsolve if t else g.solve)(want[t])
    monkeypatch.setenv("GPUKLU_PAIR_POLLS", str(polls))
    g.set_spin_limit(0)
    gave_up = 0
    for k in range(12):
        x = rhs.copy()
        try:
            (g.tsolve if k % 2 else g.solve)(x)
        except SolverError as e:
            assert e.status == N.DEVICE_TIMEOUT, e
            gave_up += 1
            continue
        assert np.array_equal(x, want[bool(k % 2)])
    if polls == 1:
        assert gave_up > 0, "no wait ran out at one poll"
    monkeypatch.delenv("GPUKLU_PAIR_POLLS")
    g.set_spin_limit(0)
    for t in (False, True):
        x = rhs.copy()
        (g.tsolve if t else g.solve)(x)
        assert np.array_equal(x, want[t])
    g.close()
