"""Small AC systems with several warps a frequency (few frequencies), against the
oracle's dense complex LU bit for bit: fully coupled networks and ladders with
fewer unknowns than threads, and the frequency counts where the warps change."""
import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import netlist as nl
from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, ac_sweep

pytestmark = pytest.mark.gpu


def _deck(n, full):
    rng = np.random.default_rng(n)
    lines = ["V1 n0 0 DC 0 AC 1 30"]
    for a in range(n):
        for b in range(a) if full else [a - 1] * (a > 0):
            lines.append(f"R{a}_{b} n{a} n{b} {100.0 * 10.0 ** (2.0 * rng.random()):.6g}")
        lines.append(f"C{a} n{a} 0 {rng.uniform(1e-13, 1e-9):.6g}")
    return nl.compile_deck("\n".join(lines) + "\n").circuit


# a device of 152 SMs: 8, 4, 2 and 1 warps to 303, 607, 1215 frequencies and beyond
@pytest.mark.parametrize("nf", [1, 5, 303, 304, 608, 1216])
@pytest.mark.parametrize("n,full", [(1, True), (2, True), (7, True), (31, True), (60, True), (40, False)])
def test_small_systems(n, full, nf):
    if nf > 5 and n > 31:
        nf = 5
    c = _deck(n, full)
    f = np.geomspace(1.0, 1e10, nf)
    want = po.ac_sweep(c, np.zeros(c.n), f)
    got = ac_sweep(GpuKluSolver(1), DeviceCircuit(c), np.zeros(c.n), f)
    assert np.array_equal(got, want)
