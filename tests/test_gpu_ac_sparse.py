"""The AC sweep's sparse elimination (k_ac_sparse) against the oracle's dense
complex LU, bit for bit: system sizes around the 32-bit words of its entry
masks, patterns with fill, capacitances large enough that the ground column
loses its pivot to another row, frequency counts on both sides of the warps
rule, and values that overflow (the dense path of that frequency)."""
import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import netlist as nl

pytestmark = pytest.mark.gpu


def _grid(rows, cols, seed, cmax=1e-11, lone=()):
    rng = np.random.default_rng(seed)
    lines, k = ["V1 n0 0 DC 0 AC 1 30"], 0
    for r in range(rows):
        for c in range(cols):
            a = r * cols + c
            for b in ([a + 1] if c + 1 < cols else []) + ([a + cols] if r + 1 < rows else []):
                lines.append(f"R{k} n{a} n{b} {100.0 * 10.0 ** (2.0 * rng.random()):.6g}")
                k += 1
            lines.append(f"C{a} n{a} 0 {rng.uniform(0.01, 1.0) * cmax:.6g}")
    lines += list(lone)
    return nl.compile_deck("\n".join(lines) + "\n").circuit


def _same(c, f):
    from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, ac_sweep
    x0 = np.zeros(c.n)
    want = po.ac_sweep(c, x0, f)
    got = ac_sweep(GpuKluSolver(1), DeviceCircuit(c), x0, f)
    assert np.array_equal(got, want, equal_nan=True)
    return want


# n = rows * cols + 2: 3, 4, 31..34, 63..66 and larger grids with fill
@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 2), (1, 29), (5, 6), (1, 31), (4, 8), (1, 61),
                                       (2, 31), (7, 9), (8, 8), (9, 12), (16, 17)])
@pytest.mark.parametrize("cmax", [1e-11, 1e-7], ids=["small", "large"])
def test_sparse_elimination_matches_the_dense_lu(rows, cols, cmax):
    _same(_grid(rows, cols, rows * 100 + cols, cmax), np.array([1.0, 3e3, 2e6, 1e9, 7e9]))


@pytest.mark.parametrize("nf", [1, 150, 1300])
def test_frequency_counts(nf):
    _same(_grid(3, 5, nf), np.geomspace(10.0, 1e10, nf))


def test_overflowing_values_take_the_dense_path():
    # the square of omega C overflows at the second frequency only
    c = _grid(3, 4, 7, lone=["CX n5 n6 1e148"])
    y = _same(c, np.array([1e3, 1e9, 2e3]))
    assert np.all(np.isfinite(y[[0, 2]])) and not np.all(np.isfinite(y[1]))
