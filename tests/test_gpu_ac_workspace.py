"""The AC sweep's device workspace: with the scratch held to one matrix the
sweep gives the same bits, and the handle keeps no more than that."""
import numpy as np
import pytest

from rustspice_gb300 import netlist as nl
from rustspice_gb300.solver import DeviceCircuit, GpuKluSolver, ac_sweep

pytestmark = pytest.mark.gpu


def _ladder(n):
    rng = np.random.default_rng(n)
    lines = ["V1 n0 0 DC 0 AC 1 30"]
    for k in range(n):
        lines.append(f"R{k} n{k} n{k + 1} {rng.uniform(100, 1000):.6g}")
        lines.append(f"C{k} n{k + 1} 0 {rng.uniform(1e-12, 1e-9):.6g}")
    return nl.compile_deck("\n".join(lines) + "\n").circuit


@pytest.mark.parametrize("n,nf", [(5, 40), (100, 3000), (300, 400)])
@pytest.mark.parametrize("scratch", ["1", "3000000"])
def test_scratch_limit(n, nf, scratch, monkeypatch):
    import torch
    c = _ladder(n)
    f = np.geomspace(1.0, 1e9, nf)
    dc = DeviceCircuit(c)
    g = GpuKluSolver(1)
    want = ac_sweep(g, dc, np.zeros(c.n), f)
    g.close()
    monkeypatch.setenv("GPUKLU_AC_SCRATCH", scratch)
    h = GpuKluSolver(1)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    got = ac_sweep(h, dc, np.zeros(c.n), f)
    kept = free - torch.cuda.mem_get_info()[0]
    assert np.array_equal(got, want)
    # one matrix or 3 MB of them, the results, the inputs (allocations come in 2 MB)
    assert kept <= max(int(scratch), 16 * c.n ** 2) + 16 * nf * c.n + (8 << 20), kept
    h.close()
