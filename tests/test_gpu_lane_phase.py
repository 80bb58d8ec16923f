"""The batch's lane kernel (one instance per lane) in front of the others: as the
first iterations of classes of small programs with many instances, parked at the
iteration cap and finished by the warp-per-instance kernel, and in front of the
warp classes. The lane kernel's order of additions is the warp-per-instance
kernel's in those iterations, so which of them runs them does not show in the
results: bit for bit, with one and with two instances per warp."""
import itertools

import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import Batch

pytestmark = pytest.mark.gpu


def _meshes(sides, per):
    cs = [cz.mesh_dc(s, s, seed=i + 1) for i, s in enumerate(sides)]
    ic = np.repeat(np.arange(len(cs)), per)
    dev = np.array([cs[i].device_index(cz.DEV_V) for i in ic])
    return cs, ic, dev, np.tile(np.linspace(0.2, 1.2, per), len(cs)), None, None


def _chains(stages, per):
    cs = [cz.inverter_chain(s, 0.0, seed=3, chain_id=i) for i, s in enumerate(stages)]
    ic = np.repeat(np.arange(len(cs)), per)
    vin = np.tile(cz.vin_points(per), len(cs))
    x0 = [wl.chain_nodeset(stages[i], v) for i, v in zip(ic, vin)]
    off = np.concatenate([[0], np.cumsum([len(x) for x in x0])[:-1]])
    return cs, ic, np.ones(len(ic), np.int64), vin, np.concatenate(x0), off


INPUTS = {"meshes": lambda: _meshes((2, 3, 4, 5), 13), "chains": lambda: _chains((2, 5, 40, 9), 61),
          "one": lambda: _meshes((3,), 1)}


@pytest.mark.parametrize("kind", list(INPUTS))
@pytest.mark.parametrize("cap", ["1", "6"])
@pytest.mark.parametrize("over", [{}, {"max_iters": 4}, {"gmin_steps": 3, "max_iters": 9}],
                         ids=["plain", "short", "gmin"])
def test_the_lane_phase_does_not_show(kind, cap, over, monkeypatch):
    monkeypatch.setenv("GPUKLU_LANE_CAP", cap)
    args = INPUTS[kind]()
    out = []
    for lanes, m in itertools.product("01", "12"):
        monkeypatch.setenv("GPUKLU_LANE_PHASE", lanes)
        monkeypatch.setenv("GPUKLU_CONT_M", m)
        b = Batch(*args)
        assert b.info()["cont_kernel"]
        for _ in range(2):  # the counters are reset between runs
            b.run(N.newton_config(**dict(wl.TIGHT, **over)))
        out.append(b.results())
        b.close()
    for got in out[1:]:
        assert all(np.array_equal(p, q, equal_nan=True) for p, q in zip(out[0], got))


def test_many_small_circuits_start_in_the_lane_kernel(monkeypatch):
    """610 3 x 3 meshes x 32 inputs are above the line, the same with 3 inputs
    below it."""
    cfg = N.newton_config(**wl.TIGHT)
    args = _meshes((3,) * 610, 32)
    b = Batch(*args)
    b.run(cfg)
    launches, ms, got = b.info()["launches"], b.phase_ms()["lanes_ms"], b.results()
    b.close()
    monkeypatch.setenv("GPUKLU_LANE_PHASE", "0")
    r = Batch(*args)
    r.run(cfg)
    assert launches == r.info()["launches"] + 1 and ms > 0.1
    assert all(np.array_equal(p, q) for p, q in zip(got, r.results()))
    r.close()
    monkeypatch.delenv("GPUKLU_LANE_PHASE")
    few = Batch(*_meshes((3,) * 610, 3))
    assert few.info()["launches"] == launches - 1
    few.close()


def test_the_lane_kernel_in_front_of_the_warp_classes(monkeypatch):
    """The warp-per-instance kernel switched off, against the oracle."""
    monkeypatch.setenv("GPUKLU_CONT_KERNEL", "0")
    B = wl.inverter_batch(12, 61, seed=11)
    it_o, rs_o, x_o = po.dc_batch(B.circuits, B.inst_circ, B.inst_dev, B.inst_val,
                                  "nativeklu_exact", nthreads=4,
                                  x_cap=max(c.n for c in B.circuits), x0=B.x0, x0_off=B.x0_off,
                                  **{k: v for k, v in wl.TIGHT.items()
                                     if k in ("max_iters", "abs_tol", "rel_tol", "gmin",
                                              "gmin_steps")})
    for cap in ("1", "6"):
        monkeypatch.setenv("GPUKLU_LANE_CAP", cap)
        b = Batch(B.circuits, B.inst_circ, B.inst_dev, B.inst_val, B.x0, B.x0_off)
        b.run(N.newton_config(**wl.TIGHT))
        ph = b.phase_ms()
        assert not b.info()["cont_kernel"] and ph["lane_cap"] == int(cap) and ph["lanes_ms"] > 0.1
        it, _, rs, x = b.results()
        conv = rs_o == 0
        assert np.array_equal(rs == 0, conv) and np.mean(it[conv] == it_o[conv]) > 0.98
        for i in np.flatnonzero(conv):
            n = B.circuits[B.inst_circ[i]].n
            xg, xo = x[b.x_off[i]:b.x_off[i] + n], x_o[i, :n]
            assert np.max(np.abs(xg - xo)) <= 1e-10 * max(1.0, np.max(np.abs(xo))), i
        b.close()
