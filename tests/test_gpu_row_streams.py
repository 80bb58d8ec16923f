"""The row streams of the batched and transient kernels at the edges of their
layout: steps of one operation up to several rows of 16 and of 32 lanes (meshes
and stars), runs of dependent operations (ladders), value lists from one record
to more than a warp adds together (a star's hub and the supply), and programs
so unequal that they fall into several classes. The arithmetic of an instance
does not depend on how many share a warp, nor, in the first iterations, on
whether the lane-per-instance kernel ran them: bit for bit. The operating
points against the oracle at the batch's bar (1e-10 of the largest entry), the
transients and their gradients at theirs (1e-9, 1e-7)."""
import numpy as np
import pytest

from oracle import pyoracle as po
from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import Batch, TranBatch

pytestmark = pytest.mark.gpu


def _build(dev, nodes, caps):
    if caps:
        for a in range(1, nodes):
            dev.add(cz.DEV_C, (a, 0), (1e-14 * (1.0 + 0.1 * (a % 7)),))
    return dev.build(nodes)


def _star(k, caps=False):
    """A hub with k leaves, every fourth loaded by a diode; device 0 is the source."""
    rng = np.random.default_rng(k)
    dev = cz._Dev()
    dev.add(cz.DEV_V, (1, 0), (0.5,))
    dev.add(cz.DEV_R, (1, 2), (100.0,))
    for i in range(k):
        dev.add(cz.DEV_R, (2, 3 + i), (float(rng.uniform(1e3, 1e4)) * k,))
        dev.add(cz.DEV_R, (3 + i, 0), (float(rng.uniform(1e3, 1e4)) * k,))
        if i % 4 == 0:
            dev.add(cz.DEV_D, (3 + i, 0), (1e-14, 1.0))
    return _build(dev, 3 + k, caps)


def _mesh(rows, cols, caps=False):
    """A resistor mesh driven at a corner, diodes on every fifth node."""
    dev = cz._Dev()
    dev.add(cz.DEV_V, (1, 0), (0.5,))
    nid = cz._mesh_resistors(dev, rows, cols, 1, cz.Stream(rows * 64 + cols, 1))
    dev.add(cz.DEV_R, (nid(rows - 1, cols - 1), 0), (1000.0,))
    for a in range(2, rows * cols + 1, 5):
        dev.add(cz.DEV_D, (a, 0), (1e-14, 1.0))
    return _build(dev, rows * cols + 1, caps)


SHAPES = {
    "stars": lambda caps: [_star(k, caps) for k in (1, 2, 15, 16, 17, 31, 32, 33, 65, 200)],
    "ladders": lambda caps: [_mesh(1, k, caps) for k in (2, 3, 16, 17, 33, 64, 150)],
    "meshes": lambda caps: [_mesh(k, k, caps) for k in (2, 3, 4, 6, 8, 11)],
    "unequal": lambda caps: [_mesh(1, 3, caps), _mesh(10, 10, caps), _star(40, caps),
                             _mesh(1, 90, caps), _mesh(2, 2, caps), _mesh(5, 5, caps)],
}


def _run(circuits, per, monkeypatch, max_iters=100, **env):
    for k in ("GPUKLU_CONT_M", "GPUKLU_CONT_KERNEL"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    ic = np.repeat(np.arange(len(circuits)), per)
    val = np.tile(np.linspace(0.1, 0.5, per), len(circuits))
    bt = Batch(circuits, ic, np.zeros(len(ic)), val)
    bt.run(N.newton_config(**dict(wl.TIGHT, max_iters=max_iters)))
    info = bt.info()
    assert info["cont_kernel"] == (env.get("GPUKLU_CONT_KERNEL") != "0")
    return bt, ic, val, bt.results()


@pytest.mark.parametrize("shape", SHAPES)
def test_batch_bits_and_oracle(shape, monkeypatch):
    circuits = SHAPES[shape](False)
    bt, ic, val, (_, it1, rs1, x1) = _run(circuits, 5, monkeypatch)
    _, _, _, (_, it2, rs2, x2) = _run(circuits, 5, monkeypatch, GPUKLU_CONT_M="2")
    assert np.array_equal(it1, it2) and np.array_equal(rs1, rs2)
    assert x1.tobytes() == x2.tobytes()
    _, _, _, (_, _, _, xa) = _run(circuits, 5, monkeypatch, max_iters=6)
    _, _, _, (_, _, _, xb) = _run(circuits, 5, monkeypatch, max_iters=6, GPUKLU_CONT_KERNEL="0")
    assert xa.tobytes() == xb.tobytes()
    it_o, rs_o, x_o = po.dc_batch(circuits, ic, np.zeros(len(ic), np.int64), val,
                                  "nativeklu_exact", nthreads=2,
                                  x_cap=max(c.n for c in circuits),
                                  **{k: wl.TIGHT[k] for k in ("max_iters", "abs_tol", "rel_tol",
                                                              "gmin", "gmin_steps")})
    assert np.array_equal(rs1 == 0, rs_o == 0) and np.mean(rs_o == 0) > 0.5
    for i in np.flatnonzero(rs_o == 0):
        n = circuits[ic[i]].n
        xg, xo = x1[bt.x_off[i]:bt.x_off[i] + n], x_o[i, :n]
        assert np.max(np.abs(xg - xo)) <= 1e-10 * max(1.0, np.max(np.abs(xo))), i


@pytest.mark.parametrize("shape", SHAPES)
def test_transient_and_adjoint(shape):
    circuits = SHAPES[shape](True)
    steps, dt, probe = 30, 1e-12, 2
    xs = [np.zeros(c.node_count) for c in circuits]
    off = np.concatenate([[0], np.cumsum([len(x) for x in xs])[:-1]]).astype(np.int64)
    tb = TranBatch(circuits, np.concatenate(xs), off, dt, steps, 7, probe, 0.2)
    cfg = dict(wl.TIGHT, abs_tol=1e-15, rel_tol=1e-14)
    loss, wave, _, rs = tb.forward(N.newton_config(**cfg), with_wave=True)
    assert np.all(rs == 0)
    grads, _ = tb.backward(N.newton_config(**cfg))
    for i, c in enumerate(circuits):
        r, _, st = po.tran(c, xs[i], dt, steps,
                           **{k: cfg[k] for k in ("max_iters", "abs_tol", "rel_tol", "gmin")})
        assert r == 0
        assert np.max(np.abs(wave[i] - st[1:, probe])) <= 1e-9
        g = po.tran_adjoint(c, st, dt, probe, 0.2)
        caps = c.type == cz.DEV_C
        assert np.max(np.abs(grads[i][caps] - g[caps])) <= 1e-7 * np.max(np.abs(g[caps])), i
