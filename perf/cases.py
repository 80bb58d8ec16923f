"""The measured work of this framework: whole calls of its public entry points
(rustspice_gb300.solver), from an 18-unknown operating point to the
249,856-instance batch, on the seeded circuits of the repository's own
workloads, tests and benchmark.

A case is a dict of plain values; ``kind`` picks the entry point:

  newton   one DC operating point on the device (newton_dc)
  lu       factor + solve through the LinearSolver calls with host arrays
  adjoint  DC operating point, then lambda and dL/dp of it (dc_forward,
           dc_backward)
  sweep    a .dc sweep of one source (dc_sweep)
  batch    independent operating points in one batched run (Batch)
  tran     fixed-step transient and its adjoint (TranBatch)
  atran    the adaptive transient (ATranBatch)
  bbd      DC operating point of a bordered-block-diagonal circuit (BbdSolver)
  ac       a small-signal .ac sweep (ac_sweep)

``prepare`` makes what a program holds before the call - the circuit compiled
for the device, the solver handle or batch, the inputs - ``run`` makes the
call, ``exact`` is the same result from plain numpy / torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import netlist as nl
from rustspice_gb300 import solver as sv
from rustspice_gb300 import waveforms as wf
from rustspice_gb300 import workloads as wl

EXACT_MAX_N = 4200  # a dense 64-bit solve per Newton iteration takes too long beyond


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest call: the operating point of a deck of a few devices,
        # where launches and host round trips are the time.
        {"name": "newton_small", "kind": "newton", "side": 4, "diodes": 4, "gmin_steps": 0},
        # The plain operating point of the benchmark: a 1024-node resistor
        # mesh with 64 diodes, gmin stepping.
        {"name": "newton_mesh", "kind": "newton", "side": 32, "diodes": 64, "gmin_steps": 10},
        # The drop-in LinearSolver: one factor and solve of an engine that
        # keeps its own matrix on the host (a 2,304-node mesh, odd border).
        {"name": "lu_mesh", "kind": "lu", "side": 48, "diodes": 96, "solver": "nativeklu"},
        # The large single circuit with sensitivities: 120x120 mesh driving
        # 1000 inverters, forward and backward.
        {"name": "adjoint_large", "kind": "adjoint", "side": 120, "inverters": 1000},
        # A .dc sweep of the source of a diode mesh, each point continued
        # from the one before.
        {"name": "sweep_mesh", "kind": "sweep", "side": 16, "diodes": 24, "points": 25},
        # A small Monte-Carlo run: 16 chains of uneven length, 61 inputs each.
        {"name": "batch_small", "kind": "batch", "chains": 16, "vin": 61, "lo": 8, "hi": 256},
        # The headline Monte-Carlo run: 4096 chains x 61 inputs from pinned
        # host memory, every solution back into a pinned buffer.
        {"name": "batch_large", "kind": "batch", "chains": 4096, "vin": 61, "lo": 8, "hi": 256},
        # Ring oscillators of uneven odd length: backward-Euler transient and
        # the checkpointed adjoint for every capacitance.
        {"name": "tran_rings", "kind": "tran", "rings": 1024, "steps": 250, "ckpt": 50},
        # The adaptive transient of pulse-driven chains.
        {"name": "atran_chains", "kind": "atran", "chains": 512, "lo": 8, "hi": 64,
         "tstop": 2e-9},
        # Coupled blocks through the Schur complement: 64 uneven meshes and
        # 1024 border nodes.
        {"name": "bbd_meshes", "kind": "bbd", "blocks": 64, "border": 1024, "lo": 30, "hi": 50,
         "diodes": 32},
        # The .ac sweep of the benchmark: a 100-section RC ladder, 500 points
        # per decade from 1 Hz to 1 GHz.
        {"name": "ac_ladder", "kind": "ac", "shape": "ladder", "size": 100, "per_decade": 500,
         "diodes": 0},
        # A larger .ac sweep: a power-grid-like RC mesh with biased diodes.
        {"name": "ac_grid", "kind": "ac", "shape": "grid", "size": 18, "per_decade": 25,
         "diodes": 30},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["newton", "newton", "lu", "lu", "adjoint", "sweep", "batch", "batch", "tran",
                       "atran", "bbd", "ac", "ac"])
    if kind == "newton":
        side = _log(rng, 4, 56)
        return {"kind": kind, "side": side, "diodes": rng.randint(1, max(1, side * side // 8)),
                "gmin_steps": rng.choice([0, 4, 10])}
    if kind == "lu":
        # the factory's choice for up to 50 unknowns is the dense kind
        solver = rng.choice(["nativeklu", "nativeklu", "nativeklu", "dense"])
        side = rng.randint(3, 7) if solver == "dense" else _log(rng, 4, 64)
        return {"kind": kind, "side": side, "diodes": rng.randint(1, max(1, side * side // 8)),
                "solver": solver}
    if kind == "adjoint":
        side = _log(rng, 12, 110)
        return {"kind": kind, "side": side, "inverters": rng.randint(1, max(2, side * side // 15))}
    if kind == "sweep":
        side = _log(rng, 4, 28)
        return {"kind": kind, "side": side, "diodes": rng.randint(1, max(1, side * side // 8)),
                "points": rng.randint(5, 31)}
    if kind == "batch":
        lo = rng.randint(2, 64)
        return {"kind": kind, "chains": _log(rng, 1, 2048), "vin": rng.randint(3, 61), "lo": lo,
                "hi": rng.randint(lo, 256)}
    if kind == "tran":
        return {"kind": kind, "rings": _log(rng, 4, 1024), "steps": rng.randint(40, 240),
                "ckpt": rng.choice([17, 25, 50])}
    if kind == "atran":
        lo = rng.randint(4, 16)
        return {"kind": kind, "chains": _log(rng, 4, 512), "lo": lo, "hi": rng.randint(lo + 4, 64),
                "tstop": rng.uniform(0.6e-9, 2e-9)}
    if kind == "bbd":
        lo = rng.randint(8, 30)
        return {"kind": kind, "blocks": rng.randint(4, 56), "border": _log(rng, 24, 800), "lo": lo,
                "hi": min(46, lo + rng.randint(0, 16)), "diodes": rng.randint(4, 32)}
    if rng.random() < 0.5:
        return {"kind": kind, "shape": "ladder", "size": _log(rng, 5, 260),
                "per_decade": _log(rng, 6, 60), "diodes": rng.choice([0, 0, 2])}
    return {"kind": kind, "shape": "grid", "size": rng.randint(3, 17),
            "per_decade": _log(rng, 4, 24), "diodes": rng.randint(0, 8)}


# ---------------------------------------------------------------- inputs
GMIN = 1e-12
ATRAN_POINTS = 512  # recorded points per circuit of an adaptive run


def _cfg(**kw):
    return N.newton_config(**dict(wl.TIGHT, **kw))


def _ac_deck(case, seed):
    """The deck of an ac case: R and C seeded as the benchmark's ladder has
    them; diodes to ground biased by the source's DC value."""
    rng = np.random.default_rng(3 + seed)
    size = case["size"]
    dc = 0.5 if case["diodes"] else 0.0
    lines = [f"V1 n0 0 DC {dc} AC 1 30"]
    if case["shape"] == "ladder":
        nodes = size + 1
        for k in range(size):
            lines.append(f"R{k} n{k} n{k + 1} {rng.uniform(100, 1000):.6g}")
            lines.append(f"C{k} n{k + 1} 0 {rng.uniform(1e-12, 1e-9):.6g}")
    else:
        nodes = size * size
        k = 0
        for r in range(size):
            for c in range(size):
                a = r * size + c
                for b in ([a + 1] if c + 1 < size else []) + ([a + size] if r + 1 < size else []):
                    lines.append(f"R{k} n{a} n{b} {100.0 * 10.0 ** (2.0 * rng.random()):.6g}")
                    k += 1
                lines.append(f"C{a} n{a} 0 {rng.uniform(1e-13, 1e-11):.6g}")
    if case["diodes"]:
        lines.append(".model dd D (IS=1e-14 N=1)")
        at = rng.choice(nodes - 1, min(case["diodes"], nodes - 1), replace=False) + 1
        lines += [f"D{k} n{int(a)} 0 dd" for k, a in enumerate(at)]
    return nl.compile_deck("\n".join(lines) + "\n").circuit


def _batch_inputs(case, seed):
    """inverter_batch's circuits and instances with the logic-level nodesets
    written as arrays. The chains' lengths are the workload's, their devices
    the seed's."""
    chains, nvin = case["chains"], case["vin"]
    sd = 3 + seed
    stages = cz.chain_lengths(chains, case["lo"], case["hi"])
    vins = cz.vin_points(nvin)
    circuits = [cz.inverter_chain(int(s), 0.0, seed=sd, chain_id=i) for i, s in enumerate(stages)]
    n = np.repeat(stages + 3, nvin)
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    vin = np.tile(vins, chains)
    pos = np.arange(off[-1], dtype=np.int64) - np.repeat(off[:-1], n)
    high = np.repeat(vin < 0.585, n)
    x0 = np.where((((pos - 3) & 1) == 0) == high, wl.VDD, 0.0)
    x0[off[:-1]] = 0.0
    x0[off[:-1] + 1] = wl.VDD
    x0[off[:-1] + 2] = vin
    return circuits, np.repeat(np.arange(chains, dtype=np.int64), nvin), vin, x0, off[:-1].copy()


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _lu_system(c, seed):
    """A mesh's matrix and right-hand side as the engine stamps them at a
    Newton iterate near the diodes' knee."""
    x = np.random.default_rng(17 + seed).uniform(0.0, 0.6, c.node_count)
    x[0] = 0.0
    return x


def _rings(case, seed):
    stages = wl.ring_stages(case["rings"])
    cs = [cz.ring_oscillator(int(s), seed=5 + seed, ring_id=i) for i, s in enumerate(stages)]
    xs = [wl.ring_initial_state(c) for c in cs]
    off = np.zeros(len(xs), np.int64)
    off[1:] = np.cumsum([len(x) for x in xs])[:-1]
    return cs, np.concatenate(xs), off


def _circuit(case, seed):
    k = case["kind"]
    if k in ("newton", "lu", "sweep"):
        return cz.mesh_dc(case["side"], case["diodes"], seed=1 + seed)
    if k == "adjoint":
        return cz.mesh_with_inverters(case["side"], case["inverters"], seed=4 + seed)
    if k == "ac":
        return _ac_deck(case, seed)
    raise ValueError(k)


def _outputs(c, seed):
    return cz.output_nodes(c, min(256, (c.node_count - 1) // 2), seed=4 + seed)


def _freqs(case):
    return sv.frequency_sweep("dec", case["per_decade"], 1.0, 1e9)


def _sweep_values(case):
    return np.linspace(0.0, 1.0, case["points"])


def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k}
    if k in ("newton", "adjoint", "sweep"):
        c = _circuit(case, seed)
        st["dc"] = sv.DeviceCircuit(c)
        st["g"] = sv.GpuKluSolver(1, pivot_mode=N.PIVOT_EXACT)
        st["cfg"] = _cfg(gmin_steps=case.get("gmin_steps", 0))
        if k == "adjoint":
            st["outs"] = _outputs(c, seed)
        if k == "sweep":
            st["src"] = c.device_index(cz.DEV_V)
            st["values"] = _sweep_values(case)
    elif k == "lu":
        c = _circuit(case, seed)
        dc = sv.DeviceCircuit(c)
        kind = case["solver"]
        st["g"] = sv.GpuKluSolver(dc.n, kind=kind,
                                  pivot_mode=N.PIVOT_EXACT if kind == "nativeklu" else
                                  N.PIVOT_REFERENCE)
        st["ap"], st["ai"] = dc.pattern()
        st["ax"], st["rhs"] = dc.stamp(st["g"], _lu_system(c, seed), gmin=GMIN)
    elif k == "batch":
        circuits, ic, vin, x0, off = _batch_inputs(case, seed)
        st["bt"] = sv.Batch(circuits, ic, np.ones(len(ic), np.int64), vin, x0, off)
        st["vin"], st["x0"] = _pinned(vin), _pinned(x0)
        st["x"] = torch.empty(st["bt"].x_len, dtype=torch.float64).pin_memory().numpy()
        st["cfg"] = _cfg()
    elif k == "tran":
        cs, x, off = _rings(case, seed)
        st["tb"] = sv.TranBatch(cs, x, off, wl.RING_DT, case["steps"], case["ckpt"], wl.RING_PROBE,
                                wl.RING_TARGET)
        st["cfg"] = _cfg()
    elif k == "atran":
        stages = cz.chain_lengths(case["chains"], case["lo"], case["hi"], 13)
        cs = [cz.inverter_chain(int(s), 0.0, seed=13 + seed, chain_id=i)
              for i, s in enumerate(stages)]
        waves = [{1: wf.pulse(**wl.ATRAN_PULSE)} for _ in cs]
        st["ab"] = sv.ATranBatch(cs, waves, [wl.chain_nodeset(int(s), 0.0) for s in stages],
                                 np.array([c.node_count - 1 for c in cs]))
        st["tstop"] = case["tstop"]
        st["cfg"] = N.newton_config(max_iters=100, abs_tol=1e-9, rel_tol=1e-6, gmin=GMIN)
    elif k == "bbd":
        c, asg, nb = _bbd_circuit(case, seed)
        st["dc"] = sv.DeviceCircuit(c)
        ap, ai = st["dc"].pattern()
        st["bb"] = sv.BbdSolver(ap, ai, asg, nb)
        st["x0"] = wl.bordered_nodeset(c)
        st["cfg"] = _cfg()
    elif k == "ac":
        c = _circuit(case, seed)
        st["dc"] = sv.DeviceCircuit(c)
        st["g"] = sv.GpuKluSolver(1, pivot_mode=N.PIVOT_EXACT)
        st["x"] = np.zeros(c.n)
        if case["diodes"]:
            st["x"][:] = sv.newton_dc(st["g"], st["dc"], _cfg()).x
        st["f"] = _freqs(case)
    return st


def _bbd_circuit(case, seed):
    """The workload's structure; the meshes' resistors in the seed's order."""
    c, asg, nb = cz.bordered_meshes(case["blocks"], case["border"], case["lo"], case["hi"],
                                    case["diodes"])
    mesh = np.flatnonzero((c.type == cz.DEV_R) & (asg[c.nodes[:, 0]] >= 0))
    c.p[mesh, 0] = c.p[np.random.default_rng(2 + seed).permutation(mesh), 0]
    return c, asg, nb


def _rows(parts):
    """Waveforms of uneven length as the rows of one array."""
    out = np.zeros((len(parts), ATRAN_POINTS))
    for row, p in zip(out, parts):
        row[:len(p)] = p
    return out


def _point(r):
    return {"x": r.x, "iterations": r.iterations, "total": r.iterations_total,
            "converged": r.converged}


# ---------------------------------------------------------------- the call
def run(st):
    k = st["kind"]
    if k == "newton":
        return _point(sv.newton_dc(st["g"], st["dc"], st["cfg"]))
    if k == "lu":
        g, x = st["g"], st["rhs"].copy()
        g.factor(st["ap"], st["ai"], st["ax"])
        g.solve(x)
        return {"x": x}
    if k == "adjoint":
        f = sv.dc_forward(st["g"], st["dc"], st["cfg"])
        dl = np.zeros(st["dc"].n)
        dl[st["outs"]] = 2.0 * (f.x[st["outs"]] - 0.6)
        lam, grad = sv.dc_backward(st["g"], st["dc"], f.x, dl)
        return dict(_point(f), lam=lam, grad=grad)
    if k == "sweep":
        r = sv.dc_sweep(st["g"], st["dc"], st["cfg"], st["src"], st["values"],
                        stop_on_failure=False)
        return {"x": r.x, "iterations": r.iterations, "total": r.iterations_total,
                "reason": r.reason}
    if k == "batch":
        b = st["bt"]
        b.update_inputs(st["vin"], st["x0"])
        b.run(st["cfg"])
        it, itt, rs, x = b.results(x_out=st["x"])
        return {"iterations": it, "total": itt, "reason": rs, "x": x}
    if k == "tran":
        loss, wave, it, rs = st["tb"].forward(st["cfg"], with_wave=True)
        grad, bit = st["tb"].backward(st["cfg"])
        return {"loss": loss, "wave": wave, "iterations": it, "reason": rs,
                "grad": np.concatenate(grad), "iterations_back": bit}
    if k == "atran":
        r = st["ab"].run(st["cfg"], wl.ATRAN_TSTEP, st["tstop"], lte_abs=1e-6, lte_rel=1e-3,
                         be_sign=1.0, max_points=ATRAN_POINTS)
        return {"status": r.status, "npoints": r.npoints, "accepted": r.accepted,
                "rejected": r.rejected, "iterations": r.iterations,
                "times": _rows(r.times), "probe": _rows(r.probe), "x": np.concatenate(r.x)}
    if k == "bbd":
        return _point(st["bb"].newton_dc(st["dc"], st["cfg"], x0=st["x0"]))
    if k == "ac":
        return {"y": sv.ac_sweep(st["g"], st["dc"], st["x"], st["f"])}
    raise ValueError(k)


# ---------------------------------------------------------------- its work
# Newton iterations of a typical operating point of each kind.
_ITERS = {"newton": 12, "adjoint": 5, "sweep": 5, "bbd": 9}


def _mesh_lu(side):
    """(multiply-adds, factor entries) of an LU of a side x side grid in a
    nested-dissection order: George's bounds for the Cholesky factor, twice."""
    s = max(side, 2)
    return 2.0 * 9.87 * s ** 3, 2.0 * 7.75 * s * s * math.log2(s)


def work(case):
    """Bytes: the device table and the starting values read once, the results
    written once. Flops: the device evaluations, factorizations and
    substitutions of the iterations it takes, two per multiply-add."""
    k = case["kind"]
    if k in ("newton", "lu", "adjoint", "sweep"):
        side = case["side"]
        n = side * side
        ndev = 2 * n + case.get("diodes", 0) + 3 * case.get("inverters", 0)
        mads, nnz = _mesh_lu(side)
        its = 1 if k == "lu" else _ITERS[k] * case.get("points", 1)
        flops = its * (2 * mads + 2 * nnz + 8 * ndev)
        if k == "lu":
            return {"bytes": 16.0 * 9 * n + 16.0 * n, "flops": flops}
        if k == "adjoint":
            return {"bytes": 68.0 * ndev + 8.0 * (3 * n + ndev),
                    "flops": flops * (its + 1) / its + 10 * ndev}
        return {"bytes": 68.0 * ndev + 8.0 * n * case.get("points", 1), "flops": flops}
    if k == "batch":
        stage = 0.5 * (case["lo"] + case["hi"])
        inst = case["chains"] * case["vin"]
        # device constants once per chain; start in, solution out; about three
        # iterations of two MOSFETs (25 operations each) and a bidiagonal row
        return {"bytes": case["chains"] * stage * 2 * 32.0 + inst * (2 * 8.0 * (stage + 4) + 32),
                "flops": inst * 3.0 * stage * 70}
    if k == "tran":
        stage = 56.0
        solves = 4.5 * case["rings"] * case["steps"]  # two Newton solves forward and again backward
        return {"bytes": case["rings"] * (stage * 3 * 32.0 + case["steps"] * 8.0 + 3 * stage * 8),
                "flops": solves * stage * 90}
    if k == "atran":
        stage = 0.5 * (case["lo"] + case["hi"])
        solves = case["chains"] * 1300.0 * case["tstop"] / 2e-9
        return {"bytes": case["chains"] * (stage * 3 * 32.0 + 220 * 16.0 + stage * 8),
                "flops": solves * stage * 90}
    if k == "bbd":
        side = 0.5 * (case["lo"] + case["hi"])
        mads, nnz = _mesh_lu(side)
        bs = case["border"]
        cols = 6.0 * bs  # border columns of all blocks together
        flops = _ITERS[k] * (case["blocks"] * 2 * mads + cols * 2 * nnz + 2.0 * bs ** 3 / 3)
        n = case["blocks"] * side * side + bs
        return {"bytes": 68.0 * (2 * n + 6 * bs) + 16.0 * n, "flops": flops}
    nf = 9 * case["per_decade"] + 1
    if case["shape"] == "ladder":
        n, mads = case["size"] + 3, 4.0 * case["size"]
    else:
        n, mads = case["size"] ** 2 + 2, _mesh_lu(case["size"])[0]
    return {"bytes": nf * (8.0 + 16.0 * n), "flops": nf * 8.0 * mads}


# ---------------------------------------------------------------- in 64 bits
def _dense_stamp(c, x, p, gmin, gdev=1e-12):
    """The MNA system of a device list at the iterate x: (A, b), dense, from
    the element equations (R, V, I, diode, level-1 Shichman-Hodges MOSFET)."""
    n = c.n
    A, b = np.zeros((n, n)), np.zeros(n)
    t, nd = c.type, c.nodes.astype(np.int64)

    def two(a, e, g):
        np.add.at(A, (a, a), g)
        np.add.at(A, (e, e), g)
        np.add.at(A, (a, e), -g)
        np.add.at(A, (e, a), -g)

    m = t == cz.DEV_R
    two(nd[m, 0], nd[m, 1], 1.0 / p[m, 0])
    for k, d in enumerate(np.flatnonzero(t == cz.DEV_V)):
        r = c.node_count + k
        for node, s in ((nd[d, 0], 1.0), (nd[d, 1], -1.0)):
            A[node, r] += s
            A[r, node] += s
        b[r] += p[d, 0]
    m = t == cz.DEV_I
    np.add.at(b, nd[m, 0], -p[m, 0])
    np.add.at(b, nd[m, 1], p[m, 0])
    m = t == cz.DEV_D
    vt = 0.02585 * p[m, 1]
    vd = x[nd[m, 0]] - x[nd[m, 1]]
    e = np.exp(vd / vt)
    gd = p[m, 0] / vt * e
    ieq = p[m, 0] * (e - 1.0) - gd * vd
    two(nd[m, 0], nd[m, 1], np.maximum(gd, gmin))
    np.add.at(b, nd[m, 0], -ieq)
    np.add.at(b, nd[m, 1], ieq)
    m = t == cz.DEV_MC
    if m.any():
        dr, gt, so = nd[m, 0], nd[m, 1], nd[m, 2]
        i, dg, dd, ds = _mos(p[m], x[dr], x[gt], x[so], gdev, np)
        ieq = i - (dg * x[gt] + dd * x[dr] + ds * x[so])
        for row, s in ((dr, 1.0), (so, -1.0)):
            np.add.at(A, (row, dr), s * dd)
            np.add.at(A, (row, gt), s * dg)
            np.add.at(A, (row, so), s * ds)
            np.add.at(b, row, -s * ieq)
    A[0, 0] += 1.0
    return A, b


def _mos(p, vd, vg, vs, gdev, xp):
    """Drain current and its partials with respect to (vg, vd, vs)."""
    pol = xp.where(p[..., 0] != 0.0, -1.0, 1.0)
    beta = p[..., 2] * 1e-4 * ((3.9 * 8.854e-12) / p[..., 3]) * p[..., 4] / p[..., 5]
    vgs, vds = pol * (vg - vs), pol * (vd - vs)
    rev = vds < 0.0
    vgs, vds = xp.where(rev, vgs - vds, vgs), xp.abs(vds)
    ov = vgs - xp.abs(p[..., 1])
    k = 1.0 + 0.02 * vds
    ve = xp.where(ov <= 0.0, 0.0 * ov, xp.minimum(vds, ov))
    q = ve * (ov - 0.5 * ve)
    i, gm = beta * q * k, beta * k * ve
    on = ov > 0.0
    gds = xp.where(on, beta * k * (ov - ve) + 0.02 * beta * q, 0.0 * ov)
    gds = xp.where(gds < gdev, 0.0 * gds + gdev, gds)
    i = xp.where(rev, -pol, pol) * i
    return (i, xp.where(rev, -gm, gm), xp.where(rev, gm + gds, gds),
            xp.where(rev, -gds, -(gm + gds)))


def _solve(A, b):
    if torch.cuda.is_available() and len(b) > 300:
        return torch.linalg.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
    return np.linalg.solve(A, b)


def _operating_point(c, p, gmin, x0):
    """Newton to rounding from x0, the damping halved when the update grows;
    None when it does not settle."""
    n, nc = c.n, c.node_count
    x = np.zeros(n)
    x[:nc] = x0
    damp, prev = 1.0, math.inf
    for _ in range(100):
        A, b = _dense_stamp(c, x, p, gmin)
        xn = _solve(A, b)
        dx = xn[:nc] - x[:nc]
        if np.all(np.abs(dx) <= 1e-13 + 1e-12 * np.abs(xn[:nc])):
            return xn
        norm = float(np.linalg.norm(dx))
        if norm > prev and damp > 0.1:
            damp = max(0.5 * damp, 0.1)
        prev = norm
        x[:nc] += damp * dx
    return None


def _first_gmin(steps):
    return max(GMIN * 1e3, 1e-6) if steps else GMIN


def exact(case, seed):
    k = case["kind"]
    if k in ("batch", "atran"):
        # some of a batch's instances end at the iteration cap, and an adaptive
        # run's points are where its own step control puts them: neither has a
        # value of its own in 64 bits
        return None
    if k == "tran":
        return _exact_tran(case, seed)
    if k == "bbd":
        c, _, _ = _bbd_circuit(case, seed)
        if c.n > EXACT_MAX_N:
            return None
        x = _operating_point(c, c.p, GMIN, wl.bordered_nodeset(c))
        return None if x is None else {"x": x, "iterations": None, "total": None,
                                       "converged": None}
    c = _circuit(case, seed)
    if c.n > EXACT_MAX_N:
        return None
    if k == "lu":
        A, b = _dense_stamp(c, np.pad(_lu_system(c, seed), (0, c.n - c.node_count)), c.p, GMIN)
        return {"x": _solve(A, b)}
    if k == "ac":
        return {"y": _exact_ac(c, case)}
    zero = np.zeros(c.node_count)
    none = {"iterations": None, "total": None}
    if k == "sweep":
        p, xs, x = c.p.copy(), [], zero
        for v in _sweep_values(case):
            p[c.device_index(cz.DEV_V), 0] = v
            xn = _operating_point(c, p, GMIN, x)
            if xn is None:
                return None
            xs.append(xn)
            x = xn[:c.node_count]
        return dict(none, x=np.stack(xs), reason=None)
    x = _operating_point(c, c.p, _first_gmin(case.get("gmin_steps", 0)), zero)
    if x is None:
        return None
    none["converged"] = None
    if k == "newton":
        return dict(none, x=x)
    A, _ = _dense_stamp(c, x, c.p, GMIN, gdev=0.0)
    g = np.zeros(c.n)
    o = _outputs(c, seed)
    g[o] = 2.0 * (x[o] - 0.6)
    lam = _solve(np.ascontiguousarray(A.T), g)
    return dict(none, x=x, lam=lam, grad=_param_grad(c, x, lam))


def _param_grad(c, x, lam):
    """dL/dp = -lam . dF/dp per device: R, the V source's value, VTO."""
    t, nd, p = c.type, c.nodes.astype(np.int64), c.p
    g = np.zeros(c.ndev)
    m = t == cz.DEV_R
    g[m] = (lam[nd[m, 0]] - lam[nd[m, 1]]) * (x[nd[m, 0]] - x[nd[m, 1]]) / p[m, 0] ** 2
    m = t == cz.DEV_V
    g[m] = lam[c.node_count:]
    m = t == cz.DEV_MC
    if m.any():
        # the current depends on the gate through vgs - |VTO| alone
        pol = np.where(p[m, 0] != 0.0, -1.0, 1.0)
        _, dg, _, _ = _mos(p[m], x[nd[m, 0]], x[nd[m, 1]], x[nd[m, 2]], 0.0, np)
        g[m] = (lam[nd[m, 0]] - lam[nd[m, 2]]) * dg * pol * np.sign(p[m, 1])
    return g


def _exact_ac(c, case):
    x = np.zeros(c.n)
    if case["diodes"]:
        x = _operating_point(c, c.p, GMIN, np.zeros(c.node_count))
        if x is None:
            return None
    n, nc = c.n, c.node_count
    G, _ = _dense_stamp(c, x, c.p, GMIN)
    G[0, :] = 0.0
    G[0, 0] = 1.0
    C, b = np.zeros((n, n)), np.zeros(n, complex)
    for d in np.flatnonzero(c.type == cz.DEV_C):
        i, j = (int(v) for v in c.nodes[d, :2])
        for r, q, s in ((i, i, 1.0), (j, j, 1.0), (i, j, -1.0), (j, i, -1.0)):
            if r != 0:
                C[r, q] += s * c.p[d, 0]
    for k, d in enumerate(np.flatnonzero(c.type == cz.DEV_V)):
        b[nc + k] = c.p[d, 1] * np.exp(1j * np.pi * c.p[d, 2] / 180.0)
    f = _freqs(case)
    out = np.empty((len(f), n), complex)
    step = max(1, 40_000_000 // (n * n))
    for a in range(0, len(f), step):
        w = 2.0 * np.pi * f[a:a + step]
        Y = G[None] + 1j * w[:, None, None] * C[None]
        B = np.broadcast_to(b[None, :, None], (len(w), n, 1)).copy()
        if torch.cuda.is_available():
            out[a:a + step] = torch.linalg.solve(torch.from_numpy(Y).cuda(),
                                                 torch.from_numpy(B).cuda())[..., 0].cpu().numpy()
        else:
            out[a:a + step] = np.linalg.solve(Y, B)[..., 0]
    return out


def _exact_tran(case, seed):
    """Backward Euler on every ring at once (padded to the longest; a ring's
    stage k drives node k from node k-1): Newton per step to rounding, then
    the discrete adjoint of the loss."""
    if case["rings"] * case["steps"] > 300_000 or not torch.cuda.is_available():
        return None  # over about 20 seconds
    cs, _, _ = _rings(case, seed)
    R, S = len(cs), max(c.node_count - 2 for c in cs)
    dev = "cuda"
    sz = torch.tensor([c.node_count - 2 for c in cs], device=dev)
    pn, pp, cap = np.ones((R, S, 6)), np.ones((R, S, 6)), np.ones((R, S))
    pn[..., 0] = 0.0
    x = np.zeros((R, S))
    for i, c in enumerate(cs):
        s = c.node_count - 2
        mos = c.p[c.type == cz.DEV_MC]
        pn[i, :s], pp[i, :s] = mos[0::2], mos[1::2]
        cap[i, :s] = c.p[c.type == cz.DEV_C, 0]
        x[i, :s] = wl.ring_initial_state(c)[2:]
    f64 = torch.float64
    pn, pp, cap, x = (torch.from_numpy(a).to(dev, f64) for a in (pn, pp, cap, x))
    idx = torch.arange(S, device=dev)
    live = (idx[None] < sz[:, None]).to(f64)
    drv = torch.where(idx[None] > 0, idx[None] - 1, sz[:, None] - 1)  # the gate of each stage
    gc = cap / wl.RING_DT
    rows = torch.arange(R, device=dev)[:, None]

    def lin(x, floor):
        vg = x.gather(1, drv)
        zero = torch.zeros_like(x)
        i0, g0, d0, _ = _mos(pn, x, vg, zero, floor, _TorchXp)
        i1, g1, d1, _ = _mos(pp, x, vg, zero + 1.2, floor, _TorchXp)
        J = torch.zeros((R, S, S), dtype=f64, device=dev)
        J[rows, idx[None], idx[None]] = live * (d0 + d1 + gc) + (1.0 - live)
        J[rows, idx[None], drv] += live * (g0 + g1)
        return i0 + i1, J

    states = [x]
    for _ in range(case["steps"]):
        xp = x
        for _ in range(60):
            i, J = lin(x, 1e-12)
            dx = torch.linalg.solve(J, (live * (i + gc * (x - xp)))[..., None])[..., 0]
            x = x - dx
            if float(dx.abs().max()) < 1e-14:
                break
        states.append(x)
    wave = torch.stack([s[:, 0] for s in states[1:]], 1)
    lam, grad = torch.zeros_like(x), torch.zeros_like(x)
    for t in range(case["steps"], 0, -1):
        _, J = lin(states[t], 0.0)
        b = live * gc * lam
        b[:, 0] += 2.0 * (states[t][:, 0] - wl.RING_TARGET)
        lam = torch.linalg.solve(J.transpose(1, 2), b[..., None])[..., 0]
        grad -= lam * (states[t] - states[t - 1]) / wl.RING_DT
    out = []
    for i, c in enumerate(cs):
        g = np.zeros(c.ndev)
        g[c.type == cz.DEV_C] = grad[i, :c.node_count - 2].cpu().numpy()
        out.append(g)
    return {"loss": ((wave - wl.RING_TARGET) ** 2).sum(1).cpu().numpy(),
            "wave": wave.cpu().numpy(), "iterations": None, "reason": None,
            "grad": np.concatenate(out), "iterations_back": None}


class _TorchXp:
    """numpy's names of the elementwise functions _mos uses, on torch."""
    abs = torch.abs
    minimum = torch.minimum

    @staticmethod
    def where(m, a, b):
        def full(v):
            return v if isinstance(v, torch.Tensor) else torch.full(m.shape, float(v), dtype=torch.float64,
                                                                    device=m.device)
        return torch.where(m, full(a), full(b))
