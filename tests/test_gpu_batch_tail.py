"""The instances of a batch that run to the iteration cap take no longer in a
batch than alone: a warp that has taken its turns at the queue runs on with all
its lanes together. Device times, the best of a few runs."""
import numpy as np
import pytest

from rustspice_gb300 import circuits as cz
from rustspice_gb300 import native as N
from rustspice_gb300 import workloads as wl
from rustspice_gb300.solver import Batch

pytestmark = pytest.mark.gpu


def _ms(b, cfg):
    best = 1e9
    for _ in range(5):
        b.run(cfg)
        best = min(best, b.phase_ms()["warps_ms"])
    return best


def test_capped_instances_of_a_small_batch():
    """16 chains of 8-256 stages x 61 inputs: a few instances run to the cap of
    100 iterations. The batch against the slowest of them alone: 9.9 and 9.9 ms;
    with a lane apart from the others 36 ms."""
    cfg = N.newton_config(**wl.TIGHT)
    B = wl.inverter_batch(16, 61, seed=3)
    b = Batch(B.circuits, B.inst_circ, B.inst_dev, B.inst_val, B.x0, B.x0_off)
    whole = _ms(b, cfg)
    its, _, reason, _ = b.results()
    b.close()
    capped = np.flatnonzero(reason != 0)
    assert 0 < len(capped) < 40
    alone = 0.0
    for i in capped:
        c = B.circuits[B.inst_circ[i]]
        x0 = B.x0[B.x0_off[i]:B.x0_off[i] + c.node_count]
        one = Batch([c], np.zeros(1, np.int64), B.inst_dev[i:i + 1], B.inst_val[i:i + 1], x0,
                    np.zeros(1, np.int64))
        alone = max(alone, _ms(one, cfg))
        assert one.results()[0][0] == its[i]
        one.close()
    assert whole <= 2.0 * alone, (whole, alone)
