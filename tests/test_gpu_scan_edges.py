"""The counting sort's scan at the edges of its blocks (4096 counts, four a thread): one count past,
short of and on a block, every remainder of a thread's four, and more blocks than a block has
threads."""
import numpy as np
import pytest

import sprout_gb300 as S
import tanks
from test_gpu_parity import compare_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(63, 65), (64, 64), (90, 45), (66, 31), (130, 63), (128, 64), (91, 90), (101, 81)])
def test_blocks_and_remainders(w, h):
    t = tanks.dam_break(w, h, width=0.7, height=0.9)
    sim, _, _ = t.engine()
    ora, _, _ = tanks.oracle_of(t)
    for k in range(2):
        sim.step(1, 1.0 / 240.0)
        ora.step(1, 1.0 / 240.0)
        problems = compare_state(sim, ora, f"{w}x{h} substep {k}")
        assert not problems, "\n".join(problems)


def test_more_blocks_than_threads():
    w, h = 2304, 1857   # 1045 blocks of counts
    t = tanks.Tank(w, h, {"cell_size": 0.002, "fixed_hz": 240.0},
                   [], [([4.0, 4.0, 20.0, 12.0], 0, None), ([w - 60.0, h - 30.0, w - 20.0, h - 10.0], 0, None)])
    sim, parts, _ = t.engine()
    sim.step(1, 1.0 / 240.0)
    p = sim.download_particles()
    live = p[p["kind"] != 0]
    assert len(live) == len(parts)
    count = sim.field("count", np.uint32)
    assert int(count.sum()) == len(parts)
    # the sort is by the cells of the counts: their expansion gives each slot's cell
    cell = np.repeat(np.arange(w * h), count)
    at = np.clip(live["pos"].astype(np.int64), 0, [w - 1, h - 1])
    assert np.array_equal(cell, at[:, 1] * w + at[:, 0])
