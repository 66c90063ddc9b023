"""A tank whose pressure solves change precision while its liquid moves: the plain and the mixed
hierarchy are kept apart and only the one in use is cleared where liquid leaves, so the other must
not bring old unknowns back when it is used again. Bit for bit against a fresh tank in which the
same liquid is solved in that precision from the start.
"""
import numpy as np
import pytest

import sprout_gb300 as S
import tanks
from test_gpu_parity import first_diff

pytestmark = pytest.mark.gpu

DT = 1.0 / 240.0
W, H = 256, 144


def fill(rect):
    """A tank with water in `rect`."""
    t = tanks.dam_break(W, H)
    t.fills = [(rect, 0, None)]
    return t


HIGH = [20.0, 66.0, 230.0, 140.0]   # rows 32 to 64 of cells, and so their coarse tiles, stay empty
LOW = [10.0, 0.0, 240.0, 28.0]


def outcome(sim):
    st = sim.stats()
    p = sim.download_particles()
    return sim.field("pres"), p[np.argsort(p["id"])].view(np.uint8), list(st.pressure_iters), st.device_error


def one_step(sim, parts, how, precision):
    sim.reset(parts)
    sim.set_precision(precision)
    if how == "alone":
        sim.step(1, DT)
    else:   # as the only tank of a batch of that precision
        batch = S.Batch([sim], precision)
        batch.step(1)
        batch.sync()
        batch.remove(sim)


@pytest.mark.parametrize("how", ["alone", "batch"])
@pytest.mark.parametrize("first,then", [("plain", "mixed"), ("mixed", "plain"), ("plain", "plain"), ("mixed", "mixed")])
def test_unknowns_do_not_come_back_with_the_precision(first, then, how):
    sim, high, _ = fill(HIGH).engine()
    _, low, _ = fill(LOW).engine()
    fresh, _, _ = fill(HIGH).engine()
    one_step(sim, high, how, first)    # the first hierarchy: unknowns in the upper tiles
    one_step(sim, low, how, then)      # they leave while the other is in use
    one_step(sim, low, how, first)     # the first again
    one_step(fresh, low, how, first)
    pres, parts, iters, err = outcome(sim)
    want_pres, want_parts, want_iters, want_err = outcome(fresh)
    assert err == 0 and want_err == 0 and np.abs(want_pres).max() > 0.0
    assert iters == want_iters
    n, k = first_diff(pres, want_pres)
    assert n == 0, f"{n} pressures differ, the first {k}"
    assert np.array_equal(parts, want_parts)
