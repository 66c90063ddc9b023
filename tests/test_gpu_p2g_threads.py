"""P2G's two block sizes on either side of the line between them (1024 particles to each of two
blocks an SM), and the particle counts around a block's: its sums bit for bit as the oracle's."""
import numpy as np
import pytest

import tanks
from test_gpu_parity import first_diff

pytestmark = pytest.mark.gpu


def few_at_most():
    torch = pytest.importorskip("torch")
    return 2 * 1024 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("n", [1, 255, 513, "line", "past the line"])
def test_sums_match_the_oracle(n):
    if isinstance(n, str):
        n = few_at_most() + (n == "past the line")

    def scatter(parts):
        rng = np.random.default_rng(n)
        p = np.repeat(parts[:1], n)
        p["id"] = np.arange(n)
        p["pos"] = rng.uniform([4, 4], [180, 100], (n, 2)).astype(np.float32)
        p["vel"] = rng.normal(0, 20, (n, 2)).astype(np.float32)
        return p
    t = tanks.dam_break(184, 104)
    t.prepare = scatter
    sim, _, _ = t.engine()
    ora, _, _ = tanks.oracle_of(t)
    sim.step(1, 1.0 / 240.0)
    ora.step(1, 1.0 / 240.0)
    a, b = sim.field("acc", np.int32), ora.field("acc", np.int32)
    assert np.count_nonzero(b) > 0
    bad, k = first_diff(a, b)
    assert bad == 0, f"{bad} sums differ, the first {k}"
