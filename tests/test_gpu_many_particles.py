"""Large particle arrays (settled by several threads) against the same particles in arrays that
one thread settles, byte for byte, at counts around the thresholds' edges; and the error for a
non-finite position."""
import numpy as np
import pytest

import sprout_gb300 as S

pytestmark = pytest.mark.gpu

W, H = 160, 120


def some(n):
    rng = np.random.default_rng(n)
    p = np.zeros(n, S.PARTICLE_DTYPE)
    p["pos"] = rng.uniform(-3, 165, (n, 2)).astype(np.float32)
    p["vel"] = rng.normal(0, 0.1, (n, 2)).astype(np.float32)
    p["kind"] = rng.integers(1, 3, n)
    p["id"] = rng.integers(0, 1 << 30, n)
    p["t"] = np.where(rng.random(n) < 0.5, -1.0e4, 20.0)
    p["s"] = np.where(rng.random(n) < 0.5, -1.0, 0.5)
    return p


def engine(n):
    return S.FluidSim(W, H, n, S.SimParams({"cell_size": 0.002, "tension_water": 0.0, "tension_honey": 0.0}))


@pytest.mark.parametrize("n", [32767, 32768, 32769, 65537, 163840, 262145, 160001])
def test_reset_in_parts(n):
    p = some(n)
    big, small = engine(n), engine(16000)
    big.reset(p)
    got = big.download_particles()
    assert len(got) == n and np.array_equal(got["id"], np.arange(n, dtype=got["id"].dtype))
    for k in range(0, n, 16000):
        small.reset(p[k:k + 16000])
        want = small.download_particles()
        want["id"] += np.uint32(k)
        assert want.tobytes() == got[k:k + 16000].tobytes(), k


def test_the_first_non_finite_position_is_named_and_nothing_changes():
    n = 150000
    p = some(n)
    sim = engine(n)
    sim.reset(p)
    before = sim.download_particles()
    q = some(n)
    q["pos"][140001, 1] = np.inf
    q["pos"][70001, 0] = np.nan
    with pytest.raises(Exception, match="particle 70001 has a non-finite position"):
        sim.reset(q)
    assert sim.download_particles().tobytes() == before.tobytes()
