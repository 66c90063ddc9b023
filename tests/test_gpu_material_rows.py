"""reset refuses a particle whose material is past the table's 96 rows, on one thread and on several,
names the first one and changes nothing; the last row is taken."""
import numpy as np
import pytest

import sprout_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 100000])
@pytest.mark.parametrize("kind", [97, 255, 0x20000 | 200])
def test_material_past_the_table_is_refused(n, kind):
    p = np.zeros(n, S.PARTICLE_DTYPE)
    p["pos"] = np.random.default_rng(n).uniform(4, 60, (n, 2)).astype(np.float32)
    p["kind"] = 96
    p["t"], p["s"] = -1.0e4, -1.0
    sim = S.FluidSim(96, 64, n, S.SimParams({"cell_size": 0.002}))
    sim.reset(p)
    before = sim.download_particles()
    q = p.copy()
    q["kind"][[n // 2, n - 1]] = kind
    with pytest.raises(S.SproutError, match=f"particle {n // 2} has no material row") as e:
        sim.reset(q)
    assert e.value.code == -1
    assert sim.download_particles().tobytes() == before.tobytes()
