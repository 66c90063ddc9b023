"""reset on several host threads against reset on one, where only one thread's part of the particles
holds a second liquid or is hot: what the parts found must be put together, whichever part it was.
The number of threads follows the CPUs that the calling thread may run on, which is how this test
asks for one."""
import os

import numpy as np
import pytest

import sprout_gb300 as S

pytestmark = pytest.mark.gpu

W, H, N = 160, 120, 131072
CPUS = os.sched_getaffinity(0) if hasattr(os, "sched_getaffinity") else {0}


def particles(part, what):
    """N particles of a liquid at rest, those from 45 to 55 % of the part's eighth of them special."""
    rng = np.random.default_rng(5)
    p = np.zeros(N, S.PARTICLE_DTYPE)
    p["pos"] = rng.uniform(4, [W - 4, H / 2], (N, 2)).astype(np.float32)
    p["kind"] = 60   # material row 59
    p["s"] = -1.0
    p["t"] = -1.0e4
    lo = N * part // 8
    some = slice(lo + N * 45 // 800, lo + N * 55 // 800)
    if what == "honey":
        p["kind"][some] = 2
    elif what == "heat":
        p["t"][some] = 80.0
    return p


def outcome(p):
    sim = S.FluidSim(W, H, N, S.SimParams({"cell_size": 0.002, "tension_honey": 0.0, "mat59.density": 1000.0,
                                                "mat59.viscosity": 1e-6, "mat59.tension": 0.0}))
    sim.reset(p)
    first = sim.download_particles()
    caps = sim.stats().caps
    sim.step(1, 1.0 / 240.0)
    st = sim.stats()
    assert st.device_error == 0
    return first, (caps, st.caps, st.viscosity_mode), sim.download_particles()


@pytest.mark.skipif(len(CPUS) < 2, reason="needs two CPUs: reset takes one thread on one")
@pytest.mark.parametrize("what", ["honey", "heat"])
@pytest.mark.parametrize("part", [0, 3, 7])
def test_parts_are_put_together(part, what):
    p = particles(part, what)
    got = outcome(p)
    os.sched_setaffinity(0, {min(CPUS)})
    try:
        want = outcome(p)
    finally:
        os.sched_setaffinity(0, CPUS)
    assert got[1] == want[1] and got[1] != outcome(particles(part, "nothing"))[1]
    assert got[0].tobytes() == want[0].tobytes()
    assert got[2].tobytes() == want[2].tobytes()
