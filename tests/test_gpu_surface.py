"""The surface pass (face coefficients, smoothed indicators, node normals and curvatures) at the
edges of its tiles, bit for bit against the oracle: grids one past, short of and on a 16-cell
tile's edge, with solids whose walls the liquid wets, two to four phase groups and tension."""
import pytest

import tanks
from test_gpu_parity import first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 16), (17, 31), (33, 18), (48, 47), (70, 33), (97, 65)])
@pytest.mark.parametrize("groups", [{}, {59: 1}, {59: 2}, {59: 3, 60: 1}, {59: 1, 60: 2, 61: 3}])
def test_ragged_tiles(w, h, groups):
    s = {"cell_size": 0.002, "fixed_hz": 240.0, "tension_water": 0.07, "gravity": 9.8}
    for row in (59, 60, 61):
        for name, v in {"density": 800.0 + 100 * (row - 58), "viscosity": 1e-6, "tension": 0.02 * (row - 57)}.items():
            s[f"mat{row}.{name}"] = v
    t = tanks.Tank(w, h, s, [{"kind": "circle", "c": [0.5 * w, 0.35 * h], "r": 0.15 * min(w, h)}],
                   [([0.0, 0.0, 0.5 * w, 0.6 * h], 0, None), ([0.5 * w, 0.0, 0.7 * w, 0.5 * h], 59, None),
                    ([0.7 * w, 0.0, 0.85 * w, 0.4 * h], 60, None), ([0.85 * w, 0.0, w, 0.3 * h], 61, None)], groups=groups)
    sim, _, _ = t.engine()
    ora, _, _ = tanks.oracle_of(t)
    for k in range(3):
        sim.step(1, 1.0 / 240.0)
        ora.step(1, 1.0 / 240.0)
        for name in ["coef", "surf", "pjump", "vel"] + (["surf2"] if any(g > 1 for g in groups.values()) else []):
            n, first = first_diff(sim.field(name), ora.field(name))
            assert n == 0, (name, k, n, first)
