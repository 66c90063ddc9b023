"""The pressure solve's level passes and tail at the edges of their tiles, bit for bit against the
oracle, and their fast quotients' fallback to IEEE divisions.

Scaling a system A x = b by a power of two scales every residual, right-hand side and dot
product exactly and leaves every quotient as it is, so the solution and the iteration counts
must come out the same to the bit. The fast quotients hold for diagonals up to 2^40 and
couplings up to 2^25: scaled past those, every tile (or, near the limit, some) is taken again
with divisions.
"""
import numpy as np
import pytest

import sprout_gb300 as S
import tanks
from test_gpu_parity import compare_state

pytestmark = pytest.mark.gpu

DT = 1.0 / 240.0


# widths and heights one past, one short of and on a tile's edge, odd ones, a tail of one level,
# of a row, and one whose first level has nearly 1500 cells
@pytest.mark.parametrize("w,h", [(17, 16), (31, 33), (47, 65), (80, 49), (97, 113), (300, 17), (101, 57)])
def test_ragged_grids_match_the_oracle(w, h):
    t = tanks.dam_break(w, h, width=0.6, height=0.7)
    sim, _, _ = t.engine()
    ora, _, _ = tanks.oracle_of(t)
    for k in range(3):
        sim.step(1, DT)
        ora.step(1, DT)
        problems = compare_state(sim, ora, f"{w}x{h} substep {k}")
        assert not problems, "\n".join(problems)


def static_solve(w, h, scale):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(w * 1000 + h)
    liquid = np.zeros((h, w), bool)
    liquid[1:-1, 1:-1] = rng.random((h - 2, w - 2)) < 0.9
    liquid[h * 3 // 4:] = False
    face_x = np.where(rng.random((h, w + 1)) < 0.1, 0.0, rng.uniform(0.1, 1.0, (h, w + 1)))
    face_y = np.where(rng.random((h + 1, w)) < 0.1, 0.0, rng.uniform(0.1, 1.0, (h + 1, w)))
    a = np.stack([face_x[:, :-1], face_x[:, 1:], face_y[:-1], face_y[1:]], 2).astype(np.float32)
    a[~liquid] = 0.0
    d = np.where(liquid, (a.sum(2) + np.float32(1e-3)).astype(np.float32), np.float32(0.0))
    b = (rng.standard_normal((h, w, 2)) * liquid[:, :, None]).astype(np.float32)
    dev = torch.device("cuda:0")
    A, D, B = (torch.from_numpy(np.ascontiguousarray(v * np.float32(scale))).to(dev) for v in (a, d, b))
    x = torch.zeros((h * w, 2), dtype=torch.float32, device=dev)
    torch.cuda.synchronize()
    iters, _ = S.pressure_solve_static(w, h, A.data_ptr(), D.data_ptr(), B.data_ptr(), x.data_ptr(), 1e-4, 1e-4, 60)
    torch.cuda.synchronize()
    return iters, x.cpu().numpy()


@pytest.mark.parametrize("w,h", [(33, 47), (160, 96)])
@pytest.mark.parametrize("power", [24, 25, 38, 45])
def test_scaled_systems_give_the_same_solution(w, h, power):
    want_iters, want = static_solve(w, h, 1.0)
    iters, got = static_solve(w, h, 2.0 ** power)
    assert np.isfinite(want).all() and np.abs(want).max() > 0.0 and max(want_iters) > 1
    assert iters == want_iters
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), f"{np.count_nonzero(got != want)} values differ"
