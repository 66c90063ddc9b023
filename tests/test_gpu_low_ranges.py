"""The pressure solve's fast quotients below their range: couplings below 2^-25, diagonals below
2^-40 and residuals below 2^-60 are divided the IEEE way.

As in the level passes' tests, scaling a system by a power of two must leave its solution the same
to the bit. Here the scaled system lies within the fast range and the unscaled one below it in most
tiles (couplings, diagonals), or the other way round (right-hand sides scaled down, so that the
solution scales with them; at 2^-40 and 2^-44 the squares that the dot products add up stay normal
numbers or too far below the sums to count in them).
"""
import numpy as np
import pytest

import sprout_gb300 as S

pytestmark = pytest.mark.gpu


def system(w, h, low):
    """A random system; low: one face in 50 nearly closed, one cell in 50 cut off from its
    neighbours with a tiny diagonal and right-hand side."""
    rng = np.random.default_rng(w * 1000 + h)
    liquid = np.zeros((h, w), bool)
    liquid[1:-1, 1:-1] = rng.random((h - 2, w - 2)) < 0.9
    liquid[h * 3 // 4:] = False
    face_x = np.where(rng.random((h, w + 1)) < 0.1, 0.0, rng.uniform(0.1, 1.0, (h, w + 1)))
    face_y = np.where(rng.random((h + 1, w)) < 0.1, 0.0, rng.uniform(0.1, 1.0, (h + 1, w)))
    alone = np.zeros((h, w), bool)
    if low:
        face_x = np.where(rng.random(face_x.shape) < 0.02, face_x * 2.0 ** -30, face_x)
        face_y = np.where(rng.random(face_y.shape) < 0.02, face_y * 2.0 ** -30, face_y)
        alone = liquid & (rng.random((h, w)) < 0.02)
        for f, a, b in ((face_x, alone[:, :-1], alone[:, 1:]), (face_y.T, alone.T[:, :-1], alone.T[:, 1:])):
            f[:, 1:-1][a | b] = 0.0
    a = np.stack([face_x[:, :-1], face_x[:, 1:], face_y[:-1], face_y[1:]], 2).astype(np.float32)
    a[~liquid] = 0.0
    d = np.where(liquid, (a.sum(2) + np.float32(1e-3)).astype(np.float32), np.float32(0.0))
    b = (rng.standard_normal((h, w, 2)) * liquid[:, :, None]).astype(np.float32)
    if low:
        d[alone] = np.float32(1.5 * 2.0 ** -45)
        b[alone] *= np.float32(2.0 ** -45)
    return a, d, b


def solve(w, h, a, d, b):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda:0")
    A, D, B = (torch.from_numpy(np.ascontiguousarray(v)).to(dev) for v in (a, d, b))
    x = torch.zeros((h * w, 2), dtype=torch.float32, device=dev)
    torch.cuda.synchronize()
    iters, _ = S.pressure_solve_static(w, h, A.data_ptr(), D.data_ptr(), B.data_ptr(), x.data_ptr(), 1e-4, 1e-4, 60)
    torch.cuda.synchronize()
    return iters, x.cpu().numpy()


def same(got, want):
    assert np.isfinite(want).all() and np.abs(want).max() > 0.0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), f"{np.count_nonzero(got != want)} values differ"


@pytest.mark.parametrize("w,h", [(33, 47), (160, 96)])
def test_small_couplings_and_diagonals(w, h):
    a, d, b = system(w, h, True)
    s = np.float32(2.0 ** 12)
    want_iters, want = solve(w, h, a * s, d * s, b * s)
    iters, got = solve(w, h, a, d, b)
    assert max(want_iters) > 1 and iters == want_iters
    same(got, want)


@pytest.mark.parametrize("w,h", [(33, 47), (160, 96)])
@pytest.mark.parametrize("power", [-40, -44])
def test_small_residuals(w, h, power):
    a, d, b = system(w, h, False)
    want_iters, want = solve(w, h, a, d, b)
    iters, got = solve(w, h, a, d, b * np.float32(2.0 ** power))
    assert max(want_iters) > 1 and iters == want_iters
    same(np.ldexp(got, -power), want)
