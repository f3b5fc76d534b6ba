"""kgk_svgf_apply on records at the ends of the float range, against the
oracle's filter."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300._lib import check, lib
from test_svgf_align_gpu import records
from test_svgf_gpu import SVGF_RTOL

pytestmark = pytest.mark.gpu


def both(W, H, noisy, cur):
    """(result, filtered, records) of the first frame, ours and the oracle's."""
    from oracle import orc
    out = []
    for gpu in (True, False):
        r, f, p, c = noisy.copy(), np.zeros_like(noisy), np.zeros_like(cur), cur.copy()
        if gpu:
            check(lib().kgk_svgf_apply(*(ctypes.c_void_p(a.ctypes.data) for a in (r, f, p, c)), W, H, 0))
        else:
            orc.svgf_compat(W, H, r, f, p.view(np.uint8), c.view(np.uint8), 0)
        out.append((r, f, c))
    return out


@pytest.mark.parametrize("gradient", [1.0, 1e30, 3e37])
def test_depth_gradients(gradient):
    """A plane seen edge-on, from slopes of 1 to slopes whose tap distances pass
    2^126: the weights depend on the ratio of depth and slope alone.  The two
    differ by the rounding of the weights, 2^-21 of them a pass."""
    W, H = 10, 8  # depths up to 2.7e38
    rng = np.random.default_rng(1)
    n = W * H
    noisy = rng.uniform(0.5, 1.5, (n, 4)).astype(np.float32)
    noisy[:, 3] = 0
    cur = records(rng, n)
    cur[:, 0:3] = 0.5
    cur[:, 8:11] = (0, 0, 1)
    cur.view(np.int32)[:, 16:18] = 3
    cur[:, 26] = np.float32(gradient) * np.tile(np.arange(W, dtype=np.float32), H)
    (r, f, c), (ro, fo, co) = both(W, H, noisy, cur)
    for a, b in ((r, ro), (f, fo), (c[:, 25:26], co[:, 25:26])):
        assert (np.abs(a - b) <= SVGF_RTOL * np.maximum(np.abs(b), 1e-3)).all()


@pytest.mark.parametrize("what", ["radiance / albedo", "albedo", "depth", "all"])
@pytest.mark.parametrize("flags", [False, True])
def test_values_that_are_no_numbers(what, flags):
    """Radiance over albedo that is infinite, an albedo and a depth that are no
    numbers, with and without pixels that have no luminance weight: NaN in the
    same places as in the oracle, also in the records.  (A pixel whose
    blurred variance is exactly 0 is not filtered; the device's multiply-adds
    leave some a rounding error there, so variances are compared where the flag
    is the same.)"""
    W, H = 112, 40
    rng = np.random.default_rng(2)
    n = W * H
    noisy = rng.uniform(0.5, 1.5, (n, 4)).astype(np.float32)
    noisy[:, 3] = 0
    cur = records(rng, n)
    grid, ids = cur.reshape(H, W, 28), cur.view(np.int32).reshape(H, W, 28)
    ids[:, :, 16] = np.where(np.arange(W)[None] // 36 == 1, -1, 3)  # the gap: columns 36 to 71
    if what in ("radiance / albedo", "all"):
        grid[10:13, 5:8, 0:3] = -np.float32(1e-4)  # a divisor of 0
    if what in ("albedo", "all"):
        grid[30, 20, 0] = np.nan
    if what in ("depth", "all"):
        grid[20, 9, 26] = np.nan
    if flags:
        ids[:, :, 27] = np.where(np.arange(H)[:, None] % 4 == 3, 0, 1)
    (r, f, c), (ro, fo, co) = both(W, H, noisy, cur)
    cols = c.view(np.int32)[:, 16:18], co.view(np.int32)[:, 16:18]
    assert np.array_equal(*cols)
    assert np.isnan(co[:, 25]).any() and np.isfinite(co[:, 25]).any()
    for a, b in ((r, ro), (f, fo), (c[:, 12:16], co[:, 12:16]), (c[:, 23:25], co[:, 23:25])):
        assert np.array_equal(np.isnan(a), np.isnan(b))
    flag = c.view(np.int32)[:, 27] == co.view(np.int32)[:, 27]
    assert flag.mean() > 0.99
    assert np.array_equal(np.isnan(c[flag, 25]), np.isnan(co[flag, 25]))
