"""kgk_svgf_apply on records whose previous position lies outside the image: a
pixel without history, whichever edge it left by.  None of the cases has a
pixel of the image among the four that history is blended from, so the results
are those of records without a previous position."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300._lib import check, lib
from test_svgf_align_gpu import records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 2), (33, 17), (260, 37)])
def test_previous_position_outside(W, H):
    rng = np.random.default_rng(W)
    n = W * H
    noisy = rng.exponential(1.0, (n, 4)).astype(np.float32)
    noisy[:, 3] = 0
    prev = records(rng, n)
    prev.view(np.int32)[:, 22] = rng.integers(0, 9, n)  # sampleNum
    prev.view(np.int32)[:, 27] = 0x101                  # both flags: history to blend
    far = 1 << 30
    at = [(x, -2) for x in (0, W - 1)] + [(x, H) for x in (0, W - 1)] + [(W, H - 1), (-2, 0), (-2, -1), (W, H),
                                                                       (5, -far), (5, far), (far, far), (-far, 3)]
    # the index of a position outside on the left or right may still be a pixel's: not these
    at = [(x, y) for x, y in at if not 0 <= W * y + x < n]
    assert len(at) >= 9
    got = []
    for outside in (False, True):
        cur = records(np.random.default_rng(W + 1), n)
        cur.view(np.int32)[:, 16] = 3  # every pixel an object
        if outside:
            pos = np.array(at, np.int32)[np.arange(n) % len(at)]
            cur.view(np.int32)[:, 18:20] = pos
            cur[:, 20:22] = pos
        res, filt, p = noisy.copy(), np.zeros_like(noisy), prev.copy()
        check(lib().kgk_svgf_apply(*(ctypes.c_void_p(a.ctypes.data) for a in (res, filt, p, cur)), W, H, 1))
        assert (cur.view(np.int32)[:, 22] == 1).all()
        cur[:, 18:22] = 0
        got.append((res, filt, cur))
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))
