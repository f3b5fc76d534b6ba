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
