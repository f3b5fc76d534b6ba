"""Cache inference at batch sizes around a tile (128 queries) and around one
round of all tiles in flight: a query's prediction does not depend on the batch
it comes in, so every prefix gives the large batch's values bit for bit; angles
far outside the unit range and NaN queries stay in their own rows."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300 import Scene, scenes
from kagayaki_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def infer(s, raw):
    out = np.full((len(raw), 3), np.nan, np.float32)
    check(lib().kgk_nrc_infer(s._h, ctypes.c_void_p(raw.ctypes.data), len(raw), ctypes.c_void_p(out.ctypes.data)))
    return out


@pytest.mark.parametrize("width", [64, 128])
def test_prefixes(width):
    tris, mats, _ = scenes.cornell_box()
    rng = np.random.default_rng(width)
    n = 152 * 4 * 128 * 2 + 77
    raw = rng.random((n, 13), dtype=np.float32)
    raw[5, :3] = 1e9
    raw[9, 3] = np.nan
    with Scene(tris, mats) as s:
        s.cache_init(width=width, seed=3)
        full = infer(s, raw)
        ok = np.ones(n, bool)
        ok[9] = False
        assert np.isfinite(full[ok]).all()
        for m in (1, 31, 127, 128, 129, 255, 257, 1000, 152 * 4 * 128, 152 * 4 * 128 + 1):
            assert np.array_equal(infer(s, raw[:m]), full[:m], equal_nan=True), m
        # rows do not mix: without the odd ones the others are the same
        plain = raw.copy()
        plain[[5, 9]] = 0.5
        ok[5] = False
        assert np.array_equal(infer(s, plain)[ok], full[ok])


@pytest.mark.parametrize("width", [64, 128])
def test_gradients_as_the_scratch_grows(width):
    """Sizes around a tile and around one round of all tiles in flight, each
    larger than the last, so that the call grows the training scratch; a second
    call of the size finds it there.  The FP32 sums differ by their order only."""
    tris, mats, _ = scenes.cornell_box()
    rng = np.random.default_rng(width)
    with Scene(tris, mats) as s:
        s.cache_init(width=width, seed=3)
        n_params = 64 * width + 4 * width * width + 3 * width
        for n in (1, 127, 129, 4096, 152 * 2 * 128, 152 * 4 * 128 + 1, 1 << 17, 1 << 18):
            raw = rng.random((n, 13), dtype=np.float32)
            tgt = rng.random((n, 3), dtype=np.float32)
            g = [np.full(n_params, np.nan, np.float32) for _ in range(2)]
            for k in range(2):
                check(lib().kgk_nrc_gradients(s._h, ctypes.c_void_p(raw.ctypes.data), ctypes.c_void_p(tgt.ctypes.data),
                                              n, ctypes.c_void_p(g[k].ctypes.data), None))
            norm = np.linalg.norm(g[1])
            assert np.isfinite(norm) and norm > 0
            assert np.linalg.norm(g[0] - g[1]) <= 1e-3 * norm, n
