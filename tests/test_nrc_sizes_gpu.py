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
