"""A tensor-core wait that runs out (give_up_waits: all of them do, at once) is
an error that the call returns; what was in flight is waited for, and the GPU
stays usable: without it the next call gives what it gave before."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300 import KgkError, Scene, scenes
from kagayaki_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def infer(s, raw):
    out = np.full((len(raw), 3), np.nan, np.float32)
    check(lib().kgk_nrc_infer(s._h, _p(raw), len(raw), _p(out)))
    return out


@pytest.fixture(params=[64, 128], ids=["w64", "w128"])
def cache(request):
    tris, mats, _ = scenes.cornell_box()
    with Scene(tris, mats) as s:
        s.width = request.param
        s.cache_init(width=s.width, seed=3)
        yield s


# one tile, a tile and a query, several rounds of all tiles in flight
@pytest.mark.parametrize("n", [1, 129, 152 * 4 * 128 * 2 + 77])
def test_inference(cache, n):
    raw = np.random.default_rng(n).random((n, 13), dtype=np.float32)
    want = infer(cache, raw)
    assert np.isfinite(want).all()
    for _ in range(2):
        cache.cache_init(width=cache.width, seed=3, give_up_waits=1)
        with pytest.raises(KgkError, match="timed out"):
            infer(cache, raw)
        cache.cache_init(width=cache.width, seed=3)
        assert np.array_equal(infer(cache, raw), want)
