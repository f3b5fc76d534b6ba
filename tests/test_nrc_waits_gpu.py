"""A tensor-core wait that runs out (give_up_waits: all of them do, at once) is
an error that the call returns; what was in flight is waited for, and the GPU
stays usable: without it the next call gives what it gave before."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300 import ESTIMATOR_UNBIASED, KgkError, Scene, camera_setup, scenes
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


@pytest.mark.parametrize("n", [1, 300, 1 << 17])
def test_training(cache, n):
    """Neither a gradient nor a step comes of it: weights and loss scale stay."""
    rng = np.random.default_rng(n)
    raw, tgt = (rng.random((n, k), dtype=np.float32) for k in (13, 3))
    w = [np.empty(64 * cache.width + 4 * cache.width**2 + 3 * cache.width, np.float32) for _ in range(3)]
    loss = np.full(1, -1, np.float32)

    def gradients(g):
        check(lib().kgk_nrc_gradients(cache._h, _p(raw), _p(tgt), n, _p(g), _p(loss)))

    gradients(w[0])
    assert loss[0] > 0
    cache.cache_init(width=cache.width, seed=3, give_up_waits=1)
    check(lib().kgk_nrc_get_weights(cache._h, _p(w[1]), w[1].size))
    loss[0] = -1
    for _ in range(2):
        with pytest.raises(KgkError, match="timed out"):
            gradients(w[2])
        with pytest.raises(KgkError, match="timed out"):
            check(lib().kgk_nrc_train(cache._h, _p(raw), _p(tgt), n, 3, _p(loss)))
    assert loss[0] == -1
    check(lib().kgk_nrc_get_weights(cache._h, _p(w[2]), w[2].size))
    assert np.array_equal(w[1], w[2])
    scale = np.zeros(1, np.float32)
    check(lib().kgk_nrc_loss_scale(cache._h, _p(scale)))
    assert scale[0] == 128
    cache.cache_init(width=cache.width, seed=3)
    gradients(w[1])  # FP32 atomics: the order of the sums differs
    assert np.linalg.norm(w[1] - w[0]) <= 1e-3 * np.linalg.norm(w[0])


def test_cached_frame(cache):
    c = scenes.cornell_box()[2]
    cache.build_bvh()
    cam = camera_setup(c["origin"], c["dist"], c["rot"], 96)
    want, _ = cache.render(cam, 96, 96, estimator=ESTIMATOR_UNBIASED, use_cache=True)
    cache.cache_init(width=cache.width, seed=3, give_up_waits=1)
    with pytest.raises(KgkError, match="timed out"):
        cache.render(cam, 96, 96, estimator=ESTIMATOR_UNBIASED, use_cache=True)
    cache.cache_init(width=cache.width, seed=3)
    got, _ = cache.render(cam, 96, 96, estimator=ESTIMATOR_UNBIASED, use_cache=True)
    assert np.array_equal(got, want)  # the first frame: untrained weights
