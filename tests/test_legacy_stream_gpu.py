"""Device memory handed to the library is filled on the legacy default stream,
while that stream is busy: what the library copies there is copied after it, and
before anything on the scene's own stream reads the copy."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300 import Scene, scenes
from kagayaki_gb300._lib import check, lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def keep_busy():
    torch.cuda._sleep(200_000_000)  # about 0.1 s


def _p(a):
    return ctypes.c_void_p(a.data_ptr() if hasattr(a, "data_ptr") else a.ctypes.data)


@pytest.mark.parametrize("width", [64, 128])
def test_cache_weights(width):
    rng = np.random.default_rng(width)
    n = 64 * width + 4 * width * width + 3 * width
    w = rng.normal(size=n).astype(np.float32) * np.float32(0.1)
    raw = rng.random((1000, 13), dtype=np.float32)
    tgt = rng.random((1000, 3), dtype=np.float32)
    out = [np.empty((1000, 3), np.float32) for _ in range(2)]
    tris, mats, _ = scenes.cornell_box()
    with Scene(tris, mats) as s:
        s.cache_init(width=width, seed=3)
        check(lib().kgk_nrc_set_weights(s._h, _p(w), n))
        check(lib().kgk_nrc_infer(s._h, _p(raw), 1000, _p(out[0])))
        s.cache_init(width=width, seed=4)
        host = torch.from_numpy(w).pin_memory()
        dev = torch.zeros(n, device="cuda")
        torch.cuda.synchronize()
        keep_busy()
        dev.copy_(host, non_blocking=True)
        check(lib().kgk_nrc_set_weights(s._h, _p(dev), n))
        check(lib().kgk_nrc_infer(s._h, _p(raw), 1000, _p(out[1])))
        assert np.array_equal(*out)
        # out again, before a step that changes them
        back = torch.zeros(n, device="cuda")
        torch.cuda.synchronize()
        keep_busy()
        check(lib().kgk_nrc_get_weights(s._h, _p(back), n))
        check(lib().kgk_nrc_train(s._h, _p(raw), _p(tgt), 1000, 1, None))
        assert np.array_equal(back.cpu().numpy(), w)


@pytest.mark.parametrize("rgba8", [False, True])
def test_textures(rgba8):
    import test_texture_gpu as T
    from kagayaki_gb300 import ESTIMATOR_UNBIASED, camera_setup
    from kagayaki_gb300.structs import KgkTexture, KgkTextureRGBA8
    rng = np.random.default_rng(5)
    if rgba8:
        tex = rng.integers(0, 256, (256, 256, 4), np.uint8)
        make, args = KgkTextureRGBA8, (256, 256)
    else:
        tex = rng.random((256, 256, 3), dtype=np.float32)
        make, args = KgkTexture, (256, 256, 3)
    tris, mats = T.quad_scene()
    env = np.ones((16, 32, 3), np.float32)
    cam = camera_setup((0.0, 0.0, 3.0), 28.0, (0.0, 0.0, 0.0), 64)

    def frame(s):
        s.build_bvh()
        return s.render(cam, 64, 64, spp=4, estimator=ESTIMATOR_UNBIASED, seed=5, max_depth=3)[0].copy()

    placeholder = [np.zeros((1, 1, 3), np.float32)]
    with Scene(tris, mats, textures=placeholder if rgba8 else [tex], env=env) as s:
        if rgba8:
            s.set_textures_rgba8([tex])
        want = frame(s)
    host = torch.from_numpy(tex).pin_memory()
    dev = torch.zeros_like(host, device="cuda")
    torch.cuda.synchronize()
    t = make()
    t.pixels = ctypes.cast(dev.data_ptr(), type(t.pixels)) if not rgba8 else dev.data_ptr()
    t.width, t.height = args[:2]
    if rgba8:
        with Scene(tris, mats, textures=placeholder, env=env) as s:
            keep_busy()
            dev.copy_(host, non_blocking=True)
            check(lib().kgk_scene_set_textures_rgba8(s._h, ctypes.byref(t), 1))
            got = frame(s)
    else:
        t.bpp = 3
        hdr = KgkTexture(env.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), 32, 16, 3)
        s = Scene.__new__(Scene)
        s._h, s.bvh = ctypes.c_void_p(), None
        keep_busy()
        dev.copy_(host, non_blocking=True)
        check(lib().kgk_scene_create(_p(tris), len(tris), _p(mats), len(mats), ctypes.byref(t), 1, ctypes.byref(hdr),
                                     ctypes.byref(s._h)))
        got = frame(s)
        s.close()
    assert np.array_equal(got, want)
