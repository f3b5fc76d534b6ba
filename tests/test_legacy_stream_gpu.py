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
