"""kgk_svgf_apply on device arrays that start on 4 bytes only (a sub-array of a
larger buffer): the same results as on 16-byte starts, for the first frame
(previous records initialised) and the next, at sizes around the filter's
tiles."""
import ctypes

import numpy as np
import pytest

from kagayaki_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def records(rng, n):
    r = np.zeros((n, 28), np.float32)
    i = r.view(np.int32)
    r[:, 0:3] = rng.uniform(0.05, 0.95, (n, 3))
    nv = rng.normal(size=(n, 3))
    r[:, 8:11] = nv / np.linalg.norm(nv, axis=1, keepdims=True)
    i[:, 16] = np.where(rng.random(n) < 0.1, -1, 3)
    i[:, 17] = rng.integers(0, 3, n)
    i[:, 18:20] = -1
    r[:, 20:22] = -1
    r[:, 23:25] = -1
    r[:, 26] = rng.uniform(1, 5, n)
    i[:, 27] = 1
    return r


@pytest.mark.parametrize("W,H", [(2, 2), (31, 9), (33, 17), (260, 37)])
def test_misaligned_arrays(W, H):
    import torch
    rng = np.random.default_rng(W)
    n = W * H
    noisy = rng.exponential(1.0, (n, 4)).astype(np.float32)
    cur, prev = records(rng, n), records(rng, n)
    got = []
    for off in (0, 1):
        bufs = []
        for a in (noisy, np.zeros_like(noisy), prev, cur):
            t = torch.zeros(a.size + 4, device="cuda")
            t[off:off + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
            bufs.append(t)
        torch.cuda.synchronize()
        out = []
        for frame in (0, 1):
            check(lib().kgk_svgf_apply(*(ctypes.c_void_p(t.data_ptr() + 4 * off) for t in bufs), W, H, frame))
            out += [t[off:off + s].cpu().numpy().view(np.int32).copy()
                    for t, s in zip(bufs, (4 * n, 4 * n, 28 * n, 28 * n))]
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)
