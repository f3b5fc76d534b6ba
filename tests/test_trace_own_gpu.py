"""Batch queries on trees of a few nodes test each lane's own triangles, on larger
ones (and for small closest-hit batches) the warp's (ray, triangle) pairs: the
same answers, on both sides of the lines in triangles and rays."""
import numpy as np
import pytest

from kagayaki_gb300 import Scene, scenes
from kagayaki_gb300.structs import LAMBERT, RAY, TRIANGLE, make_material

pytestmark = pytest.mark.gpu


def triangles(n, width, coincident=0):
    rng = np.random.default_rng(n)
    p = rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(size=(n, 3, 3)) * width
    p[:coincident] = p[0]  # ties: the smallest id
    t = np.zeros(n, TRIANGLE)
    t["verts"][:, :3, :3] = p
    t["verts"][:, 3:6, 2] = 1
    return scenes.canonical(t)


def far(tris, n):
    """n specks that no ray of rays() meets."""
    extra = np.repeat(tris[:1], n)
    rng = np.random.default_rng(1)
    extra["verts"][:, :3, :3] = np.float32((0, -1e6, 0)) + rng.uniform(-1, 1, (n, 3, 3)).astype(np.float32)
    return np.concatenate([tris, extra])


def rays(n):
    rng = np.random.default_rng(2)
    r = np.zeros(n, RAY)
    r["org"][:, :3] = rng.uniform(-2, 2, (n, 3))
    r["org"][:, 1] = np.abs(r["org"][:, 1])
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:200, 0] = 0
    d[200:400, 2] = -0.0
    d[400:500] = (0, 0, 1)
    r["dir"][:, :3] = d
    # straight down to the specks: none
    down = (d[:, 1] < 0) & (np.hypot(d[:, 0], d[:, 2]) < 1e-3)
    r["dir"][down, 1] *= -1
    limit = rng.uniform(0, 3, n).astype(np.float32)
    limit[::7] = np.array([np.inf, 0, -1, np.nan, 1e38, -0.0, 1e-6], np.float32)[np.arange(len(limit[::7])) % 7]
    return r, limit


def scene(t):
    s = Scene(t, np.stack([make_material(LAMBERT, (0.5, 0.5, 0.5))]))
    s.build_bvh()
    return s


@pytest.mark.parametrize("n,width,coincident", [(1, 0.5, 0), (2, 0.5, 2), (24, 0.3, 5), (128, 0.1, 0), (1000, 0.05, 40),
                                                (1024, 0.3, 0)])
@pytest.mark.parametrize("n_rays", [1, 31, 100_003])
def test_any_hit(n, width, coincident, n_rays):
    r, limit = rays(n_rays)
    t = triangles(n, width, coincident)
    with scene(t) as own, scene(far(t, 1100)) as pairs:
        for m in (None, limit):
            assert np.array_equal(own.trace_any(r, m), pairs.trace_any(r, m))


@pytest.mark.parametrize("n,width,coincident", [(1, 0.5, 0), (24, 0.3, 5), (128, 0.1, 30), (128, 0.5, 0)])
def test_closest_hit(n, width, coincident):
    r, _ = rays((1 << 18) + 77)
    t = triangles(n, width, coincident)
    with scene(t) as s, scene(far(t, 129 - n)) as pairs:
        ids, dist, st = s.trace_closest(r, with_stats=True)
        want_ids, want, _ = pairs.trace_closest(r, with_stats=True)
        assert np.array_equal(ids, want_ids) and np.array_equal(dist, want)
        assert (ids >= 0).any() and st["nodes_visited"] >= len(r) and st["tris_tested"] > 0
        part = [s.trace_closest(c) for c in np.array_split(r, 3)]  # below the line in rays
        assert np.array_equal(np.concatenate([p[0] for p in part]), ids)
        assert np.array_equal(np.concatenate([p[1] for p in part]), dist)
