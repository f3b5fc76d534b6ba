"""Batch queries where the warp's triangle lists take their edge forms: more
pairs than a lane lists at a time and than a warp tests at a time (stacked
triangles, every ray through all of them), equal distances (coincident
triangles: the smaller id wins), partial warps, occlusion limits on the hit
distance, and directions with negative zeros."""
import numpy as np
import pytest

from kagayaki_gb300 import Scene
from kagayaki_gb300.structs import RAY, TRIANGLE, make_material
from oracle import orc

pytestmark = pytest.mark.gpu


def stack(n, coincident):
    """n large triangles across the z axis, at z = 0, 1/8, 2/8, ... (or all at 0)."""
    tris = np.zeros(n, TRIANGLE)
    base = np.array([[-9, -8, 0], [10, -9, 0], [0.5, 11, 0]], np.float32)
    tris["verts"][:, :3, :3] = base
    if not coincident:
        tris["verts"][:, :3, 2] = np.arange(n, dtype=np.float32)[:, None] / 8
    tris["verts"][:, 3:6, 2] = 1.0
    return tris


def down(n, seed, height):
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, RAY)
    rays["org"][:, :2] = rng.uniform(-2, 2, (n, 2))
    rays["org"][:, 2] = height
    rays["dir"][:, :2] = rng.uniform(-0.05, 0.05, (n, 2))
    rays["dir"][:, 2] = -1.0
    return rays


@pytest.mark.parametrize("coincident", [False, True])
@pytest.mark.parametrize("n_tris", [1, 3, 24, 25, 200])
@pytest.mark.parametrize("n_rays", [1, 31, 32, 33, 1000])
def test_stacked(n_rays, n_tris, coincident):
    tris = stack(n_tris, coincident)
    rays = down(n_rays, n_rays + n_tris, 60.0)
    rays["org"][::3, 2] = -5.0  # from below, and away from everything
    rays["dir"][::3, 2] = 1.0
    rays["dir"][::9, 2] = -1.0
    with Scene(tris, np.stack([make_material()])) as s:
        s.build_bvh()
        ids, t = s.trace_closest(rays)
        oids, ot = orc.closest_brute(tris, rays)
        assert np.array_equal(ids >= 0, oids >= 0)
        assert np.array_equal(t, ot)
        hit = ids >= 0
        # no two of the stacked triangles share a distance; of coincident ones the first wins
        assert np.array_equal(ids[hit], np.zeros(hit.sum(), np.int32) if coincident else oids[hit])
        # an occlusion limit excludes the distance itself
        lim = np.where(hit, t, np.float32(1.0)).astype(np.float32)
        assert not s.trace_any(rays, lim).any()
        assert np.array_equal(s.trace_any(rays, np.nextafter(lim, np.float32(1e30))) != 0, hit)
        assert np.array_equal(s.trace_any(rays) != 0, hit)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_negative_zero_directions(axis):
    """-0 in a direction is 0: rays along an axis hit the same triangles."""
    rng = np.random.default_rng(axis)
    tris = np.zeros(500, TRIANGLE)
    tris["verts"][:, :3, :3] = rng.uniform(-4, 4, (500, 1, 3)) + rng.uniform(-1, 1, (500, 3, 3))
    rays = np.zeros(4096, RAY)
    rays["org"][:, :3] = rng.uniform(-4, 4, (4096, 3))
    rays["org"][:, axis] = -9.0
    rays["dir"][:, axis] = 1.0
    neg = rays.copy()
    for a in range(3):
        if a != axis:
            neg["dir"][:, a] = -0.0
    with Scene(tris, np.stack([make_material()])) as s:
        s.build_bvh()
        ids, t = s.trace_closest(rays)
        nids, nt = s.trace_closest(neg)
        occ, nocc = s.trace_any(rays), s.trace_any(neg)
    assert (ids >= 0).any()
    assert np.array_equal(ids, nids) and np.array_equal(t, nt) and np.array_equal(occ, nocc)
