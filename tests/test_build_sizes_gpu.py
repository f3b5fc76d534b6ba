"""BVH builds at the sizes where the builder changes its ways: one leaf, one
primitive per lane (32), a warp per node, one block per task (2048), large
tasks split by the grid; with coincident and flat triangles among them.  The
tree must validate and its closest hits must be the brute-force ones."""
import numpy as np
import pytest

from kagayaki_gb300 import Scene, scenes
from kagayaki_gb300.structs import TRIANGLE, make_material
from oracle import orc

pytestmark = pytest.mark.gpu


def soup(n, kind, seed):
    rng = np.random.default_rng(seed)
    tris = np.zeros(n, TRIANGLE)
    c = rng.uniform(-4, 4, (n, 1, 3))
    if kind == "flat":
        c[:, :, 2] = 1.0
    v = c + rng.uniform(-0.4, 0.4, (n, 3, 3))
    if kind == "flat":
        v[:, :, 2] = 1.0
    if kind == "coincident":  # most centroids in one bin on every axis: split by position
        v[n // 8:] = v[:1]
    tris["verts"][:, :3, :3] = v
    tris["verts"][:, 3:6, 2] = 1.0
    return tris


@pytest.mark.parametrize("kind", ["random", "flat", "coincident"])
@pytest.mark.parametrize("n", [1, 3, 4, 31, 32, 33, 34, 65, 97, 2047, 2048, 2049, 4099])
def test_build_sizes(n, kind):
    tris = soup(n, kind, n)
    rays = scenes.parity_rays(2048, (-5, -5, -5), (5, 5, 5), seed=n)
    with Scene(tris, np.stack([make_material()])) as s:
        s.build_bvh()
        s.validate_bvh()
        ids, t = s.trace_closest(rays)
        occ = s.trace_any(rays)
    oids, ot = orc.closest_brute(tris, rays)
    ok = orc.classify(tris, rays, oids, ot) == 0  # no tie, no edge graze
    assert np.array_equal(ids[ok], oids[ok])
    hit = ok & (oids >= 0)
    assert np.array_equal(t[hit], ot[hit])
    assert np.array_equal(occ[ok] != 0, oids[ok] >= 0)


def test_large_scene_leaves():
    """Above 65,536 triangles every leaf holds one triangle."""
    tris = soup(65537, "random", 3)
    with Scene(tris, np.stack([make_material()])) as s:
        info = s.build_bvh()
        s.validate_bvh()
    assert info["max_leaf_size"] == 1 and info["n_binary_nodes"] == 2 * 65537 - 1


@pytest.mark.parametrize("n", [(1 << 20) - 1, (1 << 20) + 1])
def test_large_level_chunks(n):
    """The size of the chunks that large levels are binned and partitioned in
    changes at 2^20 triangles."""
    tris = soup(n, "random", n)
    tris["verts"][:, 1:3, :3] = tris["verts"][:, :1, :3] + 0.02 * (tris["verts"][:, 1:3, :3] - tris["verts"][:, :1, :3])
    rays = scenes.parity_rays(128, (-5, -5, -5), (5, 5, 5), seed=n)
    with Scene(tris, np.stack([make_material()])) as s:
        s.build_bvh()
        s.validate_bvh()
        ids, t = s.trace_closest(rays)
    oids, ot = orc.closest_brute(tris, rays)
    ok = orc.classify(tris, rays, oids, ot) == 0
    assert np.array_equal(ids[ok], oids[ok])
    hit = ok & (oids >= 0)
    assert np.array_equal(t[hit], ot[hit])
