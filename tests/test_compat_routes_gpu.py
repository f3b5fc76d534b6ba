"""The reference's estimator renders a small scene and image a pixel per
thread, anything else in waves.  Adding triangles that no ray meets takes the
same picture from one way to the other: frames, accumulators, G-buffer records
and ray counts must not change, at sizes around a warp, a block and the rule's
pixel limit."""
import numpy as np
import pytest

from kagayaki_gb300 import ESTIMATOR_COMPAT, ESTIMATOR_UNBIASED, Scene, camera_setup, scenes

pytestmark = pytest.mark.gpu


def far_away(tris, n):
    """n specks far below the box."""
    rng = np.random.default_rng(1)
    extra = np.repeat(tris[:1], n)
    extra["verts"][:, :3, :3] = np.float32((0, -1e4, 0)) + rng.uniform(-1e-3, 1e-3, (n, 3, 3)).astype(np.float32)
    return np.concatenate([tris, extra])


@pytest.mark.parametrize("kind", ["cornell", "disney"])
@pytest.mark.parametrize("W,H,spp,depth", [(1, 1, 2, 0), (7, 5, 3, 0), (33, 31, 2, 3), (97, 61, 3, 0),
                                           (400, 380, 1, 0), (400, 400, 1, 0)])
def test_routes_agree(kind, W, H, spp, depth):
    tris, mats, c, tex, env = scenes.parity_scene(kind)
    got = []
    for t in (tris, far_away(tris, 2000)):
        with Scene(t, mats, textures=tex, env=env) as s:
            s.build_bvh()
            cam = camera_setup(c["origin"], c["dist"], c["rot"], H)
            s.accum_reset(W, H)
            frames, counts = [], []
            for f in range(2):  # the second call goes on from the first one's seeds
                img, st = s.render(cam, W, H, spp=spp, max_depth=depth, estimator=ESTIMATOR_COMPAT, frame_index=f,
                                   accumulate=True, write_gbuffer=True)
                frames.append(img)
                counts.append((st["rays_closest"], st["rays_shadow"], st["paths"]))
            rec = s.gbuffer_records(W, H)
            got.append((np.stack(frames), counts, s.accum_read(W, H), rec))
    (fa, ca, (ma, va, na), ra), (fb, cb, (mb, vb, nb), rb) = got
    assert np.array_equal(fa, fb, equal_nan=True)
    assert ca == cb and na == nb == 2 * spp
    assert np.array_equal(ma, mb, equal_nan=True) and np.array_equal(va, vb, equal_nan=True)
    for k in ("Albedo", "Normal", "Depth", "MaterialID", "ObjectID"):
        assert np.array_equal(ra[k], rb[k], equal_nan=ra[k].dtype.kind == "f"), k


@pytest.mark.parametrize("kind", ["cornell", "disney"])
@pytest.mark.parametrize("W,H,spp", [(1, 1, 1), (97, 61, 3), (640, 300, 1), (333, 207, 4)])
def test_small_tree_loops_agree(kind, W, H, spp):
    """Waves on a small scene trace a ray per lane, on a larger one by the warp's
    (ray, triangle) pairs: the same hits, so the same unbiased frames."""
    tris, mats, c, tex, env = scenes.parity_scene(kind)
    got = []
    for t in (tris, far_away(tris, 2000)):
        with Scene(t, mats, textures=tex, env=env) as s:
            s.build_bvh()
            cam = camera_setup(c["origin"], c["dist"], c["rot"], H)
            img, st = s.render(cam, W, H, spp=spp, estimator=ESTIMATOR_UNBIASED)
            got.append((img, (st["rays_closest"], st["rays_shadow"], st["paths"])))
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
    assert got[0][1] == got[1][1]
