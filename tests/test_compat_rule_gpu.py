"""The reference's estimator on small scenes, where it changes between a pixel
per thread and waves: what a call reports and renders does not depend on the way
it takes."""
import numpy as np
import pytest

from kagayaki_gb300 import ESTIMATOR_COMPAT, Scene, camera_setup, scenes

pytestmark = pytest.mark.gpu


def rendered(n_far, W, H, spp, **kw):
    from test_compat_routes_gpu import far_away
    tris, mats, c, tex, env = scenes.parity_scene("cornell")
    with Scene(far_away(tris, n_far), mats, textures=tex, env=env) as s:
        s.build_bvh()
        s.accum_reset(W, H)
        cam = camera_setup(c["origin"], c["dist"], c["rot"], H)
        img, st = s.render(cam, W, H, spp=spp, estimator=ESTIMATOR_COMPAT, accumulate=True, **kw)
        return img.copy(), st, s.accum_read(W, H)


def same(a, b):
    assert np.array_equal(a[0], b[0], equal_nan=True)
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a[2], b[2]))
    assert [a[1][k] for k in ("rays_closest", "rays_shadow", "paths")] == \
           [b[1][k] for k in ("rays_closest", "rays_shadow", "paths")]


@pytest.mark.parametrize("W,H", [(363, 362), (400, 380), (450, 450)])
def test_work_is_counted_above_the_tail_kernels_waves(W, H):
    plain, counted = rendered(0, W, H, 2), rendered(0, W, H, 2, count_work=True)
    same(plain, counted)
    st = counted[1]
    assert st["extend_launches"] >= 2
    assert st["nodes_visited"] >= st["rays_closest"] - st["rays_tail"] > 0
    assert st["tris_tested"] > 0


def test_samples_of_a_launch():
    """64 samples a launch: the same sums as a wave per sample, and no launch holds
    the GPU for a whole call of many."""
    launches = []
    for spp in (64, 65, 130):
        got = rendered(0, 33, 31, spp)
        same(got, rendered(2000, 33, 31, spp))
        launches.append(got[1]["kernel_launches"])
    assert [n - launches[0] for n in launches] == [0, 1, 2]


@pytest.mark.parametrize("n_tris,W,H,spp", [
    (n, W, H, spp) for n, W, H in ((128, 97, 61), (129, 97, 61), (129, 363, 361), (129, 364, 361))
    for spp in (1, 2, 3)] + [(36, 416, 404, 1), (36, 418, 403, 1)])
def test_both_sides_of_the_lines(n_tris, W, H, spp):
    """Triangles and samples, paths of a wave of the tail kernel (363 x 361 is the
    last size), pixels: as with more triangles than the kernel takes."""
    same(rendered(n_tris - 36, W, H, spp), rendered(2000, W, H, spp))


@pytest.mark.parametrize("kind", ["cornell", "disney"])
@pytest.mark.parametrize("n_tris", [256, 257, 1024, 1025])
def test_lines_of_the_loops(kind, n_tris):
    """Waves of 262,144 paths, whose bounces trace by loops, by loops and then by the
    warp's pairs, or by pairs: unbiased frames as with many more triangles."""
    from kagayaki_gb300 import ESTIMATOR_UNBIASED
    from test_compat_routes_gpu import far_away
    tris, mats, c, tex, env = scenes.parity_scene(kind)
    got = []
    for n in (n_tris, 4000):
        with Scene(far_away(tris, n - len(tris)), mats, textures=tex, env=env) as s:
            s.build_bvh()
            cam = camera_setup(c["origin"], c["dist"], c["rot"], 256)
            img, st = s.render(cam, 512, 256, spp=2, estimator=ESTIMATOR_UNBIASED, accumulate=False)
            got.append((img.copy(), st["extend_launches"], st["rays_closest"], st["rays_shadow"]))
    assert got[0][1] >= 2 and got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
