"""One path a pixel: small films by the pixel loop (one launch), larger ones by a lane per path; the same films."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


# 2^15 pixels on trees below 128 four-wide nodes, 2^17 on others, and either side of them
@pytest.mark.parametrize("kind,w,h,loop", [("box", 256, 128, True), ("box", 151, 218, False), ("sphere", 512, 256, True),
                                           ("sphere", 341, 385, False), ("box", 1, 1, True)])
def test_forms_by_film_size(ctx, kind, w, h, loop):
    scene = ab.Scene(ctx, scenes.box_scene(w, h) if kind == "box" else scenes.sphere_scene(w, h))
    got = scene.render(ab.render_opts(1, 5, 3, 8))
    assert (got.stats["launches"] == 1) == loop
    want = scene.render(ab.render_opts(1, 5, 3, 8, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 18, wf_block=128, wf_sort=1))
    near = np.isclose(got.film, want.film, rtol=1e-6, atol=1e-7).all(-1)
    assert (~near).sum() <= 1e-5 * w * h          # exact-distance ties, as in the other film comparisons
    for k in ("camera_rays", "closest_rays", "shadow_rays", "paths"):
        if near.all():
            assert got.stats[k] == want.stats[k], k
    f64 = scene.render_f64(ab.render_opts(1, 5, 3, 8))
    np.testing.assert_array_equal(f64.film.astype(np.float32)[..., :3], got.film[..., :3])
    scene.close()


@pytest.mark.parametrize("spp,lights,offset,loop", [(1, 1, 7, True), (1, 4, 0, True), (1, 4, 1, False), (2, 1, 0, False)])
def test_forms_by_paths_a_pixel(ctx, spp, lights, offset, loop):
    """Light samples give every sample but the render's first several paths."""
    scene = ab.Scene(ctx, scenes.box_scene(40, 30))
    o = dict(sample_offset=offset, light_samples=lights)
    got = scene.render(ab.render_opts(spp, 4, 3, 8, **o))
    assert (got.stats["launches"] == 1) == loop
    assert got.stats["paths"] == 1200 * (spp * lights - (lights - 1 if offset == 0 else 0))
    want = scene.render(ab.render_opts(spp, 4, 3, 8, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 14, wf_block=128, wf_sort=1, **o))
    np.testing.assert_allclose(got.film, want.film, rtol=1e-6, atol=1e-7)
    scene.close()
