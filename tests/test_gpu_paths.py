"""The plain renderer (one lane per path) against the pixel loop of the renderer that allocates nothing: same
films, bit for bit, and the same ray counts."""
import ctypes as C

import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _pixel_loop(scene, opts):
    import torch
    film = torch.zeros((scene.height, scene.width, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    st = _abi.RenderStats()
    _abi.check(_abi.lib().aur_render_fp64acc_noalloc(scene.handle, C.byref(opts), film.data_ptr(), C.byref(st)), "noalloc")
    return film.cpu().numpy(), st


def _scene(kind, w, h):
    if kind == "glass":
        glass = dict(type_=_abi.MAT_GLASS, specular=(0.9, 0.9, 0.9), diffuse=(0.9, 0.8, 0.9), reflectance=0.1, ior=1.4)
        return scenes.sphere_scene(w, h, env=dict(color=(0.3, 0.4, 0.5)), sphere_mat=glass)
    if kind == "shaders":
        return scenes.shader_scene(w, h)
    if kind == "terrain":        # roulette from the third bounce; enough nodes for the quantised closest hits
        return scenes.terrain_scene(w, h, grid=300, spheres=8)
    return scenes.box_scene(w, h)


@pytest.mark.parametrize("kind,depth", [("box", 1), ("box", 5), ("glass", 2), ("glass", 7), ("shaders", 4), ("terrain", 8)])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (37, 23, 5), (128, 64, 3)])
@pytest.mark.parametrize("lights,offset", [(1, 0), (3, 0), (2, 4)])
def test_films_and_counts(ctx, kind, depth, w, h, spp, lights, offset):
    data = _scene(kind, w, h)
    scene = ab.Scene(ctx, data)
    o = dict(sample_offset=offset, light_samples=lights, fp64_film=1)
    opts = ab.render_opts(spp, depth, min(depth, data.render["min_depth"]), 11, **o)
    want, st = _pixel_loop(scene, opts)
    got = scene.render(opts)
    np.testing.assert_array_equal(got.film, want)
    f64 = scene.render_f64(opts).film
    np.testing.assert_array_equal(f64.astype(np.float32)[..., :3], want[..., :3])
    for k in ("camera_rays", "closest_rays", "shadow_rays", "paths"):
        assert got.stats[k] == getattr(st, k), k
    scene.close()


def test_render_in_chunks_of_samples(ctx):
    """More samples than the 1 GiB sample buffer holds: 256 x 256 x 1100 (two chunks, FP32 and FP64 sums kept
    between them)."""
    scene = ab.Scene(ctx, scenes.box_scene(256, 256))
    for fp64 in (1, 0):
        opts = ab.render_opts(1100, 2, 2, 3, fp64_film=fp64)
        got = scene.render(opts)
        opts.fp64_film = 1
        want, st = _pixel_loop(scene, opts)
        if fp64:
            np.testing.assert_array_equal(got.film, want)
        else:       # compensated FP32 sums: within a few ulp of the FP64 ones
            np.testing.assert_allclose(got.film, want, rtol=5e-7, atol=1e-9)
        assert got.stats["closest_rays"] == st.closest_rays and got.stats["paths"] == 256 * 256 * 1100
    scene.close()
