"""Quantised boxes and exact-distance ties against the pixel loop of the renderer that allocates nothing, which
walks the binary tree's full-precision boxes: small, flat and far-off geometry, and coincident sheets."""
import ctypes as C

import numpy as np
import pytest
import torch

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _pixel_loop(scene, opts):
    film = torch.zeros((scene.height, scene.width, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    st = _abi.RenderStats()
    _abi.check(_abi.lib().aur_render_fp64acc_noalloc(scene.handle, C.byref(opts), film.data_ptr(), C.byref(st)), "noalloc")
    return film.cpu().numpy(), st


def _soup(n, scale, dist):
    r = np.random.default_rng(3)
    b = scenes.SceneBuilder(64, 48, scale / dist, name="soup")
    m = b.material(_abi.MAT_MATTE, diffuse=(0.6, 0.5, 0.4))
    size = 0.2 * (400 / n) ** (1 / 3)
    c = r.uniform(-1, 1, (n, 1, 3)) * (1.0, 1.0, 0.3)
    v = (c + r.uniform(-size, size, (n, 3, 3)) * (1.0, 1.0, 0.01)).reshape(-1, 3)
    v = np.concatenate([v, [[-2, -2, -0.5], [2, -2, -0.5], [2, 2, -0.5], [-2, 2, -0.5]]])
    f = np.concatenate([np.arange(3 * n).reshape(-1, 3), [[3 * n, 3 * n + 1, 3 * n + 2], [3 * n, 3 * n + 2, 3 * n + 3]]])
    v = v * scale + np.array([0.0, 0.0, -dist])
    b.mesh(v, f, m)
    b.square_light(scenes.translate(0, 0.5 * scale, v[:, 2].max() + scale), 0.3 * scale, 0.3 * scale, (5.0, 5.0, 5.0))
    return b.build(render=dict(spp=8, max_depth=3, min_depth=3, seed=2))


# a 4-wide node holds at most three binary ones: 384 of those make 128 four-wide nodes or more (any hit quantised),
# 98,304 make 32,768 (closest hit too)
@pytest.mark.parametrize("n,nodes", [(2000, 384), (200000, 98304)])
@pytest.mark.parametrize("scale,dist", [(1.0, 3.0), (1e-3, 0.5), (1e4, 3e5)])
def test_films_match_the_binary_tree(ctx, n, nodes, scale, dist):
    scene = ab.Scene(ctx, _soup(n, scale, dist))
    assert scene.bvh().info()["num_nodes"] >= nodes
    opts = ab.render_opts(8, 3, 3, 2, fp64_film=1)
    want, st = _pixel_loop(scene, opts)
    assert want[..., 3].max() > 0 and st.shadow_rays > 0
    plain = scene.render(opts)
    np.testing.assert_array_equal(plain.film, want)
    assert plain.stats["shadow_rays"] == st.shadow_rays and plain.stats["closest_rays"] == st.closest_rays
    if n == 2000:       # in the dense soup triangles tie, and the wavefront renderer resolves ties in the 4-wide tree's order
        wf = scene.render(ab.render_opts(8, 3, 3, 2, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 14, wf_block=128, wf_sort=0))
        np.testing.assert_allclose(wf.film, want, rtol=1e-6, atol=1e-7)
    scene.close()


# seven copies of a sheet, each with an emission of its own: below and above the quantised closest hits
@pytest.mark.parametrize("n,nodes", [(20, 384), (130, 98304)])
def test_coincident_sheets(ctx, n, nodes):
    b = scenes.SceneBuilder(61, 47, 0.4, name="sheets")
    m = b.material(_abi.MAT_MATTE, diffuse=(0.5, 0.5, 0.5))
    x = np.linspace(-2, 2, n + 1)
    X, Y = np.meshgrid(x, x)
    V = np.stack([X, Y, -4 + 0.2 * np.sin(3 * X) * np.cos(2 * Y)], -1).reshape(-1, 3)
    I, J = np.meshgrid(np.arange(n), np.arange(n))
    a = (J * (n + 1) + I).ravel()
    f = np.concatenate([np.stack([a, a + 1, a + n + 1], 1), np.stack([a + 1, a + n + 2, a + n + 1], 1)])
    for _ in range(7):
        b.mesh(V, f, m)
    b.square_light(scenes.translate(0, 0.5, -2.0), 0.4, 0.4, (3.0, 3.0, 3.0))
    data = b.build(render=dict(spp=4, max_depth=3, min_depth=3, seed=5))
    data.attr_emission = np.stack([np.arange(1, len(data.attr_material) + 1)] * 3, 1).astype(np.float32)
    scene = ab.Scene(ctx, data)
    assert scene.bvh().info()["num_nodes"] >= nodes
    opts = ab.render_opts(4, 3, 3, 5, fp64_film=1)
    want, st = _pixel_loop(scene, opts)
    assert (want[..., 3] > 0).mean() > 0.5
    got = scene.render(opts)
    np.testing.assert_array_equal(got.film, want)
    assert got.stats["closest_rays"] == st.closest_rays and got.stats["shadow_rays"] == st.shadow_rays
    scene.close()
