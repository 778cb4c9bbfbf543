"""The wavefront adjoint's vertex records and FP64 sums against the megakernel adjoint."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _many_materials(nmat):
    """A row of quads, one material each (Lambert, Cook-Torrance and Kelemen in turn), under a light."""
    b = scenes.SceneBuilder(64, 40, 0.6, name="row")
    for k in range(nmat):
        kind = (_abi.MAT_MATTE, _abi.MAT_COOKTORRANCE, _abi.MAT_KELEMEN)[k % 3]
        m = b.material(kind, diffuse=(0.2 + 0.01 * k, 0.5, 0.7), specular=(0.8, 0.7, 0.9), roughness=0.2 + 0.01 * k,
                       reflectance=0.3)
        x = -1.2 + 2.4 * k / nmat
        v, f = scenes.quad((x, -1, -3), (x + 2.4 / nmat, -1, -3), (x + 2.4 / nmat, 1, -3.5), (x, 1, -3.5))
        b.mesh(v, f, m)
    b.square_light(scenes.translate(0, 0.5, -1.0), 0.4, 0.4, (6.0, 5.0, 4.0))
    return b.build(render=dict(spp=8, max_depth=4, min_depth=4, seed=3))


# 12 materials: the largest count with a column of sums per thread; 13 and 63 (+ the light's) share columns
@pytest.mark.parametrize("nmat", [1, 11, 12, 63])
@pytest.mark.parametrize("lights", [1, 3])
def test_material_sums(ctx, nmat, lights):
    data = _many_materials(nmat)
    scene = ab.Scene(ctx, data)
    d = np.random.default_rng(nmat).normal(size=(40, 64, 4)).astype(np.float32)
    g = [scene.adjoint(ab.render_opts(8, 4, 4, 3, mode=m, light_samples=lights), d)[0]
         for m in (_abi.RENDER_PLAIN, _abi.RENDER_WAVEFRONT)]
    assert np.abs(g[0]).max() > 0
    # every vertex's factors agree to a few ulp, their sums to that times the sum of magnitudes; the
    # cancellation in "radiance after the vertex" adds some 1e-6 of a path's radiance
    np.testing.assert_allclose(g[1], g[0], rtol=2e-4, atol=2e-5 * np.abs(g[0]).max())
    scene.close()


@pytest.mark.parametrize("scale", [0.0, 0.5])      # uv lookup; triplanar (records with three texels)
def test_texel_sums(ctx, scale):
    b = scenes.SceneBuilder(48, 48, 0.6, name="texels")
    t = b.texture(np.random.default_rng(1).uniform(0.2, 0.8, (5, 7, 3)), triplanar_scale=scale)
    m = b.material(_abi.MAT_KELEMEN, diffuse=(0.5, 0.5, 0.5), specular=(1, 1, 1), roughness=0.3, reflectance=0.4,
                   diffuse_tex=t)
    v, f = scenes.icosphere(2)
    b.mesh(v, f, m, normals=v, uvs=v[:, :2] * 0.5 + 0.5, object_to_world=scenes.translate(0, 0, -3))
    b.square_light(scenes.translate(0, 0.5, -1.0), 0.4, 0.4, (6.0, 5.0, 4.0))
    scene = ab.Scene(ctx, b.build(render=dict(spp=8, max_depth=3, min_depth=3, seed=3)))
    d = np.random.default_rng(2).normal(size=(48, 48, 4)).astype(np.float32)
    g = [scene.adjoint(ab.render_opts(8, 3, 3, 3, mode=m), d)[:2] for m in (_abi.RENDER_PLAIN, _abi.RENDER_WAVEFRONT)]
    for k in (0, 1):
        assert np.abs(g[0][k]).max() > 0
        np.testing.assert_allclose(g[1][k], g[0][k], rtol=2e-4, atol=2e-5 * np.abs(g[0][k]).max())
    scene.close()
