"""The quantised 4-wide nodes against the full-precision tree: same hits, exact ties included."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _u01(seed, counter):
    """The counter-based generator of the renderers (SplitMix64)."""
    def mix(z):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
        return z ^ (z >> np.uint64(31))
    golden = np.uint64(0x9e3779b97f4a7c15)
    with np.errstate(over="ignore"):
        key = mix(np.uint64(seed) * golden + np.uint64(0x632be59bd9b4e019))
        return ((mix(key + counter * golden) >> np.uint64(40)).astype(np.float32) * np.float32(2.0 ** -24))


def _grid_scene(n, copies, w, h):
    """A bumpy sheet of 2 n^2 triangles facing the camera, laid down `copies` times: every copy
    is its own object with its own emission, so the film tells which copy a ray hit."""
    b = scenes.SceneBuilder(w, h, 0.4, name="sheets")
    m = b.material(_abi.MAT_MATTE, diffuse=(0.5, 0.5, 0.5))
    x = np.linspace(-2, 2, n + 1)
    X, Y = np.meshgrid(x, x)
    V = np.stack([X, Y, -4 + 0.2 * np.sin(3 * X) * np.cos(2 * Y)], -1).reshape(-1, 3)
    i = np.arange(n)
    I, J = np.meshgrid(i, i)
    a = (J * (n + 1) + I).ravel()
    f = np.concatenate([np.stack([a, a + 1, a + n + 1], 1), np.stack([a + 1, a + n + 2, a + n + 1], 1)])
    for _ in range(copies):
        b.mesh(V, f, m)
    d = b.build(render=dict(spp=1, max_depth=1, min_depth=1, seed=5))
    d.attr_emission = np.stack([np.arange(1, copies + 1)] * 3, 1).astype(np.float32)
    return d


# 2 copies of 2 * 300^2 triangles: above the node count from which closest hits use quantised nodes;
# 2 * 20^2: below it (full-precision closest hits); seven copies do not fit one leaf, so that the
# tied triangles lie in several
@pytest.mark.parametrize("n,copies", [(20, 2), (300, 1), (300, 2), (160, 7)])
def test_wavefront_hits_match_the_trace_queries(ctx, n, copies):
    w, h = 193, 101
    data = _grid_scene(n, copies, w, h)
    scene = ab.Scene(ctx, data)
    film = scene.render(ab.render_opts(1, 1, 1, 5, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 14, wf_block=128,
                                       wf_sort=1)).film
    pix = np.arange(w * h, dtype=np.uint64)
    j = [_u01(5, (pix << np.uint64(32)) | np.uint64(k)) for k in (0, 1)]
    rec = np.stack([np.full(w * h, data.fov), np.full(w * h, w), np.full(w * h, h), pix % w, pix // w, *j], 1)
    rays = np.zeros((w * h, 8), np.float32)
    rays[:, 4:7] = ctx.probe(4, rec.astype(np.float32))
    rays[:, 3], rays[:, 7] = 0.1, 1e7
    hits = scene.bvh().trace_closest(rays)
    want = np.where(hits["attr"] >= 0, hits["attr"] + 1, 0).astype(np.float32)
    assert (hits["attr"] >= 0).mean() > 0.5
    np.testing.assert_array_equal(film[..., 0].ravel(), want)
    scene.close()


@pytest.mark.parametrize("scale,dist", [(1.0, 3.0), (1e-3, 0.5), (1e4, 3e5)])
def test_next_event_rays_match_the_binary_tree(ctx, scale, dist):
    """Next-event rays on quantised nodes over small, flat and far-off geometry: the plain renderer (binary
    tree, full-precision boxes) gives the same film. The camera's near limit is 0.1."""
    r = np.random.default_rng(3)
    b = scenes.SceneBuilder(64, 48, scale / dist, name="soup")
    m = b.material(_abi.MAT_MATTE, diffuse=(0.6, 0.5, 0.4))
    c = r.uniform(-1, 1, (400, 1, 3)) * (1.0, 1.0, 0.3)
    v = (c + r.uniform(-0.2, 0.2, (400, 3, 3)) * (1.0, 1.0, 0.01)).reshape(-1, 3)
    v = np.concatenate([v, [[-2, -2, -0.5], [2, -2, -0.5], [2, 2, -0.5], [-2, 2, -0.5]]])
    f = np.concatenate([np.arange(1200).reshape(-1, 3), [[1200, 1201, 1202], [1200, 1202, 1203]]])
    v = v * scale + np.array([0.0, 0.0, -dist])
    b.mesh(v, f, m)
    b.square_light(scenes.translate(0, 0.5 * scale, v[:, 2].max() + scale) @ scenes.scale(1, 1, 1), 0.3 * scale,
                   0.3 * scale, (5.0, 5.0, 5.0))
    data = b.build(render=dict(spp=8, max_depth=3, min_depth=3, seed=2))
    scene = ab.Scene(ctx, data)
    films = [scene.render(ab.render_opts(8, 3, 3, 2, mode=mode, wf_pool=1 << 14 if mode else 0,
                                         wf_block=128 if mode else 0, wf_sort=0 if mode else -1)).film
             for mode in (_abi.RENDER_PLAIN, _abi.RENDER_WAVEFRONT)]
    assert films[0][..., 3].max() > 0
    np.testing.assert_allclose(films[1], films[0], rtol=1e-6, atol=1e-7)
    scene.close()
