"""Attribute tables in device memory, which scene creation does not check: a material index out of range matters
only where its triangle is shaded."""
import ctypes as C

import numpy as np
import pytest
import torch

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _film(ctx, material, mode):
    """A quad before the camera and a triangle behind it, whose attribute has the given material, at depth 1."""
    b = scenes.SceneBuilder(48, 32, 0.5, name="behind")
    m = b.material(_abi.MAT_MATTE, diffuse=(0.6, 0.5, 0.4))
    b.mesh(*scenes.quad((-1, -1, -3), (1, -1, -3), (1, 1, -3.2), (-1, 1, -3.2)), m)
    b.mesh(np.array([[0.0, 0, 9], [1, 0, 9], [0, 1, 9]]), np.array([[0, 1, 2]]), m)
    b.square_light(scenes.translate(0, 0.5, -1.0), 0.4, 0.4, (6.0, 5.0, 4.0))
    data = b.build(render=dict(spp=4, max_depth=1, min_depth=1, seed=3))
    behind = int(data.tri_attr[(data.verts[data.tri_vidx][:, :, 2] > 8).all(1)][0])
    table = np.array(data.attr_material, np.int32)
    table[behind] = material
    table = torch.from_numpy(table).cuda()
    torch.cuda.synchronize()
    desc = data.desc()
    desc.attr_material = table.data_ptr()
    h = C.c_void_p()
    _abi.check(_abi.lib().aur_scene_create(ctx.handle, C.byref(desc), None, C.byref(h)), "aur_scene_create")
    film = np.zeros((32, 48, 4), np.float32)
    opts = ab.render_opts(4, 1, 1, 3, mode=mode, wf_pool=1 << 14 if mode else 0, wf_block=128 if mode else 0,
                          wf_sort=1 if mode else -1)
    st = _abi.RenderStats()
    _abi.check(_abi.lib().aur_render(h, C.byref(opts), film.ctypes.data, C.byref(st)), "aur_render")
    _abi.check(_abi.lib().aur_scene_destroy(h), "aur_scene_destroy")
    return film


@pytest.mark.parametrize("mode", [_abi.RENDER_PLAIN, _abi.RENDER_WAVEFRONT])
@pytest.mark.parametrize("material", [-1, 1 << 20])
def test_a_material_that_is_never_shaded(ctx, material, mode):
    want = _film(ctx, 0, mode)
    assert want[..., 3].max() > 0
    np.testing.assert_array_equal(_film(ctx, material, mode), want)
