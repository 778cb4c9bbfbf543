"""Kinds of wavefront passes (refilled slots, paths that fit the pool, small launches; one graph or several
graphs of iterations) give the plain renderer's film."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


# 47 x 33 pixels x 5 samples = 7,755 paths: above a pool of 1,024 (refill), below one of 8,192 (small);
# 300 x 199 x 5 = 298,500: below 2^19 slots but above the small launches' 2^18
@pytest.mark.parametrize("w,h,pool", [(47, 33, 1024), (47, 33, 8192), (300, 199, 1 << 19), (1, 1, 1024)])
@pytest.mark.parametrize("depth", [1, 3, 9])       # odd and even queues; more iterations than one graph holds
@pytest.mark.parametrize("lights,offset,env", [(1, 0, False), (3, 0, True), (3, 2, True)])
def test_passes_match_plain(ctx, w, h, pool, depth, lights, offset, env):
    sky = dict(color=(0.3, 0.4, 0.5)) if env else None
    glass = dict(type_=_abi.MAT_GLASS, specular=(0.9, 0.9, 0.9), diffuse=(0.9, 0.8, 0.9), reflectance=0.1, ior=1.4)
    scene = ab.Scene(ctx, scenes.sphere_scene(w, h, env=sky, sphere_mat=glass if env else None))
    films = []
    for mode in (_abi.RENDER_PLAIN, _abi.RENDER_WAVEFRONT):
        wf = dict(wf_pool=pool, wf_block=128, wf_sort=depth % 2) if mode else {}
        o = ab.render_opts(5, depth, depth, 7, mode=mode, sample_offset=offset, light_samples=lights, **wf)
        films.append(scene.render(o))
    assert films[0].stats["paths"] == films[1].stats["paths"]
    np.testing.assert_allclose(films[1].film, films[0].film, rtol=1e-6, atol=1e-7)
    scene.close()
