"""What the wavefront renderer holds between calls: one pool for scenes of every tree size, and nothing that keeps
a later call from its memory."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    """Takes device memory until about `leave` bytes are free."""
    import torch
    held = []
    while _free() > leave + 64 * MIB:
        held.append(torch.empty(_free() - leave, dtype=torch.uint8, device="cuda"))
    return held


def _opts(pool, spp=4):
    return ab.render_opts(spp, 4, 4, 3, mode=_abi.RENDER_WAVEFRONT, wf_pool=pool, wf_block=128 if pool else 0,
                          wf_sort=1 if pool else -1)


def test_trees_share_a_pool():
    """Below 128 four-wide nodes, above, and above 32,768: the trees differ, the pool (0.9 GiB) is one."""
    ctx = ab.Context(0)
    box, sphere, land = (ab.Scene(ctx, d) for d in (scenes.box_scene(64, 48), scenes.sphere_scene(64, 48),
                                                    scenes.terrain_scene(64, 48, grid=300, spheres=8)))
    films, free = [], []
    for scene in (box, sphere, land):
        films.append([scene.render(_opts(1 << 22)).film, scene.render(_opts(1 << 12)).film])
        free.append(_free())
    for a, b in films:
        np.testing.assert_array_equal(a, b)
    assert free[0] - min(free) < 400 * MIB
    for scene, (a, _) in zip((box, sphere, land), films):      # back over the same pool and graphs
        np.testing.assert_array_equal(scene.render(_opts(1 << 22)).film, a)
    ctx.close()


def test_idle_pools_make_room():
    """A pool (0.9 GiB) that does not fit beside an idle one (1.8 GiB), and a tuned pool that fits no more."""
    import torch
    ctx = ab.Context(0)
    scene = ab.Scene(ctx, scenes.box_scene(256, 256))
    tuned = scene.render(_opts(0, 64))
    film = scene.render(_opts(1 << 22)).film
    scene.render(_opts(1 << 23))
    held = []
    try:
        held += _fill(300 * MIB)
        np.testing.assert_array_equal(scene.render(_opts(1 << 23)).film, film)     # the pool that is there
        np.testing.assert_array_equal(scene.render(_opts(1 << 21)).film, film)     # does not fit beside it
        held += _fill(150 * MIB)
        got = scene.render(_opts(0, 64))               # 2^20 slots or more, 236 MB, were chosen
        np.testing.assert_array_equal(got.film, tuned.film)
        with pytest.raises(ab.AuroraError):            # the caller's own size is not changed
            scene.render(_opts(1 << 25))
        np.testing.assert_array_equal(scene.render(_opts(1 << 14)).film, film)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    ctx.close()


def test_a_failed_allocation_is_reported_once():
    """The error of a pool (15 GiB) that does not fit is not found again by the next call's launch checks."""
    import torch
    ab.Context(0).close()                 # gives back what other contexts left in the stream-ordered pool
    ctx = ab.Context(0)
    scene = ab.Scene(ctx, scenes.box_scene(64, 48))
    film = scene.render(_opts(1 << 14, 2)).film
    held = _fill(4 << 30)
    try:
        with pytest.raises(ab.AuroraError, match="MemoryAllocation"):
            scene.render(_opts(1 << 26, 2))
        np.testing.assert_array_equal(scene.render(_opts(1 << 14, 2)).film, film)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    ctx.close()
