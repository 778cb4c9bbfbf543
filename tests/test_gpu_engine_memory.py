"""What the wavefront renderer holds between calls: one pool for scenes of every tree size, and nothing that keeps
a later call from its memory."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once(ctx):
    """The error of a pool (15 GiB) that does not fit is not found again by the next call's launch checks."""
    import torch
    scene = ab.Scene(ctx, scenes.box_scene(64, 48))
    o = ab.render_opts(2, 3, 3, 3, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 14, wf_block=128, wf_sort=1)
    film = scene.render(o).film
    held = torch.empty(torch.cuda.mem_get_info()[0] - (8 << 30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(ab.AuroraError, match="MemoryAllocation"):
            scene.render(ab.render_opts(2, 3, 3, 3, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 26, wf_block=128, wf_sort=1))
        np.testing.assert_array_equal(scene.render(o).film, film)
    finally:
        del held
        torch.cuda.empty_cache()
    scene.close()
