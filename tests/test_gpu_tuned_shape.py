"""What the wavefront autotuner keeps its choice by: the number of paths, light samples included."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def test_light_samples_are_part_of_the_shape():
    """64 light samples: 4.3 M paths, for which pools of 2^20 to 2^23 slots are tried. Without them 131,072, for which only
    2^20 is (a larger pool would stay mostly empty); the choice made for the many must not be taken."""
    ctx = ab.Context(0)
    scene = ab.Scene(ctx, scenes.box_scene(256, 256))
    many = scene.render(ab.render_opts(2, 4, 4, 3, mode=_abi.RENDER_WAVEFRONT, light_samples=64))
    few = scene.render(ab.render_opts(2, 4, 4, 3, mode=_abi.RENDER_WAVEFRONT))
    assert many.stats["wf_config"]["pool"] >= 1 << 20
    assert few.stats["wf_config"]["pool"] == 1 << 20
    again = scene.render(ab.render_opts(2, 4, 4, 3, mode=_abi.RENDER_WAVEFRONT, light_samples=64))
    assert again.stats["wf_config"] == many.stats["wf_config"]
    np.testing.assert_array_equal(again.film, many.film)
    ctx.close()
