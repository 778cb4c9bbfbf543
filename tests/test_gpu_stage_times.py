"""The wavefront renderer's stage times are the device's: what the host takes between the launches of a pass is no
stage's."""
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def test_host_reads_between_graphs_are_not_stage_time(ctx):
    """A pool of 1,024 slots: well over a hundred graphs, after each of which the host reads the counters. A read and
    the next graph's launch take 10 us and more; 3 is well below what they can."""
    scene = ab.Scene(ctx, scenes.box_scene(64, 64))
    opts = ab.render_opts(64, 5, 5, 3, mode=_abi.RENDER_WAVEFRONT, wf_pool=1024, wf_block=64, wf_sort=1)
    scene.render(opts)
    st = scene.render(opts).stats
    graphs = (st["launches"] - 2) // (8 * 6 + 1)     # 8 iterations of 6 launches; last regen and resolve
    assert graphs > 100
    stages = sum(st["stage_ms"].values())
    assert 0 < stages < st["kernel_ms"] - 3e-3 * graphs
    scene.close()


def test_one_graph_is_all_stage_time(ctx):
    """A pass of one graph with nothing between its launches: the stages, the last regen among them, are all of it but
    the uploads before and the resolve after."""
    scene = ab.Scene(ctx, scenes.box_scene(512, 512))
    opts = ab.render_opts(8, 5, 5, 3, mode=_abi.RENDER_WAVEFRONT, wf_pool=1 << 21, wf_block=128, wf_sort=1)
    scene.render(opts)
    st = scene.render(opts).stats
    stages = sum(st["stage_ms"].values())
    assert 0.8 * st["kernel_ms"] < stages < st["kernel_ms"]
    assert st["stage_ms"]["regen"] > 0 and st["stage_ms"]["shadow"] > 0
    scene.close()
