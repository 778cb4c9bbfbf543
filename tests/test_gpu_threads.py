"""Calls on one context from several host threads: every render and gradient is what it is alone."""
import threading

import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import _abi, scenes

pytestmark = pytest.mark.gpu

ROUNDS = 25


def _together(jobs):
    """Runs every job ROUNDS times in a thread of its own; the first exception is raised here."""
    errors, start = [], threading.Barrier(len(jobs))

    def loop(job):
        try:
            start.wait(60)
            for _ in range(ROUNDS):
                job()
        except BaseException as ex:
            errors.append(ex)
    threads = [threading.Thread(target=loop, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def _render_job(ctx, data, opts, f64=False):
    scene = ab.Scene(ctx, data)
    call = scene.render_f64 if f64 else scene.render
    alone = call(opts)

    def job():
        got = call(opts)
        np.testing.assert_array_equal(got.film, alone.film)
        for k in ("camera_rays", "closest_rays", "shadow_rays", "paths"):
            assert got.stats[k] == alone.stats[k], k
    return job


def test_plain_renders(ctx):
    """Films of different sizes, so that one's samples would not fit the other's buffer; FP32 and FP64."""
    _together([_render_job(ctx, scenes.box_scene(64, 48), ab.render_opts(4, 4, 4, 1)),
               _render_job(ctx, scenes.box_scene(301, 199), ab.render_opts(9, 4, 4, 2)),
               _render_job(ctx, scenes.sphere_scene(123, 77), ab.render_opts(6, 5, 5, 3), f64=True)])


@pytest.mark.parametrize("mode", [_abi.RENDER_WAVEFRONT, _abi.RENDER_PLAIN])
def test_adjoint_beside_plain_renders(ctx, mode):
    data = scenes.texture_scene(48, 40)
    scene = ab.Scene(ctx, data)
    d = np.random.default_rng(1).normal(size=(40, 48, 4)).astype(np.float32)
    opts = ab.render_opts(16, 4, 4, 5, mode=mode)
    gm, gt, st = scene.adjoint(opts, d)

    def job():
        m, t, s = scene.adjoint(opts, d)
        # FP64 sums whose order varies, rounded once; compensated FP32 sums in the megakernel
        np.testing.assert_allclose(m, gm, rtol=1e-5, atol=1e-6 * np.abs(gm).max())
        np.testing.assert_allclose(t, gt, rtol=1e-5, atol=1e-6 * np.abs(gt).max())
        assert s["closest_rays"] == st["closest_rays"] and s["shadow_rays"] == st["shadow_rays"]
    _together([job, _render_job(ctx, scenes.box_scene(257, 200), ab.render_opts(16, 4, 4, 2)),
               _render_job(ctx, scenes.box_scene(31, 20), ab.render_opts(2, 4, 4, 2))])


def test_wavefront_renders(ctx):
    """The same engine for both (one configuration), and another beside it."""
    def opts(spp, pool):
        return ab.render_opts(spp, 5, 5, 7, mode=_abi.RENDER_WAVEFRONT, wf_pool=pool, wf_block=128, wf_sort=1)
    _together([_render_job(ctx, scenes.box_scene(96, 64), opts(4, 1 << 14)),
               _render_job(ctx, scenes.sphere_scene(128, 80), opts(6, 1 << 14)),
               _render_job(ctx, scenes.box_scene(50, 40), opts(2, 1 << 12))])


def test_ray_queries(ctx):
    """Batches of the resident form (2^19 rays), whose cursors are the context's, and small ones."""
    def query_job(level, n, seed):
        verts, idx = scenes.icosphere(level)
        bvh = ab.Bvh(ctx, verts.astype(np.float32), idx.astype(np.uint32))
        r = np.random.default_rng(seed)
        rays = np.zeros((n, 8), np.float32)
        rays[:, :3], rays[:, 4:7], rays[:, 7] = r.uniform(-2, 2, (n, 3)), r.normal(size=(n, 3)), 1e30
        hits, occ = bvh.trace_closest(rays), bvh.trace_occluded(rays)

        def job():
            h = bvh.trace_closest(rays)
            for k in h.dtype.names:
                np.testing.assert_array_equal(h[k], hits[k])
            np.testing.assert_array_equal(bvh.trace_occluded(rays), occ)
        return job
    _together([query_job(4, 1 << 19, 1), query_job(5, (1 << 19) + 99, 2), query_job(4, 5000, 3)])
