"""Ray queries by batch size: a warp per ray, a thread per ray, the resident grid. All give the same records for the
same rays, also where triangles coincide (exact-distance ties) and for rays that are not numbers."""
import numpy as np
import pytest

import aurora_b200 as ab
from aurora_b200 import scenes

pytestmark = pytest.mark.gpu

# a warp per ray up to 96 per SM (14,208 on 148 SMs); the resident grid from 2^18 rays (large trees) or 2^19
SIZES = (1, 31, 1000, 14208, 14209, 40000, 100001, (1 << 18) - 1, 1 << 18, (1 << 19) - 1)


def _mesh(kind):
    if kind == "coincident":            # seven copies of a sheet: every hit is a tie over several leaves
        n = 60
        x = np.linspace(-2, 2, n + 1)
        X, Y = np.meshgrid(x, x)
        v = np.stack([X, Y, 0.2 * np.sin(3 * X)], -1).reshape(-1, 3).astype(np.float32)
        I, J = np.meshgrid(np.arange(n), np.arange(n))
        a = (J * (n + 1) + I).ravel()
        f = np.concatenate([np.stack([a, a + 1, a + n + 1], 1), np.stack([a + 1, a + n + 2, a + n + 1], 1)])
        return v, np.tile(f, (7, 1)).astype(np.uint32)
    if kind == "large":                 # above 2^15 four-wide nodes
        d = scenes.terrain_scene(64, 64, 1, 1, grid=300, spheres=32)
        return d.verts, d.tri_vidx
    v, f = scenes.icosphere(4)
    return v.astype(np.float32), f.astype(np.uint32)


def _rays(n, verts):
    r = np.random.default_rng(4)
    lo, hi = verts.min(0), verts.max(0)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = lo + r.uniform(-0.3, 1.3, (n, 3)) * (hi - lo + 0.5)
    d = r.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.where(r.uniform(size=n) < 0.2, 1.0, 1e30)
    axis = r.integers(0, 3, 200)
    rays[:200, 4:7] = np.eye(3)[axis] * np.where(r.uniform(size=(200, 1)) < 0.5, 1, -1)     # axis parallel
    rays[200:220, 4:7] = 0.0
    rays[220:230, 4] = np.nan
    rays[230:240, 0] = np.inf
    return rays


@pytest.mark.parametrize("kind", ["small", "large", "coincident"])
def test_routes_agree(ctx, kind):
    verts, idx = _mesh(kind)
    bvh = ab.Bvh(ctx, verts, idx, np.arange(len(idx), dtype=np.int32))
    rays = _rays((1 << 19) + 5, verts)
    hits, occ = bvh.trace_closest(rays), bvh.trace_occluded(rays)
    assert 0.05 < (hits["prim"] >= 0).mean() < 0.95
    np.testing.assert_array_equal(occ[240:] != 0, hits["prim"][240:] >= 0)
    for n in SIZES:
        h, o = bvh.trace_closest(rays[:n]), bvh.trace_occluded(rays[:n])
        for k in h.dtype.names:
            np.testing.assert_array_equal(h[k], hits[k][:n], err_msg=f"{k} of {n} rays")
        np.testing.assert_array_equal(o, occ[:n], err_msg=f"{n} rays")
    bvh.close()
