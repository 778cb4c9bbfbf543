"""The smallest BVH: one triangle, its bounds as any other mesh's."""
import numpy as np
import pytest

import aurora_b200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("verts", [[[1, 2, 3], [4, 2, 3], [1, 5, 7]], [[-3, -2, -1], [-5, -2, -1.5], [-3, -8, -1]],
                                   [[0.5, 0, 0], [0.5, 1, 0], [0.5, 0, 1]]])
def test_bounds_and_hits(ctx, verts):
    v = np.array(verts, np.float32)
    bvh = ab.Bvh(ctx, np.concatenate([np.full((2, 3), 99, np.float32), v]), np.array([[2, 3, 4]], np.uint32))   # 99s: unused
    info = bvh.info()
    np.testing.assert_array_equal(info["bounds"], np.concatenate([v.min(0), v.max(0)]))
    assert info["num_nodes"] == 1 and info["depth"] == 1
    n = np.cross(v[1] - v[0], v[2] - v[0])
    n /= np.linalg.norm(n)
    c = v.mean(0)
    rays = np.zeros((4, 8), np.float32)
    rays[:, :3] = [c + 2 * n, c - 2 * n, c + 2 * n + 20 * (v[1] - v[0]), c + 2 * n]
    rays[:, 4:7] = [-n, n, -n, n]
    rays[:, 7] = 1e30
    hits = bvh.trace_closest(rays)
    np.testing.assert_array_equal(hits["prim"], [0, 0, -1, -1])
    np.testing.assert_allclose(hits["t"][:2], 2, rtol=1e-5)
    np.testing.assert_array_equal(bvh.trace_occluded(rays), [1, 1, 0, 0])
    bvh.close()
