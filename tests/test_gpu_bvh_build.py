"""The device BVH build at the sizes where its phases change: hits against the brute-force oracle."""
import numpy as np
import pytest

import aurora_b200 as ab

pytestmark = pytest.mark.gpu


def _soup(n, seed, spread=1.0):
    r = np.random.default_rng(seed)
    c = r.uniform(-1, 1, (n, 1, 3)) * spread
    v = (c + r.normal(scale=0.4 / n ** (1 / 3), size=(n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _rays(n, seed):
    r = np.random.default_rng(seed)
    d = r.normal(size=(n, 3))
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = r.uniform(-1.5, 1.5, (n, 3)), d / np.linalg.norm(d, axis=1, keepdims=True), 1e30
    return rays


def _check(ctx, oracle_lib, verts, idx, opts=None, nrays=3000):
    attr = np.arange(len(idx), dtype=np.int32)
    bvh = ab.Bvh(ctx, verts, idx, attr, opts)
    rays = _rays(nrays, 1)
    gpu, occ = bvh.trace_closest(rays), bvh.trace_occluded(rays)
    cpu, ties = oracle_lib.trace_brute(verts, idx, attr, rays)
    ok = ties <= 1
    for k in ("prim", "attr"):
        np.testing.assert_array_equal(gpu[k][ok], cpu[k][ok])
    hit = cpu["prim"] >= 0
    for k in ("t", "u", "v"):
        np.testing.assert_array_equal(gpu[k][ok & hit], cpu[k][ok & hit])
    np.testing.assert_array_equal(gpu["t"][hit], cpu["t"][hit])      # ties share the distance
    np.testing.assert_array_equal(occ.astype(bool), hit)
    info = bvh.info()
    used = verts[idx.ravel()]
    if len(idx) > 1:
        np.testing.assert_array_equal(info["bounds"], np.concatenate([used.min(0), used.max(0)]))
    bvh.close()


# one block does all iterations up to 2048 clusters; a merge tile owns 512 - 2 r of them; sort tiles of
# 1024 pairs
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 33, 480, 1024, 1025, 2047, 2048, 2049, 2400, 30001])
@pytest.mark.parametrize("radius", [1, 16, 32])
def test_sizes(ctx, oracle_lib, n, radius):
    _check(ctx, oracle_lib, *_soup(n, n), ab.bvh_opts(ploc_radius=radius))


# binary trees just below and above 12,288 nodes: the 4-wide collapse in one block, and level by level
@pytest.mark.parametrize("n,block", [(12300, True), (13000, False)])
def test_collapse_forms(ctx, oracle_lib, n, block):
    verts, idx = _soup(n, 11)
    bvh = ab.Bvh(ctx, verts, idx, None, None)
    assert (bvh.info()["num_nodes"] <= 12288) == block
    bvh.close()
    _check(ctx, oracle_lib, verts, idx)


# the larger sort tile (4096 pairs) from 2^18 triangles on
@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 1])
def test_large_sort_tile(ctx, oracle_lib, n):
    _check(ctx, oracle_lib, *_soup(n, 3), nrays=300)


@pytest.mark.parametrize("n", [7, 3000])
@pytest.mark.parametrize("leaf", [1, 31])
def test_leaf_sizes_and_coincident_triangles(ctx, oracle_lib, n, leaf):
    v, f = _soup(n, 5)
    _check(ctx, oracle_lib, v, np.concatenate([f, f[: n // 2], f[: n // 2]]), ab.bvh_opts(max_leaf=leaf))
    flat = v.copy()
    flat[:, 2] = 0.25                                                # no extent along one axis
    _check(ctx, oracle_lib, flat, f, ab.bvh_opts(max_leaf=leaf))


def test_bad_index_in_a_late_triangle(ctx):
    v, f = _soup(5000, 2)
    f[4999, 2] = len(v)
    with pytest.raises(ab.AuroraError, match="vertex index out of range"):
        ab.Bvh(ctx, v, f)
