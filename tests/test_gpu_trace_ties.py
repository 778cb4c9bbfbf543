"""Ray queries where triangles coincide, on a tree with quantised nodes: the resident form notices exact-distance
ties and traces those rays again, so that records are those of the thread form; and the forms of a very small tree."""
import ctypes as C

import numpy as np
import pytest
import torch

import aurora_b200 as ab
from aurora_b200 import _abi, scenes
from aurora_b200.core import HIT_DTYPE, ISECT_DTYPE

pytestmark = pytest.mark.gpu


def _sheets(n, copies):
    x = np.linspace(-2, 2, n + 1)
    X, Y = np.meshgrid(x, x)
    v = np.stack([X, Y, 0.2 * np.sin(3 * X)], -1).reshape(-1, 3).astype(np.float32)
    I, J = np.meshgrid(np.arange(n), np.arange(n))
    a = (J * (n + 1) + I).ravel()
    f = np.concatenate([np.stack([a, a + 1, a + n + 1], 1), np.stack([a + 1, a + n + 2, a + n + 1], 1)])
    return v, np.tile(f, (copies, 1)).astype(np.uint32)


def _rays(n, verts, seed):
    r = np.random.default_rng(seed)
    lo, hi = verts.min(0), verts.max(0)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = lo + r.uniform(-0.3, 1.3, (n, 3)) * (hi - lo + 0.5)
    d = r.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.where(r.uniform(size=n) < 0.2, 1.0, 1e30)
    return rays


def _closest(bvh, rays):
    d = torch.from_numpy(rays).cuda()
    out = torch.empty(len(rays) * HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    _abi.check(_abi.lib().aur_trace_closest(bvh.handle, C.c_void_p(d.data_ptr()), C.c_void_p(out.data_ptr()), len(rays)), "closest")
    return out.cpu().numpy().view(HIT_DTYPE)


def _intersect(bvh, rays):
    d = torch.from_numpy(rays.copy()).cuda()
    out = torch.empty(len(rays) * ISECT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    _abi.check(_abi.lib().aur_bvh_intersect(bvh.handle, C.c_void_p(d.data_ptr()), C.c_void_p(out.data_ptr()), len(rays)), "isect")
    return out.cpu().numpy().view(ISECT_DTYPE), d.cpu().numpy()


def _same(a, b, msg):
    for k in a.dtype.names:
        np.testing.assert_array_equal(a[k], b[k], err_msg=f"{k}: {msg}")


def _shaded(ctx, verts, idx):
    bvh = ab.Bvh(ctx, verts, idx, np.arange(len(idx), dtype=np.int32))
    r = np.random.default_rng(9)
    bvh.set_shading(r.normal(size=(len(idx), 9)), r.uniform(size=(len(idx), 6)))
    return bvh


# the smallest and larger batches of the resident form, against batches of the form with a thread per ray
@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 77, 600001])
def test_coincident_triangles(ctx, n):
    verts, idx = _sheets(130, 7)
    bvh = _shaded(ctx, verts, idx)
    assert bvh.info()["num_nodes"] >= 3 * 32768        # a 4-wide node holds at most three binary ones: 2^15 or more
    rays = _rays(n, verts, 4)
    hits, (isect, moved) = _closest(bvh, rays), _intersect(bvh, rays)
    hit = hits["prim"] >= 0
    assert 0.05 < hit.mean() < 0.95
    part = (1 << 18) - 1
    for k in range(0, n, part):
        _same(hits[k:k + part], _closest(bvh, rays[k:k + part]), f"rays from {k}")
        want, shrunk = _intersect(bvh, rays[k:k + part])
        _same(isect[k:k + part], want, f"rays from {k}")
        np.testing.assert_array_equal(moved[k:k + part], shrunk)
    for key in ("t", "u", "v", "prim", "attr"):
        np.testing.assert_array_equal(isect[key], hits[key])
    np.testing.assert_array_equal(moved[:, 7], np.where(hit, hits["t"], rays[:, 7]))
    np.testing.assert_array_equal(bvh.trace_occluded(rays) != 0, hit)
    again = _closest(bvh, rays)                        # the cursor is zero again
    _same(hits, again, "second call")
    bvh.close()


# below 128 four-wide nodes: a warp per ray up to 8 (occlusion: 48) rays per SM, then the thread form throughout;
# and the full record by batch size on a tree of 5,120 triangles
@pytest.mark.parametrize("kind", ["few triangles", "small"])
def test_records_by_batch_size(ctx, kind):
    if kind == "small":
        verts, idx = scenes.icosphere(4)
        verts, idx = verts.astype(np.float32), idx.astype(np.uint32)
    else:
        d = scenes.box_scene(16, 16)
        verts, idx = d.verts, d.tri_vidx
    bvh = _shaded(ctx, verts, idx)
    rays = _rays((1 << 19) + 5, verts, 6)
    isect, moved = _intersect(bvh, rays)
    hits, occ = _closest(bvh, rays), bvh.trace_occluded(rays)
    assert 0.05 < (hits["prim"] >= 0).mean()
    np.testing.assert_array_equal(occ != 0, hits["prim"] >= 0)
    for n in (1, 33, 1184, 1185, 7104, 7105, 14208, 14209, 100001, (1 << 19) - 1):
        _same(hits[:n], _closest(bvh, rays[:n]), f"{n} rays")
        got, shrunk = _intersect(bvh, rays[:n])
        _same(isect[:n], got, f"{n} rays")
        np.testing.assert_array_equal(moved[:n], shrunk)
        np.testing.assert_array_equal(occ[:n], bvh.trace_occluded(rays[:n]))
    bvh.close()
