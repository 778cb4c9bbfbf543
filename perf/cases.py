"""Performance cases of the Aurora path-tracing core, through its public entry points.

Four kinds of work, each over the range of sizes that users have:
  trace    batched ray queries against a resident BVH (closest hit, occlusion, the full
           intersection record), from a few hundred rays to some millions
  build    a BVH over new geometry, then a batch of rays through it (a frame of an animation)
  render   frames with each renderer: previews, the repository's scenes at their configured
           sizes, odd film sizes, light samples, environment light, texture shaders, batches
  adjoint  a differentiable render and its backward pass (one step of an optimisation)
Geometry, textures, poses, rays and random-number seeds come from the seed; sizes and
options from the case.
"""
import math

import numpy as np
import torch

import aurora_b200 as ab
from aurora_b200 import _abi, pyaurora, scenes

_ctx = None


def _context():
    """One context for the whole program, as an application keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = ab.Context(0)
    return _ctx


# ---------------------------------------------------------------------------- the cases
def listed():
    return [
        # a picking or audio-probe query: a few rays, where the latency of the call counts
        dict(name="trace_few", kind="trace", query="closest", mesh="bumpy", level=5, n=1000, host=False),
        # the repository's hit-ID workload: 2^20 incoherent rays around a 20k-triangle sphere
        dict(name="trace_closest", kind="trace", query="closest", mesh="bumpy", level=5, n=1 << 20, host=False),
        # next-event visibility of a baker: surface points of a landscape towards its lights
        dict(name="trace_occluded", kind="trace", query="occluded", mesh="terrain", grid=513, spheres=64, n=1500001,
             host=False),
        # the accelerator adapter's batched intersect from host arrays (full record, maxt shrunk)
        dict(name="intersect_host", kind="trace", query="intersect", mesh="bumpy", level=5, n=99991, host=True),
        # a small deforming mesh rebuilt every frame from host arrays and queried
        dict(name="build_20k", kind="build", mesh="bumpy", level=5, n=16384, host=True),
        # a large landscape rebuilt from device arrays (the benchmark's terrain) and queried
        dict(name="build_3m", kind="build", mesh="terrain", grid=1024, spheres=256, n=262144, host=False),
        # a material preview thumbnail: the smallest frame, redrawn at every edit
        dict(name="preview_box", kind="render", scene="box", mode="wavefront", w=128, h=128, spp=4, depth=5, lights=1,
             env=False),
        # the sphere workload of the repository's configurations: glossy and Lambert, 512 x 512 x 64
        dict(name="frame_sphere", kind="render", scene="sphere", mode="wavefront", w=512, h=512, spp=64, depth=6,
             lights=1, env=False),
        # the headline frame: the 3.4 M triangle terrain at 1080p, 64 samples, depth 8, roulette
        dict(name="frame_terrain", kind="render", scene="terrain", mode="wavefront", w=1920, h=1080, spp=64, depth=8,
             lights=1, env=False, grid=1024, spheres=256),
        # a reference image with the FP64 film at an odd size: texture shaders and normal maps
        dict(name="reference_f64", kind="render", scene="shaders", mode="f64", w=201, h=149, spp=64, depth=6, lights=1,
             env=False),
        # a service rendering sixteen scenes of mixed sizes in one launch
        dict(name="batch_16", kind="batch", count=16),
        # one step of the differentiable workload: 256 x 256, 256 samples, texels and materials
        dict(name="adjoint_texture", kind="adjoint", mode="wavefront", w=256, h=256, spp=256, depth=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "build", "render", "render", "render", "batch", "adjoint"])
    if kind == "trace":
        query = rng.choice(["closest", "occluded", "intersect"])
        host = query == "intersect" or rng.random() < 0.3
        n = _log(rng, 300, 300000 if host else 2000000)
        if rng.random() < 0.5:
            return dict(kind=kind, query=query, mesh="bumpy", level=rng.choice([3, 4, 5]), n=n, host=host)
        return dict(kind=kind, query=query, mesh="terrain", grid=_log(rng, 100, 700), spheres=rng.randint(8, 64), n=n,
                    host=host)
    if kind == "build":
        if rng.random() < 0.5:
            return dict(kind=kind, mesh="bumpy", level=rng.choice([2, 3, 4, 5]), n=_log(rng, 1000, 65536),
                        host=rng.random() < 0.5)
        return dict(kind=kind, mesh="terrain", grid=_log(rng, 50, 900), spheres=rng.randint(1, 200),
                    n=_log(rng, 1000, 262144), host=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 24))
    if kind == "adjoint":
        return dict(kind=kind, mode=rng.choice(["wavefront", "wavefront", "plain"]), w=rng.randint(48, 256),
                    h=rng.randint(48, 256), spp=_log(rng, 4, 128), depth=rng.randint(3, 8))
    mode = rng.choice(["wavefront", "wavefront", "wavefront", "plain", "f64"])
    scene = rng.choice(["box", "sphere", "shaders", "terrain"])
    slow = mode != "wavefront"
    c = dict(kind=kind, scene=scene, mode=mode, w=_log(rng, 60, 640 if slow else 1600),
             h=_log(rng, 60, 480 if slow else 1000), spp=_log(rng, 1, 24 if slow else 64), depth=rng.randint(2, 8),
             lights=rng.choice([1, 1, 1, 2, 4]), env=scene == "sphere" and rng.random() < 0.5)
    c["spp"] = max(1, c["spp"] // c["lights"])
    if scene == "terrain":
        c.update(grid=_log(rng, 200, 900), spheres=rng.randint(16, 200))
    return c


# ---------------------------------------------------------------------------- inputs
def _bumpy(level, seed):
    """A displaced icosphere over a ground quad: (verts, faces, attrs, corner normals, corner uvs)."""
    r = np.random.default_rng(seed)
    v, f = scenes.icosphere(level)
    k = r.normal(size=(6, 3)) * 3.0
    ph = r.uniform(0, 6.28, 6)
    rad = 1.0 + 0.05 * np.sin(v @ k.T + ph).sum(1)
    gv = np.array([[-5, -1.4, 5], [5, -1.4, 5], [5, -1.4, -5], [-5, -1.4, -5]])
    verts = np.concatenate([gv, v * rad[:, None]]).astype(np.float32)
    faces = np.concatenate([[[0, 1, 2], [0, 2, 3]], f + 4]).astype(np.uint32)
    attr = np.concatenate([[0, 0], np.ones(len(f))]).astype(np.int32)
    nv = np.concatenate([np.tile([0.0, 1.0, 0.0], (4, 1)), v]).astype(np.float32)
    cn = np.ascontiguousarray(nv[faces].reshape(-1, 9))
    uv = np.concatenate([[[0, 0], [1, 0], [1, 1], [0, 1]], v[:, :2] * 0.5 + 0.5]).astype(np.float32)
    return verts, faces, attr, cn, np.ascontiguousarray(uv[faces].reshape(-1, 6))


def _mesh(case, seed):
    if case["mesh"] == "bumpy":
        return _bumpy(case["level"], seed)
    d = scenes.terrain_scene(64, 64, 1, 1, grid=case["grid"], spheres=case["spheres"], seed=seed, sphere_seed=seed + 1)
    return d.verts, d.tri_vidx, d.tri_attr, d.corner_normals, d.corner_uvs


def _rays(case, mesh, seed):
    """Around the bumpy sphere: incoherent rays from all over its neighbourhood. On a landscape:
    from points of the surface towards four lights above it. (n, 8) float32 aur_ray records."""
    r = np.random.default_rng(seed + 17)
    n = case["n"]
    verts, faces, _, cn, _ = mesh
    out = np.empty((n, 8), np.float32)
    if case["mesh"] == "bumpy":
        d = r.standard_normal((n, 3), np.float32)
        out[:, 0:3] = r.random((n, 3), np.float32) * 6 - 3
        out[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
        out[:, 3], out[:, 7] = 0.0, 100.0
        return out
    tri = r.integers(0, len(faces), n)
    b = r.dirichlet((1, 1, 1), n).astype(np.float32)
    p = (verts[faces[tri]] * b[:, :, None]).sum(1) + 1e-3 * cn[tri, :3]
    lo, hi = verts.min(0), verts.max(0)
    corners = np.array([[0.3, 1.0, 0.3], [0.7, 1.0, 0.3], [0.3, 1.0, 0.7], [0.7, 1.0, 0.7]], np.float32)
    lights = lo + corners * (hi - lo) + np.float32([0, 1, 0])
    d = lights[r.integers(0, 4, n)] + r.uniform(-0.75, 0.75, (n, 3)).astype(np.float32) - p
    dist = np.linalg.norm(d, axis=1)
    out[:, 0:3], out[:, 3], out[:, 4:7], out[:, 7] = p, 5e-4, d / dist[:, None], dist
    return out


def _scene_data(case, seed):
    w, h, spp, depth = case["w"], case["h"], case["spp"], case["depth"]
    if case["scene"] == "box":
        return scenes.box_scene(w, h, spp, depth, seed=seed, rng_seed=seed)
    if case["scene"] == "sphere":
        env = dict(color=(0.4, 0.5, 0.7), texture=np.random.default_rng(seed).uniform(0, 2, (32, 64, 3))) \
            if case["env"] else None
        return scenes.sphere_scene(w, h, spp, depth, seed=seed, env=env)
    if case["scene"] == "shaders":
        return scenes.shader_scene(w, h, spp, depth, seed=seed, tex_seed=seed)
    return scenes.terrain_scene(w, h, spp, depth, grid=case["grid"], spheres=case["spheres"], seed=seed,
                                sphere_seed=seed + 1, render_seed=seed)


_BATCH = [(128, 64, 5), (192, 16, 8), (512, 4, 3), (256, 16, 5), (384, 4, 8), (128, 4, 3), (256, 64, 3), (512, 16, 5)]


def _batch_shape(i):
    """(resolution, spp, depth) of the i-th scene: the mixture of the repository's 64-scene batch."""
    return _BATCH[i % len(_BATCH)]


_MODES = {"plain": _abi.RENDER_PLAIN, "wavefront": _abi.RENDER_WAVEFRONT, "f64": _abi.RENDER_PLAIN}


def _film(w, h):
    return torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")


def prepare(case, seed):
    ctx = _context()
    s = dict(case=case)
    if case["kind"] in ("trace", "build"):
        mesh = _mesh(case, seed)
        rays = _rays(case, mesh, seed)
        if case["host"]:
            s["rays"], s["mesh"] = rays, mesh
        else:
            s["rays"] = torch.from_numpy(rays).cuda()
            s["mesh"] = [torch.from_numpy(np.ascontiguousarray(a).view(np.int32) if a.dtype == np.uint32 else a).cuda()
                         for a in mesh[:3]]
            s["hits"] = torch.zeros((case["n"], 5), dtype=torch.float32, device="cuda")
            s["occ"] = torch.zeros(case["n"], dtype=torch.uint8, device="cuda")
        if case["kind"] == "trace":
            s["bvh"] = ab.Bvh(ctx, mesh[0], mesh[1], mesh[2])
            if case["query"] == "intersect":
                s["bvh"].set_shading(mesh[3], mesh[4])
    elif case["kind"] == "batch":
        shapes = [_batch_shape(i) for i in range(case["count"])]
        data = [scenes.box_scene(r, r, spp, d, seed=seed + i, rng_seed=seed + i)
                for i, (r, spp, d) in enumerate(shapes)]
        s["scenes"] = [ab.Scene(ctx, d) for d in data]
        s["opts"] = [ab.render_opts(spp, d, d, seed + i, mode=_abi.RENDER_WAVEFRONT)
                     for i, (r, spp, d) in enumerate(shapes)]
        s["films"] = [_film(r, r) for r, _, _ in shapes]
    elif case["kind"] == "adjoint":
        tex = np.random.default_rng(seed).uniform(0.2, 0.8, (64, 64, 3)).astype(np.float32)
        data = scenes.sphere_scene(case["w"], case["h"], case["spp"], case["depth"], seed=seed, ground_texture=tex)
        s["scene"] = ab.Scene(ctx, data)
        s["params"] = torch.tensor(data.material_params(), device="cuda")
        s["texels"] = torch.tensor(data.texels(), device="cuda")
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["target"] = torch.rand((case["h"], case["w"], 3), device="cuda", generator=g)
        s["options"] = dict(spp=case["spp"], max_depth=case["depth"], seed=seed & 0xffff, mode=case["mode"])
    else:
        data = _scene_data(case, seed)
        s["scene"] = ab.Scene(ctx, data)
        s["opts"] = ab.render_opts(case["spp"], case["depth"], data.render["min_depth"], seed & 0xffff,
                                   mode=_MODES[case["mode"]], light_samples=case["lights"])
        if case["mode"] != "f64":
            s["film"] = _film(case["w"], case["h"])
    return s


# ---------------------------------------------------------------------------- one pass
def _closest_on_device(handle, rays, hits):
    # device arrays go through the C entry points
    _abi.check(ab.lib().aur_trace_closest(handle, rays.data_ptr(), hits.data_ptr(), rays.shape[0]),
               "aur_trace_closest")
    return dict(tuv=hits[:, :3], ids=hits.view(torch.int32)[:, 3:])


def _closest_on_host(bvh, rays):
    h = bvh.trace_closest(rays)
    return dict(tuv=np.stack([h["t"], h["u"], h["v"]], 1), ids=np.stack([h["prim"], h["attr"]], 1))


def _run_build(s):
    rays, mesh = s["rays"], s["mesh"]
    if s["case"]["host"]:
        bvh = ab.Bvh(_context(), mesh[0], mesh[1], mesh[2])
        out = _closest_on_host(bvh, rays)
        out["bounds"] = np.array(bvh.info()["bounds"], np.float32)
        bvh.close()
        return out
    h = _abi.C.c_void_p()
    _abi.check(ab.lib().aur_bvh_build(_context().handle, mesh[0].data_ptr(), mesh[0].shape[0], mesh[1].data_ptr(),
                                      mesh[2].data_ptr(), mesh[1].shape[0], None, _abi.C.byref(h)), "aur_bvh_build")
    out = _closest_on_device(h, rays, s["hits"])
    bounds = (_abi.C.c_float * 6)()
    _abi.check(ab.lib().aur_bvh_info(h, None, None, bounds), "aur_bvh_info")
    out["bounds"] = np.array(bounds, np.float32)
    _abi.check(ab.lib().aur_bvh_destroy(h), "aur_bvh_destroy")
    return out


def run(s):
    case = s["case"]
    if case["kind"] == "build":
        return _run_build(s)
    if case["kind"] == "trace":
        bvh, rays = s["bvh"], s["rays"]
        if case["query"] == "intersect":
            rec, shrunk = bvh.intersect(rays)
            return {**{k: rec[k] for k in rec.dtype.names}, "maxt": shrunk[:, 7]}
        if case["query"] == "closest":
            return _closest_on_host(bvh, rays) if case["host"] else _closest_on_device(bvh.handle, rays, s["hits"])
        if case["host"]:
            return bvh.trace_occluded(rays)
        _abi.check(ab.lib().aur_trace_occluded(bvh.handle, rays.data_ptr(), s["occ"].data_ptr(), rays.shape[0]),
                   "aur_trace_occluded")
        return s["occ"]
    if case["kind"] == "batch":
        return ab.render_batch(s["scenes"], s["opts"], s["films"])[0]
    if case["kind"] == "adjoint":
        params = s["params"].detach().requires_grad_(True)
        texels = s["texels"].detach().requires_grad_(True)
        image = pyaurora.AuroraRender.apply(params, texels, s["scene"], s["options"])
        loss = ((image[..., :3] - s["target"]) ** 2).mean()
        loss.backward()
        return dict(image=image, params=params.grad, texels=texels.grad)
    if case["mode"] == "f64":
        return s["scene"].render_f64(s["opts"]).film
    return s["scene"].render(s["opts"], out=s["film"]).film


# ---------------------------------------------------------------------------- work and values
def _ntri(case):
    if case.get("mesh") == "bumpy":
        return 20 * 4 ** case["level"] + 2
    if case.get("mesh") == "terrain" or case.get("scene") == "terrain":
        return 2 * (case["grid"] - 1) ** 2 + 5120 * case["spheres"]
    return {"box": 36, "shaders": 5456}.get(case.get("scene"), 20804)


def _ray_flops(ntri):
    """One ray: a root-to-leaf walk of a four-wide tree (24 multiply-adds a node) and four
    triangle tests."""
    return 48.0 * max(1.0, math.log(ntri, 4)) + 4 * 46.0


def work(case):
    """Inputs read once and outputs written once. Rays per path: a closed box bounces to the
    depth limit with a next-event ray each; the open scenes average 2 closest-hit and 1.1 next-event
    rays (the terrain's measured means). Shading: about 300 operations a vertex; the adjoint
    traces each path twice (image and gradient) and shades it three times."""
    if case["kind"] in ("trace", "build"):
        nt, n = _ntri(case), case["n"]
        record = {"closest": 20, "occluded": 1, "intersect": 64 + 4}[case.get("query", "closest")]
        data = n * (32 + record)
        flops = n * _ray_flops(nt)
        if case["kind"] == "build":
            data += nt * (12 + 4 + 18)      # indices, attributes, half a vertex a triangle
            flops += nt * 30.0 * math.log2(nt)
        else:
            data += min(nt, n) * 48
        return dict(bytes=float(data), flops=float(flops))
    if case["kind"] == "batch":
        shapes = [_batch_shape(i) for i in range(case["count"])]
        paths = [(r * r * spp, d) for r, spp, d in shapes]
        return dict(bytes=float(sum(16 * r * r for r, _, _ in shapes)),
                    flops=float(sum(p * d * (2 * _ray_flops(36) + 300) for p, d in paths)))
    nt = _ntri(case)
    npix = case["w"] * case["h"]
    paths = npix * case["spp"] * case.get("lights", 1)
    rays, verts = (2.0 * case["depth"], case["depth"]) if case.get("scene") == "box" else (3.1, 2.0)
    film = 32 if case["mode"] == "f64" else 16
    data = npix * film + min(nt, paths) * (48 + 60)
    flops = paths * (rays * _ray_flops(nt) + verts * 300)
    if case["kind"] == "adjoint":
        data += npix * 16 + 2 * 4 * 64 * 64 * 3
        flops = paths * (2 * rays * _ray_flops(nt) + 3 * verts * 300)
    return dict(bytes=float(data), flops=float(flops))


def _brute_force(verts, faces, rays):
    """Closest hits in 64 bits by testing every triangle: (t, u, v, triangle) with triangle -1 for a
    miss. Moller-Trumbore in its Plucker form, a matrix product per chunk of rays."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.from_numpy(verts.astype(np.float64)).to(dev)
    f = torch.from_numpy(faces.astype(np.int64)).to(dev)
    r = torch.from_numpy(rays.astype(np.float64)).to(dev)
    p, e1, e2 = v[f[:, 0]], (v[f[:, 1]] - v[f[:, 0]]), (v[f[:, 2]] - v[f[:, 0]])
    nrm = torch.linalg.cross(e1, e2)
    # with m = o x d:  det = -d.n,  u det = (m + d x p).e2,  v det = -(m + d x p).e1,  t det = (o - p).n
    wu = torch.cat([e2, torch.linalg.cross(p, e2)], 1).T.contiguous()
    wv = -torch.cat([e1, torch.linalg.cross(p, e1)], 1).T.contiguous()
    pn = (p * nrm).sum(1)
    best = []
    step = max(1, int(3e8 / (8 * len(faces))))
    for k in range(0, len(r), step):
        o, d, lo, hi = r[k:k + step, 0:3], r[k:k + step, 4:7], r[k:k + step, 3:4], r[k:k + step, 7:8]
        det = -(d @ nrm.T)
        md = torch.cat([torch.linalg.cross(o, d), d], 1)
        u, w = (md @ wu) / det, (md @ wv) / det
        t = (o @ nrm.T - pn) / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t >= lo) & (t <= hi), t, torch.inf)
        tb, i = t.min(1)
        hit = torch.isfinite(tb)
        pick = i[:, None]
        zero = torch.zeros_like(tb)
        best.append((torch.where(hit, tb, hi[:, 0]), torch.where(hit, u.gather(1, pick)[:, 0], zero),
                     torch.where(hit, w.gather(1, pick)[:, 0], zero), torch.where(hit, i, -1)))
    return [torch.cat([b[q] for b in best]).cpu().numpy() for q in range(4)]


def exact(case, seed):
    """Ray queries on the small meshes have a value in 64 bits. A rendered film and its gradients
    have none that can be had without the renderer: they are sums over paths whose discrete
    choices (lobe, light, roulette, visibility) are decided by 32-bit numbers."""
    if case["kind"] not in ("trace", "build") or case["mesh"] != "bumpy" or case.get("query") == "occluded":
        return None
    if case["n"] * _ntri(case) > 2.5e10:
        return None
    verts, faces, attr, cn, cu = mesh = _mesh(case, seed)
    rays = _rays(case, mesh, seed)
    t, u, v, tri = _brute_force(verts, faces, rays)
    if case.get("query") != "intersect":
        out = dict(tuv=np.stack([t, u, v], 1), ids=None)
        if case["kind"] == "build":
            out["bounds"] = np.concatenate([verts.min(0), verts.max(0)]).astype(np.float64)
        return out
    hit = tri >= 0
    i = np.where(hit, tri, 0)
    w = 1.0 - u - v
    bar = np.stack([w, u, v], 1)
    d = rays[:, 4:7].astype(np.float64)
    nrm = (bar[:, :, None] * cn[i].reshape(-1, 3, 3).astype(np.float64)).sum(1)
    nrm = np.where((nrm * d).sum(1, keepdims=True) > 0, -nrm, nrm)
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-300)
    st = (bar[:, :, None] * cu[i].reshape(-1, 3, 2).astype(np.float64)).sum(1)
    z = hit[:, None]
    return dict(t=t, u=u, v=v, prim=None, attr=None, hitP=np.where(z, rays[:, :3] + d * t[:, None], 0.0),
                hitN=np.where(z, nrm, 0.0), st=np.where(z, st, 0.0),
                bar=np.where(z, np.stack([u, v, w], 1), 0.0), maxt=t)
