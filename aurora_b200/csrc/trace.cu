// trace.cu — batched closest-hit / occlusion queries over the device BVH.
// The C-ABI entry points aur_trace_closest / aur_trace_occluded / aur_bvh_intersect run these;
// they replace EmbreeAccelerator::intersect / intersectBinary
// (Aurora/src/geometry/embreeAccelerator.cpp:41-100) for arrays of rays.
//
// Three forms by the number of rays and the tree. Large batches run a resident grid whose lanes take the next
// ray as soon as theirs is finished, over the tree form the wavefront renderer uses (full-precision
// or quantised 4-wide nodes): 2^20 incoherent rays on 20,482 triangles 309 -> 254 us, 2^20 surface points
// towards a light on a 0.85 M triangle landscape 555 -> 336. Small ones cannot fill the chip and
// take as long as their longest ray's walk: a warp per ray walks it side by side, 1,000 rays
// 41 -> 22 us, of which 15 are the call's. In between, a thread per ray, spread over more warps
// with fewer rays each where there are few.
#include "aurora_b200.h"
#include "aur_kernels.h"
#include "aur_trace_split.h"
#include "aur_traverse.cuh"
#include <algorithm>

namespace aur {
namespace {

constexpr int kTraceRefill = 12;     // idle lanes of a warp that fetch new rays together
constexpr uint32_t kResidentMax = 1u << 31;   // its 32-bit cursor runs past the last ray by what is fetched at once
constexpr int kTraceRounds = 4;      // rounds between fetches (both as in the wavefront's kernels)

// Where a closest hit goes: the plain record, or the whole record of EmbreeAccelerator::intersect.
struct HitOut {
    aur_hit* hits;
    const int* tri_attr;
    __device__ __forceinline__ int& link(uint32_t i) const { return hits[i].prim; }   // a word of a record not yet written
    __device__ __forceinline__ void put(uint32_t i, const Hit& h, bool hit, const float4* rays) const {
        aur_hit* out = hits + i;
        out->t = hit ? h.t : rays[2 * (size_t)i + 1].w;
        out->u = hit ? h.u : 0.f;
        out->v = hit ? h.v : 0.f;
        out->prim = hit ? h.prim : -1;
        out->attr = hit ? (tri_attr ? tri_attr[h.prim] : 0) : -1;
    }
};

// The hit's post-process of EmbreeAccelerator::intersect (embreeAccelerator.cpp:49-91) with the
// per-corner normals and uvs the mesh retains (EmbreeMesh::normals / uvs, geometry/embreeMesh.h:62-63):
//   w = 1. - u - v (in double, rounded to float)
//   hitP = org + dir * t
//   hitN = normalize(w n0 + u n1 + v n2), negated first when it faces along dir
//   st   = w st0 + u st1 + v st2
//   barCoords = (u, v, w); ray.maxt = t on a hit (embreeAccelerator.cpp:56)
// The arithmetic is the shading frame's (hit_frame), so a hit reported here and the
// same hit shaded by the renderers agree bit for bit.
struct IsectOut {
    aur_isect* out;
    const TriShade* tri;
    __device__ __forceinline__ int& link(uint32_t i) const { return out[i].prim; }
    __device__ __forceinline__ void put(uint32_t i, const Hit& h, bool hit, float4* rays) const {
        const float4 a = rays[2 * (size_t)i], b = rays[2 * (size_t)i + 1];
        aur_isect r;
        if (!hit) {
            r.t = b.w; r.u = r.v = 0.f; r.prim = -1; r.attr = -1;
            for (int k = 0; k < 3; ++k) { r.hitP[k] = 0.f; r.hitN[k] = 0.f; r.bar[k] = 0.f; }
            r.st[0] = r.st[1] = 0.f;
            out[i] = r;
            return;
        }
        const float3 o = mk(a.x, a.y, a.z), d = mk(b.x, b.y, b.z);
        const float w = (float)(1.0 - h.u - h.v);
        const TriShade ts = load_tri(tri + h.prim);
        const float* nn = ts.n;
        float3 N = mk(w * nn[0] + h.u * nn[3] + h.v * nn[6],
                      w * nn[1] + h.u * nn[4] + h.v * nn[7],
                      w * nn[2] + h.u * nn[5] + h.v * nn[8]);
        if (dot(N, d) > 0.f) N *= -1.f;
        N = normalize(N);
        const float3 P = o + d * h.t;
        const float* uv = ts.uv;
        r.t = h.t; r.u = h.u; r.v = h.v; r.prim = h.prim;
        r.attr = ts.attr;
        r.hitP[0] = P.x; r.hitP[1] = P.y; r.hitP[2] = P.z;
        r.hitN[0] = N.x; r.hitN[1] = N.y; r.hitN[2] = N.z;
        r.st[0] = w * uv[0] + h.u * uv[2] + h.v * uv[4];
        r.st[1] = w * uv[1] + h.u * uv[3] + h.v * uv[5];
        r.bar[0] = h.u; r.bar[1] = h.v; r.bar[2] = w;
        out[i] = r;
        rays[2 * (size_t)i + 1].w = h.t;          // ray->maxt = t
    }
};

// Occlusion: no hit is put.
struct NoOut {
    __device__ __forceinline__ void put(uint32_t, const Hit&, bool, const float4*) const {}
};

template <class Out>
__global__ void __launch_bounds__(kTraceBlock) k_trace_closest(const BvhNode* __restrict__ nodes,
                                                               const BvhNode4* __restrict__ nodes4,
                                                               const BvhTri* __restrict__ tris, float4* rays, Out out,
                                                               uint32_t n, int per_warp) {
    const uint32_t i = spread_index(blockIdx.x, threadIdx.x, per_warp);
    if (i >= n) return;
    const float4 a = rays[2 * (size_t)i];
    const float4 b = rays[2 * (size_t)i + 1];
    Hit h;
    TraceWork w;
    const bool hit = bvh_closest(nodes, nodes4, tris, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, b.w, &h, w);
    out.put(i, h, hit, rays);
}

__global__ void __launch_bounds__(kTraceBlock) k_trace_occluded(const BvhNode* __restrict__ nodes,
                                                                const BvhNode4* __restrict__ nodes4,
                                                                const BvhTri* __restrict__ tris,
                                                                const float4* __restrict__ rays, uint8_t* occ,
                                                                uint32_t n, int per_warp) {
    const uint32_t i = spread_index(blockIdx.x, threadIdx.x, per_warp);
    if (i >= n) return;
    const float4 a = rays[2 * (size_t)i];
    const float4 b = rays[2 * (size_t)i + 1];
    TraceWork w;
    occ[i] = bvh_occluded(nodes, nodes4, tris, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, b.w, w) ? 1 : 0;
}

// One warp per ray: the lanes take up to 32 references off the warp's stack at a time, test their
// boxes or triangles together and push the children entered, so a ray's visits go on side by side
// instead of one dependent fetch after the other (a thousand rays take as long as the one with
// the longest walk). Without an order among the references more of them are visited. Where
// two triangles lie at exactly the closest distance the visiting order decides, and the ray is
// traced again in bvh_trace4's.
// The stack cannot overflow: fewer references are taken as it fills, down to one at a time, which
// needs three entries a level (at most kTraversalStack4, checked at build).
constexpr int kWarpStack = 1024;
template <bool kAnyHit, class Out>
__global__ void __launch_bounds__(kTraceBlock) k_trace_warp(const BvhNode4* __restrict__ nodes4,
                                                            const BvhTri* __restrict__ tris, float4* rays, Out out,
                                                            uint8_t* occ, uint32_t n) {
    __shared__ int s_stack[kTraceBlock / 32][kWarpStack];
    const int lane = threadIdx.x & 31;
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, before = (1u << lane) - 1u;
    if (i >= n) return;
    int* st = s_stack[threadIdx.x >> 5];
    const float4 ra = rays[2 * (size_t)i], rb = rays[2 * (size_t)i + 1];
    const float3 o = mk(ra.x, ra.y, ra.z), d = mk(rb.x, rb.y, rb.z);
    const float mint = ra.w;
    const float3 id = mk(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
    const float3 ood = mk(o.x * id.x, o.y * id.y, o.z * id.z);
    const float box_tmin = mint > 0.f ? mint * 0.99999905f : mint * 1.00000095f;
    const float kMiss = __int_as_float(0x7f800000);
    float tbest = rb.w, box_tmax = tbest * 1.00000095f;   // of the warp
    Hit h;                                                // of the lane
    h.t = kMiss; h.u = h.v = 0.f; h.prim = -1;
    bool tie = false, any = false;
    int sp = 1;
    if (lane == 0) st[0] = 0;
    __syncwarp();
    while (sp > 0) {
        const int room = (kWarpStack - kTraversalStack4 - sp) / 3;
        const int k = min(sp, max(1, min(32, room)));
        const int ref = lane < k ? st[sp - 1 - lane] : ~0;     // ~0: an empty leaf
        sp -= k;
        __syncwarp();
        float t[4] = {kMiss, kMiss, kMiss, kMiss};
        int r[4] = {~0, ~0, ~0, ~0};
        bool found = false;
        if (ref >= 0) {
            boxes4<kAnyHit>(nodes4 + ref, id, ood, box_tmin, box_tmax, t, r);
        } else {
            const int packed = ~ref;
            const int start = packed >> 5, end = start + (packed & 31);
            for (int q = start; q < end; ++q) {
                const float4 p = __ldg(&tris[q].p1);
                const float4 e1 = __ldg(&tris[q].e1);
                const float4 e2 = __ldg(&tris[q].e2);
                float tt, u, v;
                if (!tri_intersect(mk(p.x, p.y, p.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), o, d, mint, tbest,
                                   &tt, &u, &v)) continue;
                found = true;
                if (kAnyHit) break;
                if (h.prim >= 0 && !(tt < h.t)) {
                    tie = tie || !(tt > h.t);              // equal, or not a number
                } else {
                    tie = !(tt == tt);
                    h.t = tt; h.u = u; h.v = v; h.prim = __float_as_int(p.w);
                }
            }
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, found)) {
            if (kAnyHit) { any = true; break; }
            float best = h.t;
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, s));
            tbest = fminf(tbest, best);
            box_tmax = tbest * 1.00000095f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const bool in = t[c] != kMiss;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (in) st[sp + __popc(m & before)] = r[c];
            sp += __popc(m);
        }
        __syncwarp();
    }
    if (kAnyHit) {
        if (lane == 0) occ[i] = any ? 1 : 0;
        return;
    }
    // the lanes' closest hits: one of them is the ray's, unless several share its distance
    const uint32_t have = __ballot_sync(0xffffffffu, h.prim >= 0);
    const uint32_t bad = __ballot_sync(0xffffffffu, h.prim >= 0 && !(h.t == h.t));
    const uint32_t win = __ballot_sync(0xffffffffu, h.prim >= 0 && h.t <= tbest);
    const uint32_t tied = __ballot_sync(0xffffffffu, tie) & win;
    if (!have) {
        if (lane == 0) out.put(i, h, false, rays);
    } else if (bad || tied || __popc(win) != 1) {
        if (lane == 0) {
            TraceWork w;
            const bool hit = bvh_trace4<false>(nodes4, tris, o, d, mint, rb.w, &h, w);
            out.put(i, h, hit, rays);
        }
    } else if (lane == __ffs(win) - 1) {
        out.put(i, h, true, rays);
    }
}

// The resident form. Warps fetch ranges of rays from cursor[0]; the last block to leave clears the
// cursor (cursor[1] counts them), so that it is zero for its next user.
// Closest hits of the quantised tree that meet two triangles at exactly the same distance are traced again over the
// full-precision nodes: the thread keeps them in a list through their records (Out::link) until its warp is done.
template <bool kAnyHit, class Node4, class Out>
__global__ void __launch_bounds__(256, 4) k_trace_resident(const Node4* __restrict__ nodes, const BvhNode4* __restrict__ full,
                                                           const BvhTri* __restrict__ tris, float4* rays, Out out,
                                                           uint8_t* __restrict__ occ, uint32_t n, uint32_t* cursor) {
    constexpr bool kTies = !kAnyHit && sizeof(Node4) != sizeof(BvhNode4);
    extern __shared__ int s_stack[];
    __shared__ int s_tie[256];                    // first ray of the thread's list
    s_tie[threadIdx.x] = -1;
    LaneStack4 stack;
    stack.col = s_stack + threadIdx.x;
    stack.stride = blockDim.x;
    TraceState4<kAnyHit, Node4> ts;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t i = 0;
    bool has = false, exhausted = false;
    while (true) {
        const bool need = !has && !exhausted;
        const uint32_t m = __ballot_sync(0xffffffffu, need);
        const uint32_t act = __ballot_sync(0xffffffffu, has);
        if (m && (__popc(m) >= kTraceRefill || act == 0)) {
            const int leader = __ffs(m) - 1;
            uint32_t b = 0;
            if ((int)lane == leader) b = atomicAdd(&cursor[0], (uint32_t)__popc(m));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (need) {
                i = b + __popc(m & ((1u << lane) - 1u));
                if (i < n) {
                    const float4 o = rays[2 * (size_t)i], d = rays[2 * (size_t)i + 1];
                    ts.begin(mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), o.w, d.w);
                    has = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, has || !exhausted) == 0) break;
        for (int k = 0; k < kTraceRounds; ++k) ts.round(nodes, tris, stack);
        if (has && ts.finished()) {
            has = false;
            if constexpr (kAnyHit) {
                occ[i] = ts.hit_any ? 1 : 0;
            } else if (kTies && ts.tie) {
                out.link(i) = s_tie[threadIdx.x];
                s_tie[threadIdx.x] = (int)i;
            } else {
                Hit h;
                h.t = ts.tbest; h.u = ts.bu; h.v = ts.bv; h.prim = ts.best;
                out.put(i, h, ts.best >= 0, rays);
            }
        }
    }
    if constexpr (kTies) {
        for (int k = s_tie[threadIdx.x]; k >= 0;) {
            const int next = out.link(k);
            const float4 a = rays[2 * (size_t)k], b = rays[2 * (size_t)k + 1];
            Hit h;
            TraceWork w;
            const bool hit = bvh_trace4<false>(full, tris, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, b.w, &h, w);
            out.put(k, h, hit, rays);
            k = next;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&cursor[1], 1u) == gridDim.x - 1) {
        cursor[0] = 0u;
        cursor[1] = 0u;
    }
}

int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Up to this many rays per SM each has a warp of its own (14,208 on 148 SMs; none without a 4-wide tree). A
// warp per ray against spread threads, closest hits, 1,000 / 8,000 / 14,208 rays, incoherent: 20,482
// triangles 22 vs 38, 29 vs 44, 38 vs 51 us (occlusion 19 vs 36, 28 vs 42, 34 vs 45); 3.4 M triangles 24 vs 41,
// 32 vs 53, 40 vs 61 (21 vs 37, 28 vs 43, 34 vs 46). Past that
// camera rows and large trees turn: 20,000 rays of a camera on 0.85 M triangles 60 vs 58 us. A few
// dozen triangles leave most of a warp's lanes without work: 34 triangles, closest hits 1,000 / 4,000 /
// 8,000 rays 19.0 vs 19.1, 20.7 vs 19.8, 26.1 vs 21.0 us, any hit 15.3 vs 18.1, 16.4 vs 18.5, 19.6 vs 20.3.
uint32_t warp_rays(const DeviceBvh& bvh, bool any) {
    return !bvh.nodes4 ? 0u : bvh.num_nodes4 >= kQuantMinNodes4Any ? 96u : any ? 48u : 8u;
}

// The resident form from this many rays on. Against the thread form, closest hits, incoherent rays / surface points
// towards a light / rows of a camera: 20,482 triangles, 2^19 rays 153 vs 179, 303 vs 327, 143 vs 135 us, 2^20 rays 254 vs
// 309, 555 vs 599, 220 vs 205; any hit, 2^19 rays 123 vs 155, 205 vs 292, 114 vs 108. A camera's rows stay together by
// themselves, and on trees that sit in the caches the thread form's dense blocks are 4 to 8% ahead on them
// (walking them in step inside the resident grid, looking at a sample of the rays first, and ranges of
// each warp's own were no better). On quantised trees it is ahead on all three from 2^18 rays on: 0.85 M triangles
// 124 vs 121, 127 vs 177, 107 vs 105 (any hit 111 vs 108, 108 vs 154, 87 vs 89); 2^19 rays 164 vs 172, 195 vs 307,
// 152 vs 152; 3.4 M triangles, 2^20 rays 308 vs 402, 449 vs 744, 312 vs 374. On a few dozen triangles it gains
// nothing (34 triangles, 2^22 rays 269 vs 273, 292 vs 290, 172 vs 143).
uint32_t resident_min(const DeviceBvh& bvh) {
    return !bvh.nodes4 || bvh.num_nodes4 < kQuantMinNodes4Any ? 0xffffffffu : bvh.num_nodes4 >= kQuantMinNodes4 ? 1u << 18 : 1u << 19;
}

template <bool kAnyHit, class Node4, class Out>
cudaError_t run_resident(const DeviceBvh& bvh, const Node4* nodes, float4* rays, const Out& out, uint8_t* occ, uint32_t n,
                         int sms, uint32_t* cursor, cudaStream_t s) {
    const size_t smem = sizeof(int) * kSharedDepth * 256;
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_resident<kAnyHit, Node4, Out>, 256, smem);
    k_trace_resident<kAnyHit, Node4, Out><<<std::max(1, nb) * sms, 256, smem, s>>>(nodes, bvh.nodes4, bvh.tris, rays, out, occ, n,
                                                                                    cursor);
    return cudaGetLastError();
}

template <class Out>
cudaError_t run_closest(const DeviceBvh& bvh, float4* rays, const Out& out, uint32_t n, uint32_t* cursor, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int sms = sm_count();
    if (cursor && n >= resident_min(bvh) && n <= kResidentMax)
        return bvh.num_nodes4 >= kQuantMinNodes4 ? run_resident<false, BvhNode4Q>(bvh, bvh.nodes4q, rays, out, nullptr, n, sms, cursor, s)
                                                 : run_resident<false, BvhNode4>(bvh, bvh.nodes4, rays, out, nullptr, n, sms, cursor, s);
    if (n <= warp_rays(bvh, false) * (uint32_t)sms) {
        k_trace_warp<false, Out><<<spread_grid(n, 1), kTraceBlock, 0, s>>>(bvh.nodes4, bvh.tris, rays, out, nullptr, n);
        return cudaGetLastError();
    }
    const int r = rays_per_warp(n, sms);
    k_trace_closest<Out><<<spread_grid(n, r), kTraceBlock, 0, s>>>(bvh.nodes, bvh.nodes4, bvh.tris, rays, out, n, r);
    return cudaGetLastError();
}

}  // namespace

// rays: aur_ray records; written (maxt) by launch_intersect only
cudaError_t launch_trace_closest(const DeviceBvh& bvh, const int* tri_attr, const void* rays, void* hits, uint32_t n,
                                 uint32_t* cursor, cudaStream_t s) {
    return run_closest(bvh, (float4*)const_cast<void*>(rays), HitOut{(aur_hit*)hits, tri_attr}, n, cursor, s);
}

cudaError_t launch_intersect(const DeviceBvh& bvh, const TriShade* tri, void* rays, void* isects, uint32_t n, uint32_t* cursor,
                             cudaStream_t s) {
    return run_closest(bvh, (float4*)rays, IsectOut{(aur_isect*)isects, tri}, n, cursor, s);
}

cudaError_t launch_trace_occluded(const DeviceBvh& bvh, const void* rays, uint8_t* occ, uint32_t n, uint32_t* cursor, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int sms = sm_count();
    float4* r4 = (float4*)const_cast<void*>(rays);
    if (cursor && n >= resident_min(bvh) && n <= kResidentMax)   // such trees are past kQuantMinNodes4Any
        return run_resident<true, BvhNode4Q>(bvh, bvh.nodes4q, r4, NoOut{}, occ, n, sms, cursor, s);
    if (n <= warp_rays(bvh, true) * (uint32_t)sms) {
        k_trace_warp<true, NoOut><<<spread_grid(n, 1), kTraceBlock, 0, s>>>(bvh.nodes4, bvh.tris, r4, NoOut{}, occ, n);
        return cudaGetLastError();
    }
    const int r = rays_per_warp(n, sms);
    k_trace_occluded<<<spread_grid(n, r), kTraceBlock, 0, s>>>(bvh.nodes, bvh.nodes4, bvh.tris, r4, occ, n, r);
    return cudaGetLastError();
}

}  // namespace aur
