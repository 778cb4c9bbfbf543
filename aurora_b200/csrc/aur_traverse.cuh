// aur_traverse.cuh — closest-hit and any-hit traversal of the device BVH.
//
// Replaces EmbreeAccelerator::intersect / intersectBinary
// (Aurora/src/geometry/embreeAccelerator.cpp:41-100): closest hit in
// [mint, maxt] returning (t, u, v, prim) with Embree's barycentric convention
// (u weights vertex 1, v vertex 2), and occlusion anywhere in [mint, maxt].
// Nodes and triangles are fetched with 128-bit read-only loads; the traversal
// stack lives in registers/local memory (64 entries, ample for PLOC trees).
// The triangle test is the exact FP32 Moller-Trumbore of tri_intersect, so the
// closest prim equals a brute-force scan's whenever the minimum is unique.
#pragma once
#include <climits>
#include "aur_bvh.cuh"
#include "aur_shading.cuh"

namespace aur {

struct Hit { float t, u, v; int prim; };

// Work counters of one or more traversals: interior-node visits (one 64-byte
// record each) and triangle tests (one 48-byte record each). Kernels that do
// not store them let the compiler drop the increments.
struct TraceWork { uint32_t nodes = 0, tris = 0; };

constexpr int kTraversalStack = 64;

__device__ __forceinline__ float safe_rcp(float x) {
    return __frcp_rn(fabsf(x) > 1e-20f ? x : copysignf(1e-20f, x));
}

// Slab test against one child box; tmin/tmax already carry the rounding slack.
__device__ __forceinline__ bool slab(float lox, float hix, float loy, float hiy, float loz, float hiz,
                                     float3 id, float3 ood, float tmin, float tmax, float* tnear) {
    const float x0 = fmaf(lox, id.x, -ood.x), x1 = fmaf(hix, id.x, -ood.x);
    const float y0 = fmaf(loy, id.y, -ood.y), y1 = fmaf(hiy, id.y, -ood.y);
    const float z0 = fmaf(loz, id.z, -ood.z), z1 = fmaf(hiz, id.z, -ood.z);
    const float tn = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fmaxf(fminf(z0, z1), tmin));
    const float tf = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fminf(fmaxf(z0, z1), tmax));
    *tnear = tn;
    return tn <= tf;
}

// Slab test with the near and far planes already chosen by the ray direction's signs
// (for a positive inverse direction the near plane is lo, else hi): the same entry and
// exit distances as slab(), without the per-axis min/max.
__device__ __forceinline__ bool slab_nf(float nx, float fx, float ny, float fy, float nz, float fz, float3 id,
                                        float3 ood, float tmin, float tmax, float* tnear) {
    const float tn = fmaxf(fmaxf(fmaf(nx, id.x, -ood.x), fmaf(ny, id.y, -ood.y)), fmaxf(fmaf(nz, id.z, -ood.z), tmin));
    const float tf = fminf(fminf(fmaf(fx, id.x, -ood.x), fmaf(fy, id.y, -ood.y)), fminf(fmaf(fz, id.z, -ood.z), tmax));
    *tnear = tn;
    return tn <= tf;
}

__device__ __forceinline__ float4 ld_node(const float4* a) { return __ldg(a); }

// 32 contiguous bytes in one 256-bit read-only load (sm_100: ld.global.nc.v8.f32, address
// 32-byte aligned): one L1 request per lane where two 128-bit loads take two.
__device__ __forceinline__ void ld_node2(const float4* a, float4& x, float4& y) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w)
        : "l"(a));
}

// The four children's near and far planes of a 4-wide node, by the direction's signs
// (lox, hix, loy, hiy, loz, hiz order). kLoad256: both planes of each axis in one 256-bit
// load, then chosen by sign in registers (3 load requests instead of 6). Measured on the
// 1080p terrain: the any-hit (next-event) traversal 57.6 vs 59.5 ms per frame with it, the
// closest-hit traversal 118.2 vs 109.2 ms (its 64-register budget spills), so only the
// any-hit traversals use it.
struct Planes4 { float4 nx, fx, ny, fy, nz, fz; };
template <bool kLoad256>
__device__ __forceinline__ Planes4 load_planes4(const BvhNode4* q, float3 id) {
    const float4* p = reinterpret_cast<const float4*>(q);
    Planes4 r;
    if constexpr (kLoad256) {
        float4 lx, hx, ly, hy, lz, hz;
        ld_node2(p, lx, hx);
        ld_node2(p + 2, ly, hy);
        ld_node2(p + 4, lz, hz);
        const bool nx = id.x < 0.f, ny = id.y < 0.f, nz = id.z < 0.f;
        r.nx = nx ? hx : lx; r.fx = nx ? lx : hx;
        r.ny = ny ? hy : ly; r.fy = ny ? ly : hy;
        r.nz = nz ? hz : lz; r.fz = nz ? lz : hz;
    } else {
        const int sx = id.x < 0.f, sy = id.y < 0.f, sz = id.z < 0.f;
        r.nx = ld_node(p + sx); r.fx = ld_node(p + 1 - sx);
        r.ny = ld_node(p + 2 + sy); r.fy = ld_node(p + 3 - sy);
        r.nz = ld_node(p + 4 + sz); r.fz = ld_node(p + 5 - sz);
    }
    return r;
}

// kAnyHit=false: closest hit, returns true when hit->prim >= 0.
// kAnyHit=true : returns true as soon as any triangle is hit in [mint, maxt].
template <bool kAnyHit>
__device__ __forceinline__ bool bvh_trace(const BvhNode* __restrict__ nodes, const BvhTri* __restrict__ tris,
                                          float3 o, float3 d, float mint, float maxt, Hit* hit, TraceWork& work) {
    const float3 id = mk(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
    const float3 ood = mk(o.x * id.x, o.y * id.y, o.z * id.z);
    const float box_tmin = mint > 0.f ? mint * 0.99999905f : mint * 1.00000095f;
    float tbest = maxt;
    float box_tmax = tbest * 1.00000095f;
    int best = -1;
    float bu = 0.f, bv = 0.f;
    int stack[kTraversalStack];
    int sp = 0;
    int node = 0;
    while (true) {
        if (node >= 0) {
            ++work.nodes;
            const float4 a = __ldg(&nodes[node].a);
            const float4 b = __ldg(&nodes[node].b);
            const float4 c = __ldg(&nodes[node].c);
            const float4 e = __ldg(&nodes[node].d);
            float t0, t1;
            const bool h0 = slab(a.x, a.y, a.z, a.w, c.x, c.y, id, ood, box_tmin, box_tmax, &t0);
            const bool h1 = slab(b.x, b.y, b.z, b.w, c.z, c.w, id, ood, box_tmin, box_tmax, &t1);
            const int r0 = __float_as_int(e.x), r1 = __float_as_int(e.y);
            if (h0 && h1) {
                const bool first0 = t0 <= t1;
                if (sp < kTraversalStack) stack[sp++] = first0 ? r1 : r0;   // depth <= 63 is checked at build
                node = first0 ? r0 : r1;
                continue;
            }
            if (h0) { node = r0; continue; }
            if (h1) { node = r1; continue; }
        } else {
            const int packed = ~node;
            const int start = packed >> 5, end = start + (packed & 31);
            for (int k = start; k < end; ++k) {
                ++work.tris;
                const float4 p = __ldg(&tris[k].p1);
                const float4 e1 = __ldg(&tris[k].e1);
                const float4 e2 = __ldg(&tris[k].e2);
                float t, u, v;
                if (tri_intersect(mk(p.x, p.y, p.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), o, d, mint, tbest,
                                  &t, &u, &v)) {
                    if (kAnyHit) return true;
                    tbest = t; bu = u; bv = v;
                    best = __float_as_int(p.w);
                    box_tmax = tbest * 1.00000095f;
                }
            }
        }
        if (sp == 0) break;
        node = stack[--sp];
    }
    if (kAnyHit) return false;
    hit->t = tbest; hit->u = bu; hit->v = bv; hit->prim = best;
    return best >= 0;
}

// Entry distances of the four children of a full-precision 4-wide node (+inf where missed) and
// their references.
template <bool kAnyHit>
__device__ __forceinline__ void boxes4(const BvhNode4* __restrict__ q, float3 id, float3 ood, float tmin, float tmax,
                                       float (&t)[4], int (&r)[4]) {
    const Planes4 pl = load_planes4<kAnyHit>(q, id);
    const float4 rf = ld_node(reinterpret_cast<const float4*>(&q->ref));
    const float kMiss = __int_as_float(0x7f800000);
    float tc;
    t[0] = slab_nf(pl.nx.x, pl.fx.x, pl.ny.x, pl.fy.x, pl.nz.x, pl.fz.x, id, ood, tmin, tmax, &tc) ? tc : kMiss;
    t[1] = slab_nf(pl.nx.y, pl.fx.y, pl.ny.y, pl.fy.y, pl.nz.y, pl.fz.y, id, ood, tmin, tmax, &tc) ? tc : kMiss;
    t[2] = slab_nf(pl.nx.z, pl.fx.z, pl.ny.z, pl.fy.z, pl.nz.z, pl.fz.z, id, ood, tmin, tmax, &tc) ? tc : kMiss;
    t[3] = slab_nf(pl.nx.w, pl.fx.w, pl.ny.w, pl.fy.w, pl.nz.w, pl.fz.w, id, ood, tmin, tmax, &tc) ? tc : kMiss;
    r[0] = __float_as_int(rf.x); r[1] = __float_as_int(rf.y); r[2] = __float_as_int(rf.z); r[3] = __float_as_int(rf.w);
}

__device__ __forceinline__ void ld_words8(const uint32_t* a, uint32_t (&v)[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(a));
}
// byte k of w as 1 + byte * 2^-15: one byte permutation, no integer conversion
__device__ __forceinline__ float plane_f(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7604u | ((uint32_t)k << 4)));
}
// a * m + c for two planes in one packed FMA (each half rounded as fmaf)
__device__ __forceinline__ float2 fma_pair(float2 a, float m, float c) {
    float2 r;
    asm("{.reg .b64 x, y, z, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mov.b64 z, {%5, %5};\n"
        " fma.rn.f32x2 w, x, y, z;\n mov.b64 {%0, %1}, w;}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(m), "f"(c));
    return r;
}

// The same for a quantised node. The traversals are bound by the L1's request rate and by the
// latency of dependent fetches, not by instruction issue alone (an extra prefetch per leaf made
// the any-hit kernel 15% slower; 68% of issue slots are busy): two 256-bit loads a visit replace
// seven requests (four in the any-hit form). A plane at byte q lies at p + s (1 + q 2^-15), so
// its distance is one FMA of the byte permuted into a float's mantissa; packed FMAs take two
// children at a time. 1080p terrain frame, closest hit / any hit: full precision 106.8 / 54.8 ms,
// quantised 102.0 / 49.1, with packed FMAs 98.0 / 45.5, with the rounds below free of a lane's
// live flags and 12 idle lanes to a refill 95.9 / 44.2.
template <bool kAnyHit>
__device__ __forceinline__ void boxes4(const BvhNode4Q* __restrict__ node, float3 id, float3 ood, float tmin, float tmax,
                                       float (&t)[4], int (&r)[4]) {
    uint32_t a[8], b[8];
    const uint32_t* q = reinterpret_cast<const uint32_t*>(node);
    ld_words8(q, a);
    ld_words8(q + 8, b);
    const float kMiss = __int_as_float(0x7f800000);
    const float3 S = mk(__uint_as_float(a[3]) * id.x, __uint_as_float(a[4]) * id.y, __uint_as_float(a[5]) * id.z);
    const float3 B = mk(fmaf(__uint_as_float(a[0]), id.x, -ood.x), fmaf(__uint_as_float(a[1]), id.y, -ood.y),
                        fmaf(__uint_as_float(a[2]), id.z, -ood.z));
    const bool sx = id.x < 0.f, sy = id.y < 0.f, sz = id.z < 0.f;
    const uint32_t nx = sx ? a[7] : a[6], fx = sx ? a[6] : a[7];
    const uint32_t ny = sy ? b[1] : b[0], fy = sy ? b[0] : b[1];
    const uint32_t nz = sz ? b[3] : b[2], fz = sz ? b[2] : b[3];
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        auto two = [&](uint32_t w, float m, float c) {
            return fma_pair(make_float2(plane_f(w, k), plane_f(w, k + 1)), m, c);
        };
        const float2 ax = two(nx, S.x, B.x), ay = two(ny, S.y, B.y), az = two(nz, S.z, B.z);
        const float2 bx = two(fx, S.x, B.x), by = two(fy, S.y, B.y), bz = two(fz, S.z, B.z);
        const float n0 = fmaxf(fmaxf(ax.x, ay.x), fmaxf(az.x, tmin)), f0 = fminf(fminf(bx.x, by.x), fminf(bz.x, tmax));
        const float n1 = fmaxf(fmaxf(ax.y, ay.y), fmaxf(az.y, tmin)), f1 = fminf(fminf(bx.y, by.y), fminf(bz.y, tmax));
        t[k] = n0 <= f0 ? n0 : kMiss;
        t[k + 1] = n1 <= f1 ? n1 : kMiss;
    }
    for (int k = 0; k < 4; ++k) r[k] = (int)b[4 + k];
}

// Puts the entered children in ascending order of entry distance, misses last: a five-exchange
// network; unless kSorted only the first place is right (any hit, where the order of the rest
// matters less than its cost: 45.1 vs 45.5 ms per 1080p terrain frame).
template <bool kSorted>
__device__ __forceinline__ void order4(float (&t)[4], int (&r)[4]) {
    auto cx = [&](int i, int j) {
        if (t[j] < t[i]) { const float tt = t[i]; t[i] = t[j]; t[j] = tt; const int rr = r[i]; r[i] = r[j]; r[j] = rr; }
    };
    cx(0, 1); cx(2, 3); cx(0, 2);
    if (kSorted) { cx(1, 3); cx(1, 2); }
}

// The same traversal over a 4-wide tree, children nearest first. *tie (may be null): a second
// triangle was accepted at exactly the best distance, so that the hit's identity depends on the
// visiting order.
constexpr int kTraversalStack4Local = 96;
template <bool kAnyHit, class Node4>
__device__ __forceinline__ bool bvh_trace4(const Node4* __restrict__ nodes, const BvhTri* __restrict__ tris,
                                           float3 o, float3 d, float mint, float maxt, Hit* hit, TraceWork& work,
                                           bool* tie = nullptr) {
    const float3 id = mk(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
    const float3 ood = mk(o.x * id.x, o.y * id.y, o.z * id.z);
    const float box_tmin = mint > 0.f ? mint * 0.99999905f : mint * 1.00000095f;
    const float kMiss = __int_as_float(0x7f800000);
    float tbest = maxt;
    float box_tmax = tbest * 1.00000095f;
    int best = -1;
    float bu = 0.f, bv = 0.f;
    int stack[kTraversalStack4Local];
    int sp = 0;
    int node = 0;
    while (true) {
        if (node >= 0) {
            ++work.nodes;
            float t[4];
            int r[4];
            boxes4<kAnyHit>(nodes + node, id, ood, box_tmin, box_tmax, t, r);
            order4<true>(t, r);
            if (t[0] != kMiss) {
                if (t[3] != kMiss && sp < kTraversalStack4Local) stack[sp++] = r[3];
                if (t[2] != kMiss && sp < kTraversalStack4Local) stack[sp++] = r[2];
                if (t[1] != kMiss && sp < kTraversalStack4Local) stack[sp++] = r[1];
                node = r[0];
                continue;
            }
        } else {
            const int packed = ~node;
            const int start = packed >> 5, end = start + (packed & 31);
            for (int k = start; k < end; ++k) {
                ++work.tris;
                const float4 p = __ldg(&tris[k].p1);
                const float4 e1 = __ldg(&tris[k].e1);
                const float4 e2 = __ldg(&tris[k].e2);
                float t, u, v;
                if (tri_intersect(mk(p.x, p.y, p.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), o, d, mint, tbest,
                                  &t, &u, &v)) {
                    if (kAnyHit) return true;
                    if (tie) *tie = *tie || (!(t < tbest) && best >= 0);   // equal, or not a number
                    tbest = t; bu = u; bv = v;
                    best = __float_as_int(p.w);
                    box_tmax = tbest * 1.00000095f;
                }
            }
        }
        if (sp == 0) break;
        node = stack[--sp];
    }
    if (kAnyHit) return false;
    hit->t = tbest; hit->u = bu; hit->v = bv; hit->prim = best;
    return best >= 0;
}

__device__ __forceinline__ bool bvh_closest(const BvhNode* nodes, const BvhTri* tris, float3 o, float3 d, float mint,
                                            float maxt, Hit* hit, TraceWork& work) {
    return bvh_trace<false>(nodes, tris, o, d, mint, maxt, hit, work);
}
__device__ __forceinline__ bool bvh_occluded(const BvhNode* nodes, const BvhTri* tris, float3 o, float3 d, float mint,
                                             float maxt, TraceWork& work) {
    Hit h;
    return bvh_trace<true>(nodes, tris, o, d, mint, maxt, &h, work);
}
// The 4-wide tree when there is one, else the binary tree.
__device__ __forceinline__ bool bvh_closest(const BvhNode* nodes, const BvhNode4* nodes4, const BvhTri* tris, float3 o,
                                            float3 d, float mint, float maxt, Hit* hit, TraceWork& work) {
    if (nodes4) return bvh_trace4<false>(nodes4, tris, o, d, mint, maxt, hit, work);
    return bvh_trace<false>(nodes, tris, o, d, mint, maxt, hit, work);
}
__device__ __forceinline__ bool bvh_occluded(const BvhNode* nodes, const BvhNode4* nodes4, const BvhTri* tris, float3 o,
                                             float3 d, float mint, float maxt, TraceWork& work) {
    Hit h;
    if (nodes4) return bvh_trace4<true>(nodes4, tris, o, d, mint, maxt, &h, work);
    return bvh_trace<true>(nodes, tris, o, d, mint, maxt, &h, work);
}

}  // namespace aur

namespace aur {

// Traversal stack of one thread: the first kSharedDepth entries live in shared
// memory laid out [depth][thread] (consecutive threads hit consecutive banks at
// any mix of depths, one wavefront per warp access), deeper entries in local memory.
constexpr int kSharedDepth = 24;   // all-local stacks measured 1.7% slower in k_extend
// A 4-wide node pushes up to three entries: the stack of its traversal holds 96
// (the collapse checks 3 x 4-wide depth + 1 against it).
constexpr int kTraversalStack4 = 96;
template <int kCap>
struct LaneStackT {
    int* col;                       // &s_stack[threadIdx.x]
    int stride;                     // blockDim.x
    int deep[kCap - kSharedDepth];
    __device__ __forceinline__ void set(int i, int v) {
        if (i < kSharedDepth) col[i * stride] = v; else deep[i - kSharedDepth] = v;
    }
    __device__ __forceinline__ int get(int i) const {
        return i < kSharedDepth ? col[i * stride] : deep[i - kSharedDepth];
    }
};
using LaneStack = LaneStackT<kTraversalStack>;
using LaneStack4 = LaneStackT<kTraversalStack4>;

// Resumable traversal of one ray, for persistent kernels whose lanes take a new ray as soon
// as theirs finishes (lane refill). Same slack and exact triangle test as bvh_trace.
//
// round() advances every lane of a warp by one round of "while-while" traversal with
// speculative leaf postponing (Aila & Laine, "Understanding the Efficiency of Ray Traversal
// on GPUs", HPG 2009): in the interior phase a lane walks down until it holds a leaf, and one
// that holds one walks on speculatively; then all lanes test their leaf's triangles together.
// The interior phase ends when at most kMaxSearching lanes are still without a leaf (they go on
// in the next round) instead of when none is: waiting for the last few left most of the warp
// idle. Measured per 1080p terrain frame on the full-precision 4-wide nodes, at a limit of 0 /
// 4 / 6 / 8 / 10 lanes: closest hit 120.9 / 107.7 / 106.8 / 107.0 / 107.2 ms, any hit 60.3 /
// 55.0 / 54.8 / 55.2 / 55.6 ms. The order in which a ray tests its leaves does not depend on it.
// All 32 lanes of the warp must call round(); lanes without a ray hold node = leaf = kNoNode.
constexpr int kMaxSearching = 6;
constexpr int kNoNode = INT_MIN;

// What every form of the resumable traversal keeps per ray.
struct TraceLane {
    float3 o, d, id, ood;
    float mint, tbest, box_tmin, box_tmax, bu, bv;
    int node = kNoNode, leaf = kNoNode;   // next node (>= 0) or leaf reference; the postponed leaf
    int sp = 0, best;                 // stack entries: none once finished
    bool hit_any;                     // any hit: something was hit
    bool tie;                         // closest hit: a second triangle lies at exactly the best distance

    __device__ __forceinline__ void begin(float3 o_, float3 d_, float mint_, float maxt_) {
        o = o_; d = d_;
        id = mk(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
        ood = mk(o.x * id.x, o.y * id.y, o.z * id.z);
        mint = mint_;
        box_tmin = mint > 0.f ? mint * 0.99999905f : mint * 1.00000095f;
        tbest = maxt_;
        box_tmax = tbest * 1.00000095f;
        bu = bv = 0.f;
        node = 0; sp = 0; best = -1;
        leaf = kNoNode;
        hit_any = tie = false;
    }
    __device__ __forceinline__ bool finished() const { return node == kNoNode && leaf == kNoNode; }

    template <class Stack>
    __device__ __forceinline__ int pop(Stack& stack) { return sp > 0 ? stack.get(--sp) : kNoNode; }

    // The postponed leaf's triangles.
    template <bool kAnyHit>
    __device__ __forceinline__ void test_leaf(const BvhTri* __restrict__ tris) {
        const int packed = ~leaf;
        const int start = packed >> 5, end = start + (packed & 31);
        leaf = kNoNode;
        for (int k = start; k < end; ++k) {
            const float4 p = __ldg(&tris[k].p1);
            const float4 e1 = __ldg(&tris[k].e1);
            const float4 e2 = __ldg(&tris[k].e2);
            float t, u, v;
            if (tri_intersect(mk(p.x, p.y, p.z), mk(e1.x, e1.y, e1.z), mk(e2.x, e2.y, e2.z), o, d, mint, tbest,
                              &t, &u, &v)) {
                if (kAnyHit) { hit_any = true; node = kNoNode; sp = 0; return; }
                tie = tie || (!(t < tbest) && best >= 0);   // equal, or not a number
                tbest = t; bu = u; bv = v;
                best = __float_as_int(p.w);
                box_tmax = tbest * 1.00000095f;
            }
        }
    }
};

// One round over any of the trees: `visit` steps a lane whose node is an interior one.
template <bool kAnyHit, class Stack, class Visit>
__device__ __forceinline__ void trace_round(TraceLane& s, const BvhTri* __restrict__ tris, Stack& stack, Visit visit) {
    while (true) {
        if (s.node >= 0) visit();
        if (s.node < 0 && s.leaf == kNoNode) {   // postpone this leaf (kNoNode stays kNoNode: the stack is empty then)
            s.leaf = s.node;
            s.node = s.pop(stack);
        }
        const bool searching = s.leaf == kNoNode && s.node != kNoNode;
        if (__popc(__ballot_sync(0xffffffffu, searching)) <= kMaxSearching) break;
    }
    if (s.leaf != kNoNode) s.test_leaf<kAnyHit>(tris);
}

// Over the binary tree, in the visiting order of bvh_trace.
template <bool kAnyHit>
struct TraceState : TraceLane {
    __device__ __forceinline__ void visit(const BvhNode* __restrict__ nodes, LaneStack& stack) {
        const float4 a = __ldg(&nodes[node].a);
        const float4 b = __ldg(&nodes[node].b);
        const float4 c = __ldg(&nodes[node].c);
        const float4 e = __ldg(&nodes[node].d);
        float t0, t1;
        const bool h0 = slab(a.x, a.y, a.z, a.w, c.x, c.y, id, ood, box_tmin, box_tmax, &t0);
        const bool h1 = slab(b.x, b.y, b.z, b.w, c.z, c.w, id, ood, box_tmin, box_tmax, &t1);
        const int r0 = __float_as_int(e.x), r1 = __float_as_int(e.y);
        if (h0 && h1) {
            const bool first0 = t0 <= t1;
            if (sp < kTraversalStack) stack.set(sp++, first0 ? r1 : r0);   // depth <= 63 is checked at build
            node = first0 ? r0 : r1;
        } else if (h0) node = r0;
        else if (h1) node = r1;
        else node = pop(stack);
    }
    __device__ __forceinline__ void round(const BvhNode* __restrict__ nodes, const BvhTri* __restrict__ tris,
                                          LaneStack& stack) {
        trace_round<kAnyHit>(*this, tris, stack, [&]() { visit(nodes, stack); });
    }
};

// Over a 4-wide tree: the nearest child entered comes next, the others go on the stack, farthest
// first (three entries a level at most: checked against the stack at build).
template <bool kAnyHit, class Node4>
struct TraceState4 : TraceLane {
    __device__ __forceinline__ void visit(const Node4* __restrict__ nodes, LaneStack4& stack) {
        const float kMiss = __int_as_float(0x7f800000);
        float t[4];
        int r[4];
        boxes4<kAnyHit>(nodes + node, id, ood, box_tmin, box_tmax, t, r);
        order4<!kAnyHit>(t, r);
        if (t[0] == kMiss) { node = pop(stack); return; }
        if (t[3] != kMiss) stack.set(sp++, r[3]);
        if (t[2] != kMiss) stack.set(sp++, r[2]);
        if (t[1] != kMiss) stack.set(sp++, r[1]);
        node = r[0];
    }
    __device__ __forceinline__ void round(const Node4* __restrict__ nodes, const BvhTri* __restrict__ tris,
                                          LaneStack4& stack) {
        trace_round<kAnyHit>(*this, tris, stack, [&]() { visit(nodes, stack); });
    }
};

}  // namespace aur
