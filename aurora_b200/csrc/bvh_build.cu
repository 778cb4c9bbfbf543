// bvh_build.cu — SAH-quality BVH built entirely on the device.
//
// Stands in for embree::rtcCreateAccel("bvh4.spatialsplit", "triangle4", ...)
// (Aurora/src/geometry/embreeAccelerator.cpp:24-32) over the flattened
// camera-space triangle soup of Renderer::buildRenderEnvironment
// (Aurora/src/frontend/renderer.cpp:99-145, triangleMesh.cpp:57-81).
//
// Pipeline (all kernels in this file, no library calls):
//   1. scene and centroid bounds, index check         k_bounds
//   2. 30-bit Morton codes, stable LSD radix sort     k_morton, k_sort_*
//   3. PLOC agglomerative clustering (Meister & Bittner, "Parallel Locally-
//      Ordered Clustering for BVH Construction", IEEE TVCG 2018): every cluster
//      finds its nearest neighbour (smallest merged surface area) within a
//      window of the Morton order; mutual pairs merge; the list is compacted
//      in order. Ties are broken on the index pair so that the globally best
//      pair is always mutual (guaranteed progress).
//      A merge also decides, from its two finished children, whether the new
//      node collapses into a leaf by the SAH, and its row of the dynamic
//      program that groups binary nodes into 4-wide ones (step 5); both need
//      nothing but the children, and as passes of their own they climbed the
//      finished tree with an atomic and a fence a level.
//   4. deterministic depth-first layout: every node derives its output slot by
//      walking to the root, so the result is independent of thread timing.
//   5. the 4-wide tree: an SAH-optimal grouping of the binary nodes, built
//      level by level, and its quantised form.
//
// Small meshes are bound by launches and host reads, large ones by the traffic of each pass:
// two launches a PLOC iteration (search and merge, compaction) where there were eight, one block
// for all iterations from kFinish clusters on, no pass over the finished tree for the SAH and the
// grouping, boxes recomputed from the vertices instead of kept, one allocation. Build and a
// batch of rays: 3.4 M triangles from device arrays with 262,144 rays 6.2 -> 2.55 ms, 20,482
// triangles from host arrays with 16,384 rays 2.0 -> 0.74 ms.
#include "aur_bvh.cuh"
#include "aur_shading.cuh"
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

namespace aur {
namespace {

#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return e_; } while (0)

template <typename T>
cudaError_t dalloc(T** p, size_t n, cudaStream_t s) { return cudaMallocAsync((void**)p, sizeof(T) * (n ? n : 1), s); }

inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// Exclusive prefix of v over the block (at most 1024 threads; all of them call it) and the
// block's total. s: 33 words, free for reuse after the caller's next barrier.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) s[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t x = lane < nw ? s[lane] : 0u;
        const uint32_t y = warp_incl_scan(x);
        s[lane] = y - x;
        if (lane == 31) s[32] = y;
    }
    __syncthreads();
    *total = s[32];
    return incl - v + s[warp];
}

// ------------------------------------------------------------ radix sort
// Stable LSD sort of (key, value) pairs, 10 bits per pass, three passes for the 30-bit codes. A
// block of 8 warps takes a tile of up to 4096 pairs in order, each warp a contiguous eighth: per warp
// and digit counts (phase 1), a prefix over the warps (phase 2), then every pair's place from its
// warp's counter and its rank among the equal digits of its 32 (phase 3). One warp per block
// over 2048 pairs, 8 bits a pass, spent 56 + 36 us a pass however small the array.
constexpr int kDigits = 1024;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// pairs per thread: 16, or 4 (tiles of 1024) for arrays of up to kSmallSort pairs, which
// otherwise occupy a few SMs for the length of a tile
constexpr int kSmallSort = 1 << 18;

template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const uint32_t* __restrict__ keys, int n, int shift,
                                                            uint32_t* __restrict__ hist, int nb) {
    __shared__ uint32_t s_h[kDigits];
    for (int d = threadIdx.x; d < kDigits; d += kSortThreads) s_h[d] = 0;
    __syncthreads();
    const int base = blockIdx.x * (kSortThreads * kItems);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = base + k * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&s_h[(keys[i] >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSortThreads) hist[(size_t)d * nb + blockIdx.x] = s_h[d];
}

inline int sort_tile(long long n) { return kSortThreads * (n <= kSmallSort ? 4 : 16); }

// One warp per digit: exclusive prefix of the digit's counts over the tiles, in place, and its total.
__global__ void k_sort_rows(uint32_t* hist, int nb, uint32_t* __restrict__ total) {
    const int d = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (d >= kDigits) return;
    uint32_t* row = hist + (size_t)d * nb;
    uint32_t run = 0;
    for (int b = 0; b < nb; b += 32) {
        const uint32_t v = b + lane < nb ? row[b + lane] : 0u;
        const uint32_t incl = warp_incl_scan(v);
        if (b + lane < nb) row[b + lane] = run + incl - v;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) total[d] = run;
}

template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(const uint32_t* __restrict__ keys,
                                                               const uint32_t* __restrict__ vals, uint32_t* okeys,
                                                               uint32_t* ovals, int n, int shift,
                                                               const uint32_t* __restrict__ rows,
                                                               const uint32_t* __restrict__ total, int nb) {
    __shared__ uint32_t s_cnt[kSortWarps][kDigits];
    __shared__ uint32_t s_scan[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < kSortWarps * kDigits; d += kSortThreads) (&s_cnt[0][0])[d] = 0;
    __syncthreads();
    const int base = blockIdx.x * (kSortThreads * kItems) + warp * (32 * kItems);
    uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = base + k * 32 + lane;
        key[k] = i < n ? keys[i] : 0xffffffffu;
        val[k] = i < n ? vals[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const bool valid = base + k * 32 + lane < n;
        const uint32_t d = (key[k] >> shift) & (kDigits - 1);
        const uint32_t peers = __match_any_sync(0xffffffffu, valid ? d : kDigits);
        rank[k] = 0;
        if (valid) rank[k] = s_cnt[warp][d] + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) s_cnt[warp][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // digits 4 t .. 4 t + 3 of thread t: the digit's first place in the output, then its warps in order
    uint32_t sum = 0, tot[kDigits / kSortThreads], unused;
#pragma unroll
    for (int q = 0; q < kDigits / kSortThreads; ++q) { tot[q] = total[threadIdx.x * (kDigits / kSortThreads) + q]; sum += tot[q]; }
    uint32_t first = block_excl_scan(sum, s_scan, &unused);
#pragma unroll
    for (int q = 0; q < kDigits / kSortThreads; ++q) {
        const int d = threadIdx.x * (kDigits / kSortThreads) + q;
        uint32_t at = first + rows[(size_t)d * nb + blockIdx.x];
        for (int w = 0; w < kSortWarps; ++w) { const uint32_t c = s_cnt[w][d]; s_cnt[w][d] = at; at += c; }
        first += tot[q];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if (base + k * 32 + lane >= n) continue;
        const uint32_t at = s_cnt[warp][(key[k] >> shift) & (kDigits - 1)] + rank[k];
        okeys[at] = key[k];
        ovals[at] = val[k];
    }
}

// ------------------------------------------------------------ primitives
__device__ __forceinline__ int f2ord(float f) { int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7fffffff; }
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
inline float host_ord2f(int i) { const int b = i >= 0 ? i : i ^ 0x7fffffff; float f; memcpy(&f, &b, 4); return f; }

__device__ __forceinline__ float3 ld3(const float* v, uint32_t i) { return mk(v[3 * (size_t)i], v[3 * (size_t)i + 1], v[3 * (size_t)i + 2]); }

__device__ __forceinline__ void tri_box(const float* verts, const uint32_t* idx, size_t i, float3* lo, float3* hi) {
    const float3 a = ld3(verts, idx[3 * i]), b = ld3(verts, idx[3 * i + 1]), d = ld3(verts, idx[3 * i + 2]);
    *lo = mk(fminf(fminf(a.x, b.x), d.x), fminf(fminf(a.y, b.y), d.y), fminf(fminf(a.z, b.z), d.z));
    *hi = mk(fmaxf(fmaxf(a.x, b.x), d.x), fmaxf(fmaxf(a.y, b.y), d.y), fmaxf(fmaxf(a.z, b.z), d.z));
}

// What the build keeps beside its arrays; read back by the host between its phases.
constexpr int kMaxLevels = 96;
struct BuildState {
    int gb[12];                   // ordered ints: centroid min, max, scene min, max
    uint32_t bad;                 // an index out of range
    int m[2];                     // cluster counts, ping-pong
    int node;                     // next node id
    int root, num_nodes;          // after the last merge
    int depth;                    // binary levels
    int front[kMaxLevels + 2];    // 4-wide nodes per level
};

__global__ void k_init_state(BuildState* st, int n) {
    const int t = threadIdx.x;
    if (t < 12) st->gb[t] = f2ord((t / 3) % 2 == 0 ? FLT_MAX : -FLT_MAX);
    if (t < kMaxLevels + 2) st->front[t] = t == 0 ? 1 : 0;
    if (t == 0) { st->bad = 0u; st->m[0] = n; st->m[1] = n; st->node = n; st->root = 0; st->num_nodes = 0; st->depth = 0; }
}

// Bounds of the boxes and of their centroids, and the check that every vertex index is below nvert
// (a triangle with a bad one is not read). A resident grid reduces per block before its twelve
// atomics: one set per warp of a thread-per-triangle grid took 456 us for 3.4 M triangles.
__global__ void __launch_bounds__(256) k_bounds(const float* __restrict__ verts, const uint32_t* __restrict__ idx, int n,
                                                uint32_t nvert, BuildState* st) {
    float v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = (k / 3) % 2 == 0 ? FLT_MAX : -FLT_MAX;
    uint32_t bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (idx[3 * (size_t)i] >= nvert || idx[3 * (size_t)i + 1] >= nvert || idx[3 * (size_t)i + 2] >= nvert) { bad = 1; continue; }
        float3 lo, hi;
        tri_box(verts, idx, i, &lo, &hi);
        const float3 c = (lo + hi) * 0.5f;
        const float a[12] = {c.x, c.y, c.z, c.x, c.y, c.z, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = (k / 3) % 2 == 0 ? fminf(v[k], a[k]) : fmaxf(v[k], a[k]);
    }
    __shared__ int s_v[12];
    __shared__ uint32_t s_bad;
    if (threadIdx.x < 12) s_v[threadIdx.x] = f2ord((threadIdx.x / 3) % 2 == 0 ? FLT_MAX : -FLT_MAX);
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        const bool mn = (k / 3) % 2 == 0;
        const int o = f2ord(v[k]);
        const int r = mn ? __reduce_min_sync(0xffffffffu, o) : __reduce_max_sync(0xffffffffu, o);
        if ((threadIdx.x & 31) == 0) { if (mn) atomicMin(&s_v[k], r); else atomicMax(&s_v[k], r); }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) s_bad = 1;
    __syncthreads();
    if (threadIdx.x < 12) {
        if ((threadIdx.x / 3) % 2 == 0) atomicMin(&st->gb[threadIdx.x], s_v[threadIdx.x]);
        else atomicMax(&st->gb[threadIdx.x], s_v[threadIdx.x]);
    }
    if (threadIdx.x == 0 && s_bad) atomicOr(&st->bad, 1u);
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__global__ void k_morton(const float* __restrict__ verts, const uint32_t* __restrict__ idx, int n,
                         const BuildState* __restrict__ st, uint32_t* keys, uint32_t* vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float lo[3], sc[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = ord2f(st->gb[k]);
        float ext = ord2f(st->gb[3 + k]) - lo[k];
        sc[k] = ext > 0.f ? 1023.f / ext : 0.f;
    }
    float3 blo, bhi;
    tri_box(verts, idx, i, &blo, &bhi);
    const float3 c = (blo + bhi) * 0.5f;
    uint32_t q[3];
    float cc[3] = {c.x, c.y, c.z};
    for (int k = 0; k < 3; ++k) {
        float f = (cc[k] - lo[k]) * sc[k];
        f = fminf(fmaxf(f, 0.f), 1023.f);
        q[k] = (uint32_t)f;
    }
    keys[i] = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
    vals[i] = (uint32_t)i;
}

__device__ __forceinline__ float half_area(float3 lo, float3 hi) {
    float3 d = hi - lo;
    return d.x * d.y + d.y * d.z + d.z * d.x;
}

// Outward padding: 2^-19 of the box's own magnitude, and at least 2^-20 of the
// scene's magnitude (covers the rounding of slab distances for rays whose
// origin lies anywhere inside the scene bounds).
__device__ __forceinline__ void pad_box(float& lo, float& hi, float floor_pad) {
    const float m = fmaxf(fmaxf(fabsf(lo), fabsf(hi)), hi - lo);
    const float p = fmaxf(m * 1.9073486e-6f, floor_pad) + 1e-30f;
    lo -= p;
    hi += p;
}

// ------------------------------------------------------------ nodes
// The tree under construction, by node id (the n leaves in Morton order, then the merges).
struct Tree {
    float4* lo;       // box, SAH cost
    float4* hi;       // box, triangles << 1 | collapsed (int bits)
    int* icount;      // interior nodes of the subtree that are not inside collapsed ones
    int2* child;
    // To the parent: (parent, what the depth-first index and the first triangle grow by on the way
    // down from it, whether it is collapsed). Parent -1 at the root.
    int4* up;
    // SAH-optimal grouping into 4-wide nodes: a dynamic program over the binary tree, bottom up
    // (the 8-wide form is in Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs
    // Through Compressed Wide BVHs", HPG 2017). The leaves are fixed, so groupings differ in SAH
    // cost only by the summed surface area of the 4-wide nodes. S(x, j) is the least such sum for
    // the subtree of binary node x when it may fill j of its parent's child slots (a leaf costs
    // nothing): S(x, 1) = A(x) + D(x, 4), and for j > 1 S(x, j) = min(S(x, 1), D(x, j)), with
    // D(x, j) = min over k in [1, j) of S(left, k) + S(right, j - k). dec(x, j) is the k that
    // reaches S(x, j), or 0 where x fills one slot; dec(x, 4) is the split of x's slots when x
    // roots a 4-wide node.
    float4* S;        // S(x, 1..4)
    uchar4* dec;      // dec(x, 1..4) (dec(x, 1) = 0)
};
struct Sah { int max_leaf; float ct, ci, floor_pad; };

struct Kid { float3 lo, hi; float cost; int cnt, icount; bool collapsed; float4 S; };

__device__ __forceinline__ Kid load_kid(const Tree& t, int x) {
    const float4 a = __ldcg(&t.lo[x]), b = __ldcg(&t.hi[x]);
    Kid k;
    k.lo = mk(a.x, a.y, a.z);
    k.hi = mk(b.x, b.y, b.z);
    k.cost = a.w;
    const int w = __float_as_int(b.w);
    k.cnt = w >> 1;
    k.collapsed = (w & 1) != 0;
    k.icount = __ldcg(&t.icount[x]);
    k.S = k.collapsed ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcg(&t.S[x]);
    return k;
}

__global__ void k_init_leaves(const uint32_t* __restrict__ sorted, int n, const float* __restrict__ verts,
                              const uint32_t* __restrict__ idx, Tree t, Sah sah, int* clusters) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float3 lo, hi;
    tri_box(verts, idx, sorted[k], &lo, &hi);
    t.lo[k] = make_float4(lo.x, lo.y, lo.z, sah.ci * half_area(lo, hi));
    t.hi[k] = make_float4(hi.x, hi.y, hi.z, __int_as_float((1 << 1) | 1));
    t.icount[k] = 0;
    clusters[k] = k;
}

// Makes node `x` the parent of clusters a and b, whose data are l and r: its box, SAH cost and
// collapse, and its row of the 4-wide grouping. Returns the new node's data.
__device__ __forceinline__ Kid merge_kids(const Tree& t, const Sah& sah, int x, int a, int b, const Kid& l, const Kid& r) {
    const float3 lo = mk(fminf(l.lo.x, r.lo.x), fminf(l.lo.y, r.lo.y), fminf(l.lo.z, r.lo.z));
    const float3 hi = mk(fmaxf(l.hi.x, r.hi.x), fmaxf(l.hi.y, r.hi.y), fmaxf(l.hi.z, r.hi.z));
    const float A = half_area(lo, hi);
    const int c = l.cnt + r.cnt;
    const float split = sah.ct * A + l.cost + r.cost;
    const float leaf = c <= sah.max_leaf ? sah.ci * A * (float)c : FLT_MAX;
    const bool collapsed = leaf <= split;
    t.lo[x] = make_float4(lo.x, lo.y, lo.z, collapsed ? leaf : split);
    t.hi[x] = make_float4(hi.x, hi.y, hi.z, __int_as_float((c << 1) | (collapsed ? 1 : 0)));
    t.icount[x] = collapsed ? 0 : 1 + l.icount + r.icount;
    t.child[x] = make_int2(a, b);
    t.up[a] = make_int4(x, 1, 0, collapsed ? 1 : 0);
    t.up[b] = make_int4(x, 1 + l.icount, l.cnt, collapsed ? 1 : 0);
    // the grouping's areas are of the padded child boxes' union, as the stored nodes have them
    float al[3] = {l.lo.x, l.lo.y, l.lo.z}, ah[3] = {l.hi.x, l.hi.y, l.hi.z};
    float bl[3] = {r.lo.x, r.lo.y, r.lo.z}, bh[3] = {r.hi.x, r.hi.y, r.hi.z};
    float d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        pad_box(al[k], ah[k], sah.floor_pad);
        pad_box(bl[k], bh[k], sah.floor_pad);
        d[k] = fmaxf(ah[k], bh[k]) - fminf(al[k], bl[k]);
    }
    const float sc[2][5] = {{0.f, l.S.x, l.S.y, l.S.z, l.S.w}, {0.f, r.S.x, r.S.y, r.S.z, r.S.w}};
    float D[5] = {0.f, 0.f, FLT_MAX, FLT_MAX, FLT_MAX};
    int kd[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 2; j <= 4; ++j)
#pragma unroll
        for (int k = 1; k < j; ++k) {
            const float cost = sc[0][k] + sc[1][j - k];
            if (cost < D[j]) { D[j] = cost; kd[j] = k; }
        }
    const float s1 = (d[0] * d[1] + d[1] * d[2] + d[2] * d[0]) + D[4];
    const bool one2 = s1 <= D[2], one3 = s1 <= D[3];      // s1 = A + D(x, 4) > D(x, 4)
    const float4 S = make_float4(s1, one2 ? s1 : D[2], one3 ? s1 : D[3], D[4]);
    t.S[x] = S;
    t.dec[x] = make_uchar4(0, (unsigned char)(one2 ? 0 : kd[2]), (unsigned char)(one3 ? 0 : kd[3]), (unsigned char)kd[4]);
    Kid k;
    k.lo = lo; k.hi = hi;
    k.cost = collapsed ? leaf : split;
    k.cnt = c;
    k.icount = collapsed ? 0 : 1 + l.icount + r.icount;
    k.collapsed = collapsed;
    k.S = collapsed ? make_float4(0.f, 0.f, 0.f, 0.f) : S;
    return k;
}
__device__ __forceinline__ void merge_node(const Tree& t, const Sah& sah, int x, int a, int b) {
    merge_kids(t, sah, x, a, b, load_kid(t, a), load_kid(t, b));
}

// ------------------------------------------------------------ PLOC
constexpr int kPlocThreads = 256;
constexpr int kPlocTile = 2 * kPlocThreads;
// Iterations between host reads of the count: as many as it takes to get to kFinish if each keeps
// kPlocKeep of the clusters, 16 at most (an even number, so that the count ends in m[0]).
// Iterations past that point cost two empty launches each (8 us), a further read of the count
// 20 us: of the 16 iterations that a fixed eight between reads took at 20,480 triangles, seven
// were empty.
constexpr double kPlocKeep = 0.78;
constexpr int kPlocBatch = 16;
constexpr int kMaxRadius = 32;
constexpr int kSuper = 64;         // tiles per partial sum of the compaction
constexpr int kFinish = 2048;      // from this many clusters on, one block does the rest

// The nearest neighbours of clusters i and i + 1 of m (either may lie outside [0, m)), whose boxes are
// at lo/hi[at] on: within r places, limited to [0, m). Strict order on unordered pairs: (area, min
// index, max index); j increases, so for equal area the first j seen has the smaller pair key.
// Every box of the joint window is read once.
__device__ __forceinline__ void nearest2(const float3* lo, const float3* hi, int at, int i, int m, int r, int (&nn)[2]) {
    const bool in0 = i >= 0 && i < m, in1 = i + 1 >= 0 && i + 1 < m;
    const float3 z = mk(0.f, 0.f, 0.f);
    const float3 lo0 = in0 ? lo[at] : z, hi0 = in0 ? hi[at] : z;
    const float3 lo1 = in1 ? lo[at + 1] : z, hi1 = in1 ? hi[at + 1] : z;
    float b0 = FLT_MAX, b1 = FLT_MAX;
    int n0 = -1, n1 = -1;
    const int j0 = max(0, i - r), j1 = min(m - 1, i + 1 + r);
    for (int j = j0; j <= j1; ++j) {
        const int k = at + (j - i);
        const float3 l = lo[k], h = hi[k];
        const float a0 = half_area(mk(fminf(lo0.x, l.x), fminf(lo0.y, l.y), fminf(lo0.z, l.z)),
                                   mk(fmaxf(hi0.x, h.x), fmaxf(hi0.y, h.y), fmaxf(hi0.z, h.z)));
        const float a1 = half_area(mk(fminf(lo1.x, l.x), fminf(lo1.y, l.y), fminf(lo1.z, l.z)),
                                   mk(fmaxf(hi1.x, h.x), fmaxf(hi1.y, h.y), fmaxf(hi1.z, h.z)));
        if (a0 < b0 && j != i && j <= i + r) { b0 = a0; n0 = j; }
        if (a1 < b1 && j != i + 1 && j >= i + 1 - r) { b1 = a1; n1 = j; }
    }
    nn[0] = in0 ? n0 : -1;
    nn[1] = in1 ? n1 : -1;
}

// One iteration's search and merges. A block owns kPlocTile - 2 r clusters and finds the
// neighbours of r more on either side, so that it can tell its own mutual pairs without another
// launch. Each thread searches for two adjacent clusters, whose windows share all but two boxes:
// the search is bound by the shared-memory reads of its 2 r boxes a cluster.
// out[i]: cluster i after the iteration, -1 if it was merged into its partner. Counts of
// kept clusters per tile and per kSuper tiles. From kFinish clusters on it only passes them on.
__global__ void __launch_bounds__(kPlocThreads) k_ploc_merge(const int* __restrict__ clusters, BuildState* st, int parity,
                                                             Tree t, Sah sah, int r, int* __restrict__ out,
                                                             uint32_t* __restrict__ cnt, uint32_t* super) {
    __shared__ float3 s_lo[kPlocTile + 2 * kMaxRadius], s_hi[kPlocTile + 2 * kMaxRadius];
    __shared__ int s_nn[kPlocTile];
    __shared__ uint32_t s_scan[33];
    __shared__ int s_base;
    const int m = st->m[parity];
    const int tile = kPlocTile - 2 * r, start = blockIdx.x * tile;
    if (start >= m) return;
    const int tid = threadIdx.x, g0 = start - r + 2 * tid;
    bool own[2], keep[2], merges[2] = {false, false};
    int id[2], j[2] = {-1, -1};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int k = 2 * tid + q, g = g0 + q;
        own[q] = k >= r && k < r + tile && g < m;
        keep[q] = own[q];
        id[q] = own[q] ? clusters[g] : -1;
    }
    if (m > kFinish) {
        for (int k = tid; k < kPlocTile + 2 * r; k += kPlocThreads) {
            const int q = start - 2 * r + k;
            if (q >= 0 && q < m) {
                const int c = clusters[q];
                const float4 a = t.lo[c], b = t.hi[c];
                s_lo[k] = mk(a.x, a.y, a.z);
                s_hi[k] = mk(b.x, b.y, b.z);
            }
        }
        __syncthreads();
        int nn[2] = {-1, -1};
        if (g0 + 1 >= 0 && g0 < m) nearest2(s_lo, s_hi, 2 * tid + r, g0, m, r, nn);
        s_nn[2 * tid] = nn[0];
        s_nn[2 * tid + 1] = nn[1];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!own[q]) continue;
            const int g = g0 + q;
            j[q] = nn[q];
            const bool mutual = j[q] >= 0 && s_nn[j[q] - (start - r)] == g;
            merges[q] = mutual && g < j[q];
            keep[q] = !mutual || merges[q];
        }
    }
    // both counts in one scan: merges in the low half, kept clusters in the high one
    uint32_t total;
    const uint32_t pre = block_excl_scan((uint32_t)(merges[0] + merges[1]) | ((uint32_t)(keep[0] + keep[1]) << 16), s_scan, &total);
    const int nmerge = (int)(total & 0xffffu);
    if (tid == 0) {
        s_base = nmerge ? atomicAdd(&st->node, nmerge) : 0;
        cnt[blockIdx.x] = total >> 16;
        atomicAdd(&super[blockIdx.x / kSuper], total >> 16);
    }
    __syncthreads();
    int x = s_base + (int)(pre & 0xffffu);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (!own[q]) continue;
        if (merges[q]) {
            merge_node(t, sah, x, id[q], clusters[j[q]]);
            id[q] = x++;
        }
        out[g0 + q] = keep[q] ? id[q] : -1;
    }
}

// Compacts the iteration's clusters in order (same tiles) and hands on their count; clears the
// partial sums of the next iteration.
__global__ void __launch_bounds__(kPlocThreads) k_ploc_compact(const int* __restrict__ in, BuildState* st, int parity, int r,
                                                               const uint32_t* __restrict__ cnt,
                                                               const uint32_t* __restrict__ super, uint32_t* next_super,
                                                               int* __restrict__ clusters) {
    __shared__ uint32_t s_scan[33];
    const int m = st->m[parity];
    const int tile = kPlocTile - 2 * r, start = blockIdx.x * tile;
    if (start >= m) return;
    const int tid = threadIdx.x, sb = blockIdx.x / kSuper;
    uint32_t before = 0, base, own;
    for (int k = tid; k < sb; k += kPlocThreads) before += super[k];
    for (int k = sb * kSuper + tid; k < (int)blockIdx.x; k += kPlocThreads) before += cnt[k];
    block_excl_scan(before, s_scan, &base);
    __syncthreads();
    int id[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) id[q] = 2 * tid + q < tile && start + 2 * tid + q < m ? in[start + 2 * tid + q] : -1;
    uint32_t at = base + block_excl_scan((uint32_t)(id[0] >= 0) + (uint32_t)(id[1] >= 0), s_scan, &own);
    if (id[0] >= 0) clusters[at++] = id[0];
    if (id[1] >= 0) clusters[at] = id[1];
    if (blockIdx.x % kSuper == 0 && tid == 0) next_super[sb] = 0u;
    if (tid == 0 && start + tile >= m) st->m[parity ^ 1] = (int)(base + own);
}

// The nearest neighbour of cluster i, its window dealt out to a group of `lanes` lanes (all of the
// warp take part), which all get the result: the smallest area, of equal ones the smallest j.
__device__ __forceinline__ int nearest_lanes(const float3* lo, const float3* hi, int i, int m, int r, int lanes, int q) {
    float best = FLT_MAX;
    int bj = -1;
    if (i < m) {
        const float3 mlo = lo[i], mhi = hi[i];
        const int j1 = min(m - 1, i + r);
        for (int j = max(0, i - r) + q; j <= j1; j += lanes) {
            if (j == i) continue;
            const float a = half_area(mk(fminf(mlo.x, lo[j].x), fminf(mlo.y, lo[j].y), fminf(mlo.z, lo[j].z)),
                                      mk(fmaxf(mhi.x, hi[j].x), fmaxf(mhi.y, hi[j].y), fmaxf(mhi.z, hi[j].z)));
            if (a < best) { best = a; bj = j; }
        }
    }
    for (int o = lanes >> 1; o; o >>= 1) {
        const float a = __shfl_xor_sync(0xffffffffu, best, o);
        const int j = __shfl_xor_sync(0xffffffffu, bj, o);
        if (a < best || (a == best && (uint32_t)j < (uint32_t)bj)) { best = a; bj = j; }
    }
    return bj;
}

// The clusters of the last iterations, in shared memory. Order, boxes and slots move every
// iteration; what only a merge reads stays in a slot, and the parent takes the slot of its first child.
struct FinishMem {
    float3 lo[kFinish], hi[kFinish];
    int slot[kFinish], nn[kFinish];
    int2 merge[kFinish / 2];                        // slots of the iteration's pairs
    float3 klo[kFinish], khi[kFinish];
    float4 S[kFinish];
    float cost[kFinish];
    int id[kFinish], cnt[kFinish], icount[kFinish];   // cnt: as in Tree::hi, with the collapse bit
    __device__ __forceinline__ Kid get(int k) const {
        Kid r;
        r.lo = klo[k]; r.hi = khi[k]; r.cost = cost[k];
        r.cnt = cnt[k] >> 1; r.collapsed = (cnt[k] & 1) != 0;
        r.icount = icount[k]; r.S = S[k];
        return r;
    }
    __device__ __forceinline__ void put(int k, int id_, const Kid& r) {
        id[k] = id_;
        klo[k] = r.lo; khi[k] = r.hi; cost[k] = r.cost;
        cnt[k] = (r.cnt << 1) | (r.collapsed ? 1 : 0);
        icount[k] = r.icount; S[k] = r.S;
    }
};

// All remaining iterations in one block, whatever a merge reads in shared memory. Then the root:
// never a leaf (a tree has at least one interior node). Some thirty iterations, bound by the
// search while there are many clusters and by their chain of barriers after that: few clusters
// share the block's threads for their search; the pairs are put in a list, so that full warps
// merge them, beside the next iteration's search, which needs the boxes alone; warps without a
// cluster go from barrier to barrier. A thread per cluster that merges where it stands, its nodes in
// global memory: 179 us from 2048 clusters; nodes in shared memory and shared searches 131; the
// list 115; now 105 (at 59% of the SM's issue slots).
__global__ void __launch_bounds__(1024) k_ploc_finish(const int* __restrict__ clusters, BuildState* st, int parity, Tree t,
                                                      Sah sah, int r) {
    extern __shared__ __align__(16) char s_mem[];
    FinishMem& c = *reinterpret_cast<FinishMem*>(s_mem);
    __shared__ uint32_t s_scan[32];
    int m = st->m[parity];
    if (m > kFinish) return;
    const int tid = threadIdx.x;
    int node = st->node, nmerge = 0;
    for (int k = tid; k < m; k += 1024) {
        const int x = clusters[k];
        const Kid kid = load_kid(t, x);
        c.put(k, x, kid);
        c.lo[k] = kid.lo; c.hi[k] = kid.hi;
        c.slot[k] = k;
    }
    __syncthreads();
    // the merges of the iteration before, from the last thread on (the first ones search)
    auto merge_pairs = [&]() {
        const int q = 1023 - tid;                    // at most kFinish / 2 = 1024 pairs
        if (q >= nmerge) return;
        const int2 e = c.merge[q];
        const int x = node - nmerge + q;
        const Kid kid = merge_kids(t, sah, x, c.id[e.x], c.id[e.y], c.get(e.x), c.get(e.y));
        c.put(e.x, x, kid);
    };
    while (m > 1) {
        merge_pairs();
        if (m > 1024) {
            int nn[2] = {-1, -1};
            if (2 * tid < m) nearest2(c.lo, c.hi, 2 * tid, 2 * tid, m, r, nn);
            if (2 * tid < m) c.nn[2 * tid] = nn[0];
            if (2 * tid + 1 < m) c.nn[2 * tid + 1] = nn[1];
        } else {
            int shift = 0;
            while (shift < 3 && (m << (shift + 1)) <= 1024) ++shift;
            const int i = tid >> shift, q = tid & ((1 << shift) - 1);
            if ((tid & ~31) >> shift < m) {          // the warp has a cluster
                const int nn = nearest_lanes(c.lo, c.hi, i, m, r, 1 << shift, q);
                if (i < m && q == 0) c.nn[i] = nn;
            }
        }
        __syncthreads();
        // thread t has clusters 2 t and 2 t + 1, so that ranks follow the order
        int j[2];
        bool keep[2] = {false, false}, mer[2] = {false, false};
        const bool busy = 2 * (tid & ~31) < m;       // the warp has any
        uint32_t own = 0, incl = 0;                  // merges in the low half, kept clusters in the high one
        if (busy) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int k = 2 * tid + q;
                j[q] = k < m ? c.nn[k] : -1;
                const bool mutual = j[q] >= 0 && c.nn[j[q]] == k;
                mer[q] = mutual && k < j[q];
                keep[q] = k < m && (!mutual || mer[q]);
            }
            own = (mer[0] + mer[1]) | ((uint32_t)(keep[0] + keep[1]) << 16);
            incl = warp_incl_scan(own);
        }
        if ((tid & 31) == 31) s_scan[tid >> 5] = incl;
        __syncthreads();
        // every warp adds up the warps before its own
        const uint32_t w = s_scan[tid & 31];
        const uint32_t total = __reduce_add_sync(0xffffffffu, w);
        uint32_t pre = 0;
        if (busy) pre = __reduce_add_sync(0xffffffffu, (tid & 31) < tid >> 5 ? w : 0u) + incl - own;
        nmerge = (int)(total & 0xffffu);
        if (nmerge == 0) break;                      // no progress: the host reports it
        int mr = (int)(pre & 0xffffu), kr = (int)(pre >> 16);
        int slot[2];
        float3 lo[2], hi[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int k = 2 * tid + q;
            if (!keep[q]) continue;
            lo[q] = c.lo[k];
            hi[q] = c.hi[k];
            slot[q] = c.slot[k];
            if (!mer[q]) continue;
            const float3 l = c.lo[j[q]], h = c.hi[j[q]];
            lo[q] = mk(fminf(lo[q].x, l.x), fminf(lo[q].y, l.y), fminf(lo[q].z, l.z));
            hi[q] = mk(fmaxf(hi[q].x, h.x), fmaxf(hi[q].y, h.y), fmaxf(hi[q].z, h.z));
            c.merge[mr++] = make_int2(slot[q], c.slot[j[q]]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!keep[q]) continue;
            c.lo[kr] = lo[q];
            c.hi[kr] = hi[q];
            c.slot[kr++] = slot[q];
        }
        node += nmerge;
        m = (int)(total >> 16);
        __syncthreads();
    }
    merge_pairs();
    __syncthreads();
    if (tid != 0) return;
    st->node = node;
    st->m[0] = st->m[1] = m;
    if (m != 1) return;
    const int root = c.id[c.slot[0]];
    const int2 ch = t.child[root];
    const int n = 1 + t.icount[ch.x] + t.icount[ch.y];   // as if the root were not collapsed
    t.up[root] = make_int4(-1, 0, 0, 0);
    t.up[ch.x].w = 0;
    t.up[ch.y].w = 0;
    st->root = root;
    st->num_nodes = n;
}

// ------------------------------------------------------------ layout
__global__ void k_layout_tris(int n, Tree t, const uint32_t* __restrict__ sorted, const float* __restrict__ verts,
                              const uint32_t* __restrict__ idx, BvhTri* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int pos = 0;
    for (int x = k; x >= 0;) {
        const int4 u = __ldg(&t.up[x]);
        pos += u.z;
        x = u.x;
    }
    const uint32_t prim = sorted[k];
    float3 a = ld3(verts, idx[3 * (size_t)prim]), b = ld3(verts, idx[3 * (size_t)prim + 1]), c = ld3(verts, idx[3 * (size_t)prim + 2]);
    float3 e1 = xsub(b, a), e2 = xsub(c, a);
    BvhTri tr;
    tr.p1 = make_float4(a.x, a.y, a.z, __int_as_float((int)prim));
    tr.e1 = make_float4(e1.x, e1.y, e1.z, 0.f);
    tr.e2 = make_float4(e2.x, e2.y, e2.z, 0.f);
    out[pos] = tr;
}

// dec: the 4-wide grouping's decisions, by depth-first index
__global__ void k_layout_nodes(int n, int total, Tree t, float floor_pad, BuildState* st, BvhNode* __restrict__ out,
                               uchar4* __restrict__ dec) {
    const int x = n + blockIdx.x * blockDim.x + threadIdx.x;
    int depth = 0;
    bool live = x < total && (x == st->root || !(__float_as_int(t.hi[x].w) & 1));
    if (live) {
        int idx = 0, start = 0;
        depth = 1;
        for (int4 u = __ldg(&t.up[x]); u.x >= 0; u = __ldg(&t.up[u.x])) {
            if (u.w) { live = false; depth = 0; break; }      // inside a collapsed leaf subtree
            idx += u.y;
            start += u.z;
            ++depth;
        }
        if (live) {
            const int2 ch = t.child[x];
            const int c[2] = {ch.x, ch.y};
            const int lw = __float_as_int(t.hi[ch.x].w);
            const int cidx[2] = {idx + 1, idx + 1 + t.icount[ch.x]};
            const int cstart[2] = {start, start + (lw >> 1)};
            int ref[2], cnt[2];
            float blo[2][3], bhi[2][3];
            for (int k = 0; k < 2; ++k) {
                const float4 a = t.lo[c[k]], b = t.hi[c[k]];
                const int w = __float_as_int(b.w);
                if (w & 1) { ref[k] = ~((cstart[k] << 5) | (w >> 1)); cnt[k] = w >> 1; }
                else { ref[k] = cidx[k]; cnt[k] = 0; }
                blo[k][0] = a.x; blo[k][1] = a.y; blo[k][2] = a.z;
                bhi[k][0] = b.x; bhi[k][1] = b.y; bhi[k][2] = b.z;
                for (int d = 0; d < 3; ++d) pad_box(blo[k][d], bhi[k][d], floor_pad);
            }
            BvhNode nd;
            nd.a = make_float4(blo[0][0], bhi[0][0], blo[0][1], bhi[0][1]);
            nd.b = make_float4(blo[1][0], bhi[1][0], blo[1][1], bhi[1][1]);
            nd.c = make_float4(blo[0][2], bhi[0][2], blo[1][2], bhi[1][2]);
            nd.d = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), __int_as_float(cnt[0]), __int_as_float(cnt[1]));
            out[idx] = nd;
            dec[idx] = t.dec[x];
        }
    }
    depth = __reduce_max_sync(0xffffffffu, depth);
    if ((threadIdx.x & 31) == 0 && depth > *(volatile int*)&st->depth) atomicMax(&st->depth, depth);
}

// single triangle: one node with a leaf child and an empty child
__global__ void k_single(const float* verts, const uint32_t* idx, BvhNode* nodes, BvhTri* tris,
                         uchar4* dec, BuildState* st) {
    float3 a = ld3(verts, idx[0]), b = ld3(verts, idx[1]), c = ld3(verts, idx[2]);
    float lo[3] = {fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z)};
    float hi[3] = {fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z)};
    for (int d = 0; d < 3; ++d) pad_box(lo[d], hi[d], 0.f);
    BvhNode nd;
    nd.a = make_float4(lo[0], hi[0], lo[1], hi[1]);
    nd.b = make_float4(FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX);
    nd.c = make_float4(lo[2], hi[2], FLT_MAX, -FLT_MAX);
    nd.d = make_float4(__int_as_float(~1), __int_as_float(~0), __int_as_float(1), __int_as_float(0));
    nodes[0] = nd;
    dec[0] = make_uchar4(0, 1, 1, 1);   // two leaves
    st->depth = 1;
    st->num_nodes = 1;
    float3 e1 = xsub(b, a), e2 = xsub(c, a);
    tris[0].p1 = make_float4(a.x, a.y, a.z, __int_as_float(0));
    tris[0].e1 = make_float4(e1.x, e1.y, e1.z, 0.f);
    tris[0].e2 = make_float4(e2.x, e2.y, e2.z, 0.f);
}

// ------------------------------------------------------------ 4-wide tree
__device__ __forceinline__ void child_of(const BvhNode& nd, int k, float lo[3], float hi[3], int* ref) {
    if (k == 0) {
        lo[0] = nd.a.x; hi[0] = nd.a.y; lo[1] = nd.a.z; hi[1] = nd.a.w; lo[2] = nd.c.x; hi[2] = nd.c.y;
        *ref = __float_as_int(nd.d.x);
    } else {
        lo[0] = nd.b.x; hi[0] = nd.b.y; lo[1] = nd.b.z; hi[1] = nd.b.w; lo[2] = nd.c.z; hi[2] = nd.c.w;
        *ref = __float_as_int(nd.d.y);
    }
}

__device__ __forceinline__ int dec_for(uchar4 v, int j) { return j == 2 ? v.y : j == 3 ? v.z : j == 4 ? v.w : 0; }

// One level of the collapse by the program's decisions: the node's four slots are split
// between its binary children by dec(x, 4), and a child given j > 1 slots is opened while
// dec(child, j) says so. Slots always add up to four, so a node gets at most four children.
// front: the level's binary nodes, whose 4-wide nodes are first + 0, 1, ...; interior children
// get the next indices in the order their warps arrive (one add a warp) and form the next level.
__device__ __forceinline__ void collapse_level(const BvhNode* __restrict__ n2, const uchar4* __restrict__ dec,
                                               const int* front, int m, int first, int* children,
                                               BvhNode4* __restrict__ out, int* next, int cap) {
    const int child0 = first + m;
    const int lane = threadIdx.x & 31;
    for (int b = blockIdx.x * blockDim.x; b < m; b += gridDim.x * blockDim.x) {
        const int i = b + threadIdx.x;
        const bool valid = i < m;
        float lo[4][3], hi[4][3];
        int ref[4] = {~0, ~0, ~0, ~0}, bud[4], n = 0, interior = 0;
        if (valid) {
            const int x = __ldcg(&front[i]);
            n = 2;
            {
                const BvhNode nd = n2[x];
                child_of(nd, 0, lo[0], hi[0], &ref[0]);
                child_of(nd, 1, lo[1], hi[1], &ref[1]);
                const int k = dec[x].w;
                bud[0] = k;
                bud[1] = 4 - k;
            }
            while (n < 4) {
                int e = -1, dd = 0;
                for (int q = 0; q < n && e < 0; ++q) {
                    if (ref[q] < 0 || bud[q] < 2) continue;
                    const int v = dec_for(dec[ref[q]], bud[q]);
                    if (v > 0) { e = q; dd = v; }
                }
                if (e < 0) break;
                const BvhNode c = n2[ref[e]];
                child_of(c, 1, lo[n], hi[n], &ref[n]);
                bud[n] = bud[e] - dd;
                child_of(c, 0, lo[e], hi[e], &ref[e]);
                bud[e] = dd;
                ++n;
            }
            for (int k = 0; k < n; ++k) interior += ref[k] >= 0 ? 1 : 0;
        }
        const uint32_t incl = warp_incl_scan((uint32_t)interior);
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        int base = 0;
        if (lane == 0 && all) base = atomicAdd(children, (int)all);
        base = __shfl_sync(0xffffffffu, base, 0) + (int)incl - interior;
        if (!valid) continue;
        float v[6][4];
        int r[4];
        for (int k = 0; k < 4; ++k) {
            if (k >= n) {
                for (int d = 0; d < 6; ++d) v[d][k] = __int_as_float(0x7f800000);   // +inf: never entered
                r[k] = ~0;
                continue;
            }
            v[0][k] = lo[k][0]; v[1][k] = hi[k][0]; v[2][k] = lo[k][1];
            v[3][k] = hi[k][1]; v[4][k] = lo[k][2]; v[5][k] = hi[k][2];
            r[k] = ref[k];
            if (ref[k] >= 0) {
                if (base < cap) next[base] = ref[k];
                r[k] = child0 + base;
                ++base;
            }
        }
        if (first + i >= cap) continue;
        BvhNode4 o;
        o.lox = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
        o.hix = make_float4(v[1][0], v[1][1], v[1][2], v[1][3]);
        o.loy = make_float4(v[2][0], v[2][1], v[2][2], v[2][3]);
        o.hiy = make_float4(v[3][0], v[3][1], v[3][2], v[3][3]);
        o.loz = make_float4(v[4][0], v[4][1], v[4][2], v[4][3]);
        o.hiz = make_float4(v[5][0], v[5][1], v[5][2], v[5][3]);
        o.ref = make_int4(r[0], r[1], r[2], r[3]);
        o.pad = make_int4(0, 0, 0, 0);
        out[first + i] = o;
    }
}

__global__ void __launch_bounds__(256) k_collapse4_dp(const BvhNode* __restrict__ n2, const uchar4* __restrict__ dec,
                                                      const int* front, BuildState* st, int level,
                                                      BvhNode4* __restrict__ out, int* next, int cap) {
    int first = 0;
    for (int k = 0; k < level; ++k) first += st->front[k];
    collapse_level(n2, dec, front, st->front[level], first, &st->front[level + 1], out, next, cap);
}

// All levels in one block, for trees whose levels are no more than a few nodes a thread: a level is
// one chain of fetches either way, and a launch for each adds its start and a sum over the counts.
// Whole builds, a launch per level / one block: 38 binary nodes 197 / 170 us, 700 nodes 266 / 240,
// 2,810 nodes 370 / 330, 11,212 nodes 486 / 482, 44,909 nodes 602 / 790.
constexpr int kCollapseBlock = 3 << 12;
__global__ void __launch_bounds__(1024) k_collapse4_block(const BvhNode* __restrict__ n2, const uchar4* __restrict__ dec,
                                                          int* fa, int* fb, BuildState* st, BvhNode4* __restrict__ out,
                                                          int cap) {
    __shared__ int s_count[2];
    if (threadIdx.x == 0) s_count[0] = 0;
    __syncthreads();
    int first = 0, m = 1;
    for (int level = 0; level < kMaxLevels && m > 0; ++level) {
        int* const front = level & 1 ? fb : fa;
        int* const next = level & 1 ? fa : fb;
        if (threadIdx.x == 0) s_count[(level & 1) ^ 1] = 0;      // the next level's
        collapse_level(n2, dec, front, m, first, &s_count[level & 1], out, next, cap);
        __syncthreads();
        first += m;
        m = s_count[level & 1];
        if (threadIdx.x == 0) st->front[level + 1] = m;
        __syncthreads();
    }
}

// One axis of a node's quantised boxes. The decoded plane of byte q is p + s (1 + q 2^-15) in
// exact arithmetic; planes are rounded outward with a margin of 1/64 cell for the traversal's
// rounding (2^-8 cell at most). The cell grows until every plane fits.
__device__ void quantise_axis(const float (&lo)[4], const float (&hi)[4], const bool (&used)[4], float* p_out,
                              float* s_out, uint32_t* qlo, uint32_t* qhi) {
    double mn = 1e300, mx = -1e300;
    for (int k = 0; k < 4; ++k)
        if (used[k]) { mn = fmin(mn, (double)lo[k]); mx = fmax(mx, (double)hi[k]); }
    double cell = fmax((mx - mn) / 250.0, 1e-30);
    float p = 0.f, s = 0.f;
    int l[4], h[4];
    for (int it = 0; it < 64; ++it) {
        s = (float)(cell * 32768.0);
        p = (float)(mn - (double)s - 2.0 * cell);
        bool ok = true;
        for (int k = 0; k < 4; ++k) {
            if (!used[k]) { l[k] = 255; h[k] = 0; continue; }
            const double a = floor((((double)lo[k] - p) / s - 1.0) * 32768.0 - 1.0 / 64.0);
            const double b = ceil((((double)hi[k] - p) / s - 1.0) * 32768.0 + 1.0 / 64.0);
            ok = ok && a >= 0.0 && b <= 255.0;
            l[k] = (int)fmin(fmax(a, 0.0), 255.0);
            h[k] = (int)fmin(fmax(b, 0.0), 255.0);
        }
        if (ok) break;
        cell *= 1.25;
    }
    *p_out = p;
    *s_out = s;
    *qlo = *qhi = 0u;
    for (int k = 0; k < 4; ++k) { *qlo |= (uint32_t)l[k] << (8 * k); *qhi |= (uint32_t)h[k] << (8 * k); }
}

__global__ void k_quantise4(const BvhNode4* __restrict__ in, int n, BvhNode4Q* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const BvhNode4 nd = in[i];
    const int r[4] = {nd.ref.x, nd.ref.y, nd.ref.z, nd.ref.w};
    const float lx[4] = {nd.lox.x, nd.lox.y, nd.lox.z, nd.lox.w}, hx[4] = {nd.hix.x, nd.hix.y, nd.hix.z, nd.hix.w};
    const float ly[4] = {nd.loy.x, nd.loy.y, nd.loy.z, nd.loy.w}, hy[4] = {nd.hiy.x, nd.hiy.y, nd.hiy.z, nd.hiy.w};
    const float lz[4] = {nd.loz.x, nd.loz.y, nd.loz.z, nd.loz.w}, hz[4] = {nd.hiz.x, nd.hiz.y, nd.hiz.z, nd.hiz.w};
    bool used[4];
    for (int k = 0; k < 4; ++k) used[k] = r[k] != ~0 && lx[k] <= hx[k] && ly[k] <= hy[k] && lz[k] <= hz[k];
    BvhNode4Q q;
    quantise_axis(lx, hx, used, &q.p[0], &q.s[0], &q.lox, &q.hix);
    quantise_axis(ly, hy, used, &q.p[1], &q.s[1], &q.loy, &q.hiy);
    quantise_axis(lz, hz, used, &q.p[2], &q.s[2], &q.loz, &q.hiz);
    for (int k = 0; k < 4; ++k) q.ref[k] = r[k];
    out[i] = q;
}


// Scratch of one build: one allocation, cut into arrays.
struct Arena {
    char* base = nullptr;
    size_t used = 0;
    template <typename T> T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base + used);
        used += (sizeof(T) * (n ? n : 1) + 255) & ~(size_t)255;
        return p;
    }
};

struct Scratch {
    BuildState* st;
    uint32_t *keys, *vals, *keys2, *vals2, *hist, *dsum;
    Tree t;
    int *ca, *cb, *out;
    uint32_t *cnt, *super[2];
    uchar4* dec;
    int *fa, *fb;
    void cut(Arena& a, size_t n, int tile) {
        const size_t total = 2 * n, nb = (n + sort_tile(n) - 1) / sort_tile(n), tiles = (n + tile - 1) / tile;
        st = a.take<BuildState>(1);
        keys = a.take<uint32_t>(n); vals = a.take<uint32_t>(n);
        keys2 = a.take<uint32_t>(n); vals2 = a.take<uint32_t>(n);
        hist = a.take<uint32_t>(kDigits * nb); dsum = a.take<uint32_t>(kDigits);
        t.lo = a.take<float4>(total); t.hi = a.take<float4>(total); t.icount = a.take<int>(total);
        t.child = a.take<int2>(total); t.up = a.take<int4>(total);
        t.S = a.take<float4>(total); t.dec = a.take<uchar4>(total);
        ca = a.take<int>(n); cb = a.take<int>(n); out = a.take<int>(n);
        cnt = a.take<uint32_t>(tiles);
        for (uint32_t*& s : super) s = a.take<uint32_t>(tiles / kSuper + 1);
        dec = a.take<uchar4>(n);
        fa = a.take<int>(n); fb = a.take<int>(n);
    }
};

cudaError_t read_state(BuildState* host, const BuildState* st, cudaStream_t s) {
    cudaError_t e = cudaMemcpyAsync(host, st, sizeof(BuildState), cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

cudaError_t build_with(Scratch& w, const float* verts, const uint32_t* idx, int n, uint32_t nvert,
                       const BvhBuildOptions& opt, DeviceBvh* out, bool* in_range, cudaStream_t s) {
    const int T = 256;
    BuildState h;
    int sms = 148;
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    k_init_state<<<1, 128, 0, s>>>(w.st, n);
    k_bounds<<<std::min(div_up(n, T), sms * 8), T, 0, s>>>(verts, idx, n, nvert, w.st);
    CK(cudaGetLastError());
    CK(read_state(&h, w.st, s));
    *in_range = h.bad == 0;
    if (h.bad) return cudaSuccess;
    // scene bounds for the caller and the scene-relative box padding
    float scale = 0.f;
    for (int k = 0; k < 3; ++k) {
        out->lo[k] = host_ord2f(h.gb[6 + k]);
        out->hi[k] = host_ord2f(h.gb[9 + k]);
        scale = fmaxf(scale, fmaxf(fabsf(out->lo[k]), fabsf(out->hi[k])));
    }
    const Sah sah{opt.max_leaf < 1 ? 1 : opt.max_leaf, opt.cost_traverse, opt.cost_intersect, scale * 9.5367432e-7f};
    CK(dalloc(&out->tris, n, s));
    if (n == 1) {
        CK(dalloc(&out->nodes, 1, s));
        k_single<<<1, 1, 0, s>>>(verts, idx, out->nodes, out->tris, w.dec, w.st);
        out->num_nodes = 1;
    } else {
        k_morton<<<div_up(n, T), T, 0, s>>>(verts, idx, n, w.st, w.keys, w.vals);
        const int nb = div_up(n, sort_tile(n));
        for (int shift = 0; shift < 30; shift += 10) {
            const bool small = n <= kSmallSort;
            auto hist = small ? k_sort_hist<4> : k_sort_hist<16>;
            auto scatter = small ? k_sort_scatter<4> : k_sort_scatter<16>;
            hist<<<nb, kSortThreads, 0, s>>>(w.keys, n, shift, w.hist, nb);
            k_sort_rows<<<kDigits / 8, 256, 0, s>>>(w.hist, nb, w.dsum);
            scatter<<<nb, kSortThreads, 0, s>>>(w.keys, w.vals, w.keys2, w.vals2, n, shift, w.hist, w.dsum, nb);
            std::swap(w.keys, w.keys2);
            std::swap(w.vals, w.vals2);
        }
        k_init_leaves<<<div_up(n, T), T, 0, s>>>(w.vals, n, verts, idx, w.t, sah, w.ca);
        CK(cudaGetLastError());
        const int r = opt.ploc_radius < 1 ? 1 : (opt.ploc_radius > kMaxRadius ? kMaxRadius : opt.ploc_radius);
        const int tile = kPlocTile - 2 * r;
        const size_t smem = sizeof(FinishMem);
        CK(cudaFuncSetAttribute(k_ploc_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        for (int m = n; ;) {
            if (m > kFinish) {
                const int tiles = div_up(m, tile);
                CK(cudaMemsetAsync(w.super[0], 0, sizeof(uint32_t) * (tiles / kSuper + 1), s));
                const int its = std::min(kPlocBatch, ((int)std::ceil(std::log((double)m / kFinish) / -std::log(kPlocKeep)) + 1) & ~1);
                for (int it = 0; it < its; ++it) {
                    k_ploc_merge<<<tiles, kPlocThreads, 0, s>>>(w.ca, w.st, it & 1, w.t, sah, r, w.out, w.cnt, w.super[it & 1]);
                    k_ploc_compact<<<tiles, kPlocThreads, 0, s>>>(w.out, w.st, it & 1, r, w.cnt, w.super[it & 1],
                                                                  w.super[(it & 1) ^ 1], w.cb);
                    std::swap(w.ca, w.cb);
                }
            }
            k_ploc_finish<<<1, 1024, smem, s>>>(w.ca, w.st, 0, w.t, sah, r);
            CK(cudaGetLastError());
            CK(read_state(&h, w.st, s));
            if (h.m[0] == 1) break;
            // no progress: impossible with the strict pair order, unless areas are not finite
            if (h.m[0] < 1 || h.m[0] >= m || h.m[0] <= kFinish) return cudaErrorUnknown;
            m = h.m[0];
        }
        out->num_nodes = h.num_nodes;
        CK(dalloc(&out->nodes, h.num_nodes, s));
        k_layout_tris<<<div_up(n, T), T, 0, s>>>(n, w.t, w.vals, verts, idx, out->tris);
        k_layout_nodes<<<div_up(n - 1, T), T, 0, s>>>(n, 2 * n - 1, w.t, sah.floor_pad, w.st, out->nodes, w.dec);
    }
    CK(cudaGetLastError());
    // the 4-wide form, level by level
    const int cap = out->num_nodes;             // it has at most as many nodes as the binary tree
    CK(dalloc(&out->nodes4, cap, s));
    // every 4-wide node must start on a 128-byte line (the traversals read it in 32-byte and
    // 16-byte vector loads): the allocator's alignment, checked rather than assumed
    if ((uintptr_t)out->nodes4 % sizeof(BvhNode4) != 0) return cudaErrorMisalignedAddress;
    CK(cudaMemsetAsync(w.fa, 0, sizeof(int), s));   // the root
    // levels between host reads: as many as a balanced tree has, and a few more
    int levels = 6;
    for (long long c = 1; c < cap; c *= 3) ++levels;
    bool done = false;
    if (cap <= kCollapseBlock) {
        k_collapse4_block<<<1, 1024, 0, s>>>(out->nodes, w.dec, w.fa, w.fb, w.st, out->nodes4, cap);
        CK(cudaGetLastError());
        CK(read_state(&h, w.st, s));
        done = h.front[kMaxLevels] == 0;
    } else for (int level = 0; level < kMaxLevels && !done;) {
        for (int k = 0; k < levels && level < kMaxLevels; ++k, ++level) {
            const long long bound = level < 12 ? std::min<long long>(cap, 1ll << (2 * level)) : cap;
            k_collapse4_dp<<<std::min(div_up(bound, T), sms * 8), T, 0, s>>>(out->nodes, w.dec, w.fa, w.st, level, out->nodes4,
                                                                            w.fb, cap);
            std::swap(w.fa, w.fb);
        }
        CK(cudaGetLastError());
        CK(read_state(&h, w.st, s));
        done = h.front[level] == 0;
    }
    out->depth = h.depth;
    int nodes4 = 0, depth4 = 0;
    for (int k = 0; k < kMaxLevels && h.front[k] > 0; ++k) { nodes4 += h.front[k]; ++depth4; }
    if (!done) {                      // deeper than any stack holds: the binary tree only
        cudaFreeAsync(out->nodes4, s);
        out->nodes4 = nullptr;
        return cudaSuccess;
    }
    if (nodes4 > cap) return cudaErrorUnknown;
    out->num_nodes4 = nodes4;
    out->depth4 = depth4;
    CK(dalloc(&out->nodes4q, nodes4, s));
    k_quantise4<<<div_up(nodes4, 128), 128, 0, s>>>(out->nodes4, nodes4, out->nodes4q);
    return cudaGetLastError();
}

}  // namespace

cudaError_t bvh_build_device(const float* verts, const uint32_t* idx, int n, uint32_t nvert, const BvhBuildOptions& opt,
                             DeviceBvh* out, bool* in_range, cudaStream_t s) {
    *in_range = true;
    if (n < 1) return cudaErrorInvalidValue;
    *out = DeviceBvh();
    out->num_tris = n;
    const int tile = kPlocTile - 2 * kMaxRadius;      // the smallest tile
    Arena a;
    Scratch w;
    w.cut(a, n, tile);                                // sizes
    const size_t bytes = a.used;
    CK(cudaMallocAsync((void**)&a.base, bytes, s));
    a.used = 0;
    w.cut(a, n, tile);
    const cudaError_t e = build_with(w, verts, idx, n, nvert, opt, out, in_range, s);
    cudaFreeAsync(a.base, s);
    return e;
}

void bvh_free_device(DeviceBvh* bvh, cudaStream_t s) {
    if (bvh->nodes) cudaFreeAsync(bvh->nodes, s);
    if (bvh->tris) cudaFreeAsync(bvh->tris, s);
    if (bvh->nodes4) cudaFreeAsync(bvh->nodes4, s);
    if (bvh->nodes4q) cudaFreeAsync(bvh->nodes4q, s);
    *bvh = DeviceBvh();
}

}  // namespace aur
