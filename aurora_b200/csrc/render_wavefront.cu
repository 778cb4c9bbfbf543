// render_wavefront.cu — the batched (wavefront) renderer.
//
// Same estimator as Integrator::integrateCameraSample (Aurora/src/frontend/
// integrator.cpp:152-300) and the plain kernel, reorganised for the GPU:
// a pool of P path slots lives in HBM (structure of arrays) and every
// iteration runs one bounce of every live path as separate stages:
//
//   regen   the slots that the shading stage left work for: next-event radiance is added,
//           finished slots write their sample and take the next work item (scene, pixel, sample)
//           from a global counter -> camera ray
//   extend  closest hit for the extension queue (persistent warps, traversal only)
//   sort    optional: counting sort of the hits by material type
//   shade   emission, lobe choice, next-event rays + their contributions, BRDF
//           continuation, throughput and roulette -> next extension queue
//   shadow  occlusion for the next-event rays
//
// Queue appends and work fetches are aggregated per block (one atomic per block). Many scenes of
// different resolution, spp and depth share one pool (batched launch). The
// per-iteration kernels are captured once into a CUDA graph and replayed.
// Every (pixel, sample) result goes to a per-sample buffer and is resolved in
// sample order with the plain kernel's compensated sum, so both renderers
// produce the same film for the same seed.
#include "aur_capi_internal.h"
#include "aur_adjoint.cuh"
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <type_traits>

namespace aur {
namespace {

// What regen has to do for a slot, alone or above the slot's number (below 2^26).
constexpr uint32_t kPending = 1u << 31;   // next-event rays in flight: their radiance is to be added
constexpr uint32_t kDone = 1u << 30;      // the path is finished: write its sample, take new work
constexpr uint32_t kNoRec = 0xffffffffu;  // WfPool::rec_cur of a vertex without a parameter
// lane refill: a warp takes new rays once this many lanes are idle, and runs kRounds
// traversal rounds (interior phase + leaf phase) between refill checks
// (swept on the quantised 4-wide tree, 1080p terrain frame, closest + any hit: rounds 3 / 4 / 5 at
// 16 idle lanes 142.6 / 141.0 / 141.0 ms; 12 / 16 / 20 idle lanes at 4 rounds 140.1 / 141.0 / 143.8)
constexpr int kRefill = 12;
constexpr int kRounds = 4;
// resident 256-thread blocks per SM the traversal kernels are compiled for (register cap)
#ifndef AUR_TRAV_MINB
#define AUR_TRAV_MINB 4
#endif
enum : int { B_MISS = 0, B_MATTE = 1, B_KELEMEN = 2, B_CT = 3, B_METAL = 4, B_CONST = 5, kBuckets = 6 };
// counters
enum : int {
    C_EXT0 = 0, C_EXT1 = 1, C_SHADOW = 2, C_WORK = 3, C_TOTAL = 4, C_CUR_EXT = 5, C_CUR_SHADE = 6,
    C_CUR_SHADOW = 7, C_CUR_SORT = 8, C_CUR_SHADE2 = 9, C_LIST = 10, C_FRESH = 11, C_SCENES = 12,
    C_BUCKET = 16, C_FILL = 24, kCounters = 32
};
// What a pass keeps beside the queues; copied to the host in one piece.
struct WfState {
    uint32_t ctr[kCounters];
    int32_t stage;                    // the stage that is running (-1: none yet)
    int32_t pad;
    unsigned long long stamp;         // when it began
    // summed over the passes of a render:
    unsigned long long rays[2];       // closest-hit rays, any-hit rays
    unsigned long long stage_ns[5];   // device time of regen, extend, sort, shade, shadow
};

struct WfScene {
    DevScene sc;
    PathParams p;          // spp = samples of this pass, sample_offset = first sample index of this pass
    uint64_t key;
    uint32_t npix, item_base, items, rec_depth, rec_stride;
    // Light samples: every camera sample of the pass has lsub sub-samples q = sl * lsub + j
    // (lsub = light_samples, 1 without them); sub-sample j of sample s traces the path j of
    // Integrator::integrateCameraSample(sample, numSamples) and draws from random-number sample
    // index s * lsub + j = rng_offset + q, its camera ray from s * lsub. The render's sample 0
    // has one path only (renderer.cpp:231-258): its sub-samples j > 0 are skipped.
    uint32_t lsub, rng_offset;
    float4* samples;       // [spp_pass * lsub][npix]
    // resolve: the film and, for renders of several passes, the sums between them
    float4 *film, *acc_s, *acc_c;
    int32_t total_spp, first_pass, last_pass;
    // record mode (path-replay adjoint): per item (sample-major, sl * npix + pixel)
    float4* rec;           // [items][rec_depth][rec_stride] vertex records (kVertexRec)
    float4* lo_raw;        // [items] unclamped path radiance, w = number of recorded vertices
};

// Per-slot state in 32-byte pairs (one DRAM sector per slot and pair), structure of arrays
// over the slots: the stages gather slots in queue order (material buckets, not slot order),
// so a float4 of its own array would pull a half-used sector per field; a pair of fields that
// are read together fills its sector, and slot-order sweeps (regen) stay coalesced.
//   ray    origin + mint, direction + maxt        (extend, shade; written by regen, shade)
//   hitid  hit (t, u, v, prim), id (scene, pixel, sub-sample, flags)   (extend, sort, shade, regen)
//   tplo   throughput + roulette factor, radiance + alpha              (shade, regen)
//   neeA   shading point, first next-event direction + maxt            (shadow)
//   neeB   second next-event direction + maxt, its contribution        (shadow, regen)
//   neeC   first next-event contribution, throughput + nvis            (regen)
struct WfPool {
    float4 *ray, *hitid, *tplo, *neeA, *neeB, *neeC;   // [P][2] each
    uint32_t* q_regen;          // what regen has to do: by slot (sweep), or a list of the slots (see k_regen)
    uint32_t* sh_vis;           // bit k: next-event ray k of the slot is unoccluded
    uint32_t* rec_cur;          // record mode: record index << 1 | specular lobe of the vertex whose next-event rays
                                // are in flight, kNoRec if it has no parameter
    uint8_t* bucket;            // material bucket of the slot's last hit (written by the sorting extend)
    uint32_t *q_ext0, *q_ext1, *q_sort, *q_shadow;
    uint32_t* ctr;              // WfState::ctr
    WfState* st;
    const WfScene* scenes;
    uint32_t P;
    __device__ __forceinline__ float4& ray_o(uint32_t i) const { return ray[2 * (size_t)i]; }
    __device__ __forceinline__ float4& ray_d(uint32_t i) const { return ray[2 * (size_t)i + 1]; }
    __device__ __forceinline__ float4& hit(uint32_t i) const { return hitid[2 * (size_t)i]; }
    __device__ __forceinline__ uint4& id(uint32_t i) const { return reinterpret_cast<uint4*>(hitid)[2 * (size_t)i + 1]; }
    __device__ __forceinline__ float4& tp(uint32_t i) const { return tplo[2 * (size_t)i]; }
    __device__ __forceinline__ float4& lo(uint32_t i) const { return tplo[2 * (size_t)i + 1]; }
    __device__ __forceinline__ float4& sh_p(uint32_t i) const { return neeA[2 * (size_t)i]; }
    __device__ __forceinline__ float4& sh_d0(uint32_t i) const { return neeA[2 * (size_t)i + 1]; }
    __device__ __forceinline__ float4& sh_d1(uint32_t i) const { return neeB[2 * (size_t)i]; }
    __device__ __forceinline__ float4& sh_c1(uint32_t i) const { return neeB[2 * (size_t)i + 1]; }
};

// flags in id.w; kNoClamp: the sample is the environment seen by the camera ray, which
// the reference adds without the firefly filter
constexpr uint32_t kNoClamp = 1u << 21;
__device__ __forceinline__ uint32_t pack_flags(int vtx, int bounces, int kind, bool matte) {
    return (uint32_t)vtx | ((uint32_t)bounces << 9) | ((uint32_t)kind << 18) | ((uint32_t)matte << 20);
}
__device__ __forceinline__ int f_vtx(uint32_t f) { return f & 511; }
__device__ __forceinline__ int f_bounces(uint32_t f) { return (f >> 9) & 511; }
__device__ __forceinline__ int f_kind(uint32_t f) { return (f >> 18) & 3; }
__device__ __forceinline__ bool f_matte(uint32_t f) { return (f >> 20) & 1; }

// A slot's 32-byte pair in one 256-bit access (the pool's arrays are written and read by the stages
// in turn: no read-only loads, and no reordering around the stage's own stores)
__device__ __forceinline__ void ld_pair(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p) : "memory");
}
__device__ __forceinline__ void st_pair(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w) : "memory");
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t lanemask_lt() { return (1u << lane_id()) - 1u; }

// Block 0's first thread charges the time since the previous stage began to that stage: two
// timer reads and a few stores a launch, where event records between the launches cost every
// graph as many nodes again. Stage -1: nothing runs that is to be charged.
__device__ __forceinline__ void stage_begins(WfState* st, int stage) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    unsigned long long now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    if (st->stage >= 0) st->stage_ns[st->stage] += now - st->stamp;
    st->stamp = now;
    st->stage = stage;
}

// After the graphs that the host reads the counters between: its time is no stage's.
__global__ void k_stage_end(WfPool w) { stage_begins(w.st, -1); }

// Block-aggregated append to kQ queues: every thread of the block calls it (uniform control
// flow) with its flags; it returns each flagged thread's slot in the queue. One atomic per
// queue per block instead of one per warp.
struct BlockScan { uint32_t cnt[16][4]; uint32_t base[4]; };
template <int kQ>
__device__ __forceinline__ void block_reserve(BlockScan& sh, const bool (&p)[kQ], uint32_t* const (&ctr)[kQ],
                                              uint32_t (&pos)[kQ]) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t m[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) m[q] = __ballot_sync(0xffffffffu, p[q]);
    if (lane_id() == 0)
#pragma unroll
        for (int q = 0; q < kQ; ++q) sh.cnt[warp][q] = __popc(m[q]);
    __syncthreads();
    if (threadIdx.x < kQ) {
        const int q = threadIdx.x;
        uint32_t t = 0;
        for (int j = 0; j < nw; ++j) { const uint32_t c = sh.cnt[j][q]; sh.cnt[j][q] = t; t += c; }
        sh.base[q] = t ? atomicAdd(ctr[q], t) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kQ; ++q) pos[q] = sh.base[q] + sh.cnt[warp][q] + __popc(m[q] & lanemask_lt());
    __syncthreads();   // sh is reused by the next call
}

// Work items for the flagged threads, as many as there are left, and places in the ray queue for those
// that get one: thread 0 takes both, as the items go to the lowest ranks. True if this thread got an
// item. Two barriers where a reservation each took six: regen of 16 small frames 4.17 -> 3.80 ms,
// of the 1080p terrain frame 14.3 -> 14.0 (the rest is its scattered records).
__device__ __forceinline__ bool block_take_items(BlockScan& sh, bool want, uint32_t* next_item, uint32_t total,
                                                 uint32_t* queue, uint32_t* item, uint32_t* pos) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t m = __ballot_sync(0xffffffffu, want);
    if (lane_id() == 0) sh.cnt[warp][0] = __popc(m);
    __syncthreads();
    uint32_t rank = __popc(m & lanemask_lt());
    for (int j = 0; j < warp; ++j) rank += sh.cnt[j][0];
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int j = 0; j < nw; ++j) t += sh.cnt[j][0];
        const uint32_t first = t ? atomicAdd(next_item, t) : total;
        const uint32_t got = first < total ? min(t, total - first) : 0u;
        sh.base[0] = first;
        sh.base[1] = got ? atomicAdd(queue, got) : 0u;
    }
    __syncthreads();   // the next call's writes are behind its own barriers: cnt is read before this one
    *item = sh.base[0] + rank;
    *pos = sh.base[1] + rank;
    return want && *item < total;
}

// random-number sample index of sub-sample q, and that of its camera ray
__device__ __forceinline__ uint32_t rng_index(const WfScene& S, uint32_t q) { return S.rng_offset + q; }
__device__ __forceinline__ uint32_t cam_index(const WfScene& S, uint32_t q) {
    return S.lsub > 1 ? S.rng_offset + q - q % S.lsub : S.rng_offset + q;
}
// The k-th sub-sample that a pass traces per pixel: all of them, but for the render's sample 0,
// which has one path (its sub-samples j > 0 are no work items).
__device__ __forceinline__ uint32_t sub_sample(const WfScene& S, uint32_t k) {
    return S.p.sample_offset == 0 && k > 0 ? k + S.lsub - 1 : k;
}

__device__ __forceinline__ int scene_of(const WfPool& w, uint32_t item) {
    int lo = 0, hi = (int)w.ctr[C_SCENES] - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (w.scenes[mid].item_base <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ------------------------------------------------------------------ regen
// Slots that the last shading stage left something to do for (next-event radiance to add, or a
// finished path); in a pass's first iteration (C_FRESH) as many unused slots as there is work.
// Two ways to find them. kSweep: every slot's flags are read in slot order, and the records of
// those that have work. Otherwise the shading stage appends them to a list. A pass whose paths
// all fit the pool takes the list, where nothing is refilled and ever fewer slots are left: the
// 512 x 512 sphere frame's regen 3.0 -> 1.2 ms of 14.4. One that refills its slots takes the
// sweep, which hands consecutive pixels to consecutive slots; the list hands them out in the
// shading stage's order, and on the 1080p terrain frame the pool's gathers lost what locality
// they had (regen 13.6 -> 30.5, shade 51.7 -> 62.8 ms).
template <bool kRec, bool kSweep>
__global__ void k_regen(WfPool w, int in_q) {
    __shared__ BlockScan s_scan;
    stage_begins(w.st, 0);
    uint32_t* qin = in_q ? w.q_ext1 : w.q_ext0;
    uint32_t* cin = &w.ctr[in_q ? C_EXT1 : C_EXT0];
    const uint32_t total = w.ctr[C_TOTAL];
    const bool fresh = w.ctr[C_FRESH] != 0;
    const uint32_t n = fresh ? (total < w.P ? total : w.P) : kSweep ? w.P : w.ctr[C_LIST];
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t k = base + threadIdx.x;
        bool want = false;
        uint32_t i = k;
        if (fresh) {
            want = k < n;
        } else if (const uint32_t e = k < n ? w.q_regen[k] : 0u) {
            if (kSweep) w.q_regen[k] = 0u;
            else i = e & (kDone - 1);
            // the slot's records are loaded together, so that their latencies overlap (c0 and t
            // share one 32-byte pair)
            float4 lo = w.lo(i);
            const uint4 id = w.id(i);
            if (e & kPending) {
                // next-event estimate of the last vertex: Lo += ((vis0 c0 + vis1 c1) nvis) T, the
                // plain kernel's order of operations (integrate_direct)
                const uint32_t vis = w.sh_vis[i];
                float4 c0, t;
                ld_pair(w.neeC + 2 * (size_t)i, c0, t);
                const float nvis = t.w;   // the number of visible lights rides in the throughput record
                float3 res = mk(0.f, 0.f, 0.f);
                if (vis & 1u) res += mk(c0.x, c0.y, c0.z);   // only unoccluded contributions are added
                if (vis & 2u) { const float4 c1 = w.sh_c1(i); res += mk(c1.x, c1.y, c1.z); }
                const float3 add = (res * nvis) * mk(t.x, t.y, t.z);
                lo.x += add.x; lo.y += add.y; lo.z += add.z;
                if (!(e & kDone)) w.lo(i) = lo;
                if (kRec) {   // the next-event estimate's derivative and the radiance so far complete the record
                    const uint32_t rc = w.rec_cur[i];
                    if (rc != kNoRec) {
                        const WfScene& S = w.scenes[id.x];
                        float4* r = S.rec + (size_t)(rc >> 1) * S.rec_stride;
                        const float4 c1 = w.sh_c1(i);
                        float3 d = mk(0.f, 0.f, 0.f);
                        if (rc & 1u) {   // roughness: each contribution times its d ln f (c0.w, c1.w)
                            if (vis & 1u) d += mk(c0.x, c0.y, c0.z) * c0.w;
                            if (vis & 2u) d += mk(c1.x, c1.y, c1.z) * c1.w;
                        } else if (vis & 1u) {
                            d = mk(c1.x, c1.y, c1.z);
                        }
                        const float3 g = mk(t.x, t.y, t.z) * (d * nvis);
                        r->x = lo.x; r->y = lo.y; r->z = lo.z;
                        r[1] = make_float4(g.x, g.y, g.z, 0.f);
                    }
                }
            }
            if (e & kDone) {
                const WfScene& S = w.scenes[id.x];
                if (kRec) {
                    S.lo_raw[(size_t)id.z * S.npix + id.y] = make_float4(lo.x, lo.y, lo.z, __int_as_float(f_vtx(id.w)));
                } else {
                    const float3 L = (id.w & kNoClamp) ? mk(lo.x, lo.y, lo.z) : firefly_clamp(mk(lo.x, lo.y, lo.z));
                    // with light samples, alpha 2 marks the environment seen by the camera ray: the
                    // sample is that radiance, not the mean of its sub-samples (integrator.cpp:287-298)
                    const float a = (S.lsub > 1 && (id.w & kNoClamp)) ? 2.f : lo.w;
                    S.samples[(size_t)id.z * S.npix + id.y] = make_float4(L.x, L.y, L.z, a);
                }
                want = *(volatile uint32_t*)&w.ctr[C_WORK] < total;
            }
        }
        uint32_t item, pos;
        const bool start = block_take_items(s_scan, want, &w.ctr[C_WORK], total, cin, &item, &pos);
        if (start) {
            const int s = scene_of(w, item);
            const WfScene& S = w.scenes[s];
            const uint32_t local = item - S.item_base;
            const uint32_t pixel = local % S.npix, q = sub_sample(S, local / S.npix);
            PathRng rng;
            rng.key = S.key;
            rng.base = path_base(pixel, cam_index(S, q));
            const RayF r = camera_ray(S.sc.cam, (int)(pixel % (uint32_t)S.sc.cam.w), (int)(pixel / (uint32_t)S.sc.cam.w),
                                      rng.u(kDimCamera), rng.u(kDimCamera + 1));
            st_pair(w.ray + 2 * (size_t)i, make_float4(r.o.x, r.o.y, r.o.z, r.mint), make_float4(r.d.x, r.d.y, r.d.z, r.maxt));
            st_pair(w.tplo + 2 * (size_t)i, make_float4(1.f, 1.f, 1.f, 1.f), make_float4(0.f, 0.f, 0.f, 0.f));
            w.id(i) = make_uint4((uint32_t)s, pixel, q, pack_flags(0, 0, RAY_CAMERA, false));
        }
        if (start) qin[pos] = i;
    }
}

// ------------------------------------------------------------------ extend
__device__ __forceinline__ int bucket_of(const ShadeScene& sh, int prim) {
    if (prim < 0) return B_MISS;
    static_assert(B_MATTE == MAT_MATTE + 1 && B_KELEMEN == MAT_KELEMEN + 1 && B_CT == MAT_COOKTORRANCE + 1 &&
                  B_METAL == MAT_METAL + 1 && B_CONST == MAT_CONSTANT + 1 && MAT_GLASS > MAT_CONSTANT, "bucket order");
    return min((int)__ldg(sh.tri_type + prim), (int)MAT_CONSTANT) + 1;
}

// The tree a traversal kernel walks.
enum : int { TREE_BINARY = 0, TREE_WIDE = 1, TREE_QUANT = 2 };
template <int kTree, bool kAnyHit> struct TreeTypes;
template <bool kAnyHit> struct TreeTypes<TREE_BINARY, kAnyHit> {
    using Node = BvhNode;
    using Stack = LaneStack;
    using Trace = TraceState<kAnyHit>;
    __device__ static const Node* nodes(const DevScene& sc) { return sc.nodes; }
};
template <bool kAnyHit> struct TreeTypes<TREE_WIDE, kAnyHit> {
    using Node = BvhNode4;
    using Stack = LaneStack4;
    using Trace = TraceState4<kAnyHit, BvhNode4>;
    __device__ static const Node* nodes(const DevScene& sc) { return sc.nodes4; }
};
template <bool kAnyHit> struct TreeTypes<TREE_QUANT, kAnyHit> {
    using Node = BvhNode4Q;
    using Stack = LaneStack4;
    using Trace = TraceState4<kAnyHit, BvhNode4Q>;
    __device__ static const Node* nodes(const DevScene& sc) { return sc.nodes4q; }
};

// Closest hit for the extension queue. Each lane keeps a resumable traversal;
// finished lanes are refilled from the queue (one atomic per warp) while the
// others continue, so a warp is not held up by its slowest ray.
template <bool kSort, int kTree>
__global__ void __launch_bounds__(256, AUR_TRAV_MINB) k_extend(WfPool w, int in_q) {
    using Tree = TreeTypes<kTree, false>;
    const uint32_t* qin = in_q ? w.q_ext1 : w.q_ext0;
    const uint32_t n = w.ctr[in_q ? C_EXT1 : C_EXT0];
    // Outputs of the later stages start empty. Only counters that no block of
    // this kernel touches are reset here; the bucket counters this kernel
    // increments were reset by the previous next-event stage (or the pass start).
    stage_begins(w.st, 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.ctr[C_LIST] = 0;
        w.ctr[C_FRESH] = 0;
        w.ctr[in_q ? C_EXT0 : C_EXT1] = 0;
        w.ctr[C_SHADOW] = 0;
        w.ctr[C_CUR_SHADE] = 0;
        w.ctr[C_CUR_SHADE2] = 0;
        w.ctr[C_CUR_SHADOW] = 0;
        w.ctr[C_CUR_SORT] = 0;
        w.st->rays[0] += n;
    }
    extern __shared__ int s_stack[];
    __shared__ uint32_t s_bucket[kBuckets];   // per-block material counts, added to the global ones at exit
    __shared__ uint32_t s_tie[256];           // per thread: first slot of its list of exact-distance ties
    if (kSort && threadIdx.x < kBuckets) s_bucket[threadIdx.x] = 0;
    s_tie[threadIdx.x] = 0xffffffffu;
    __syncthreads();
    typename Tree::Stack stack;
    stack.col = s_stack + threadIdx.x;
    stack.stride = blockDim.x;
    typename Tree::Trace ts;
    const typename Tree::Node* nodes = nullptr;
    const BvhTri* tris = nullptr;
    const WfScene* S = nullptr;
    uint32_t slot = 0;
    bool has = false, exhausted = false;
    while (true) {
        const bool need = !has && !exhausted;
        const uint32_t m = __ballot_sync(0xffffffffu, need);
        const uint32_t act = __ballot_sync(0xffffffffu, has);
        if (m && (__popc(m) >= kRefill || act == 0)) {
            const int leader = __ffs(m) - 1;
            uint32_t b = 0;
            if ((int)lane_id() == leader) b = atomicAdd(&w.ctr[C_CUR_EXT], (uint32_t)__popc(m));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (need) {
                const uint32_t k = b + __popc(m & lanemask_lt());
                if (k < n) {
                    slot = qin[k];
                    S = &w.scenes[w.id(slot).x];
                    nodes = Tree::nodes(S->sc);
                    tris = S->sc.tris;
                    float4 o, d;
                    ld_pair(w.ray + 2 * (size_t)slot, o, d);
                    ts.begin(mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), o.w, d.w);
                    has = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, has || !exhausted) == 0) break;
        for (int k = 0; k < kRounds; ++k) ts.round(nodes, tris, stack);   // all lanes take part in every round
        const bool done = has && ts.finished();
        int bucket = -1;
        if (done) {
            if (kTree == TREE_QUANT && ts.tie) {   // traced again below; the thread's ties are a list through q_sort
                w.q_sort[slot] = s_tie[threadIdx.x];
                s_tie[threadIdx.x] = slot;
            } else {
                w.hit(slot) = make_float4(ts.tbest, ts.bu, ts.bv, __int_as_float(ts.best));
                if (kSort) {
                    bucket = bucket_of(S->sc.sh, ts.best);
                    w.bucket[slot] = (uint8_t)bucket;   // the scatter reads it instead of the hit's material
                }
            }
            has = false;
        }
        if (kSort) {   // per-bucket counts, one shared atomic per (warp, bucket)
            const uint32_t fin = __ballot_sync(0xffffffffu, bucket >= 0);
            if (bucket >= 0) {
                const uint32_t peers = __match_any_sync(fin, bucket);
                if ((int)lane_id() == __ffs(peers) - 1) atomicAdd(&s_bucket[bucket], (uint32_t)__popc(peers));
            }
        }
    }
    if constexpr (kTree == TREE_QUANT) {
        // rays that met two triangles at exactly the same distance take the hit that the
        // full-precision tree's visiting order gives (out of the main loop, so that the second
        // traversal adds no registers to it)
        for (uint32_t i = s_tie[threadIdx.x]; i != 0xffffffffu; i = w.q_sort[i]) {
            const WfScene& T = w.scenes[w.id(i).x];
            const float4 o = w.ray_o(i), d = w.ray_d(i);
            Hit h;
            TraceWork work;
            bvh_trace4<false>(T.sc.nodes4, T.sc.tris, mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), o.w, d.w, &h, work);
            w.hit(i) = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
            if (kSort) {
                const int b = bucket_of(T.sc.sh, h.prim);
                w.bucket[i] = (uint8_t)b;
                atomicAdd(&s_bucket[b], 1u);
            }
        }
    }
    if (kSort) {
        __syncthreads();
        if (threadIdx.x < kBuckets && s_bucket[threadIdx.x]) atomicAdd(&w.ctr[C_BUCKET + threadIdx.x], s_bucket[threadIdx.x]);
    }
}

// counting-sort scatter of the extension queue into q_sort, grouped by bucket
__global__ void k_sort_scatter(WfPool w, int in_q) {
    stage_begins(w.st, 2);
    const uint32_t* qin = in_q ? w.q_ext1 : w.q_ext0;
    const uint32_t n = w.ctr[in_q ? C_EXT1 : C_EXT0];
    __shared__ uint32_t s_ofs[kBuckets], s_cnt[kBuckets], s_base[kBuckets];
    __shared__ uint32_t s_fetch;
    if (threadIdx.x == 0) {
        uint32_t a = 0;
        for (int b = 0; b < kBuckets; ++b) { s_ofs[b] = a; a += w.ctr[C_BUCKET + b]; }
    }
    while (true) {   // a block takes blockDim entries at a time; one atomic per bucket per block
        if (threadIdx.x == 0) s_fetch = atomicAdd(&w.ctr[C_CUR_SORT], blockDim.x);
        if (threadIdx.x < kBuckets) s_cnt[threadIdx.x] = 0;
        __syncthreads();
        const uint32_t b = s_fetch;
        if (b >= n) break;
        const uint32_t k = b + threadIdx.x;
        int bucket = -1;
        uint32_t slot = 0, local = 0;
        if (k < n) {
            slot = qin[k];
            bucket = w.bucket[slot];
        }
        const uint32_t active = __ballot_sync(0xffffffffu, bucket >= 0);
        if (bucket >= 0) {
            const uint32_t peers = __match_any_sync(active, bucket);
            const int leader = __ffs(peers) - 1;
            uint32_t wb = 0;
            if ((int)lane_id() == leader) wb = atomicAdd(&s_cnt[bucket], (uint32_t)__popc(peers));
            local = __shfl_sync(peers, wb, leader) + __popc(peers & lanemask_lt());
        }
        __syncthreads();
        if (threadIdx.x < kBuckets)
            s_base[threadIdx.x] = s_cnt[threadIdx.x] ? atomicAdd(&w.ctr[C_FILL + threadIdx.x], s_cnt[threadIdx.x]) : 0u;
        __syncthreads();
        if (bucket >= 0) w.q_sort[s_ofs[bucket] + s_base[bucket] + local] = slot;
        __syncthreads();   // s_fetch and s_cnt are rewritten next round
    }
}

// ------------------------------------------------------------------ shade
// A ray that missed in a scene with environment lights: the camera ray sees the
// environment (alpha 1, no firefly filter), an escaping mirror ray adds it times the
// throughput, both along the camera ray's direction (integrator.cpp:262-288). Out of line.
__device__ __noinline__ float4 shade_env_miss(const WfPool* w, const WfScene* S, uint32_t slot, uint4 id, int vtx,
                                              float4 lo) {
    PathRng rng;
    rng.key = S->key;
    rng.base = path_base(id.y, cam_index(*S, id.z));
    const RayF cr = camera_ray(S->sc.cam, (int)(id.y % (uint32_t)S->sc.cam.w), (int)(id.y / (uint32_t)S->sc.cam.w),
                               rng.u(kDimCamera), rng.u(kDimCamera + 1));
    const float3 e = env_radiance_of(S->sc.sh.lights, S->sc.sh.nlights, S->sc.sh.texs, S->sc.sh.texels, cr.d);
    if (vtx == 0) {
        w->id(slot).w = id.w | kNoClamp;
        return make_float4(e.x, e.y, e.z, 1.f);
    }
    const float4 t = w->tp(slot);
    const float3 a = e * mk(t.x, t.y, t.z);
    return make_float4(lo.x + a.x, lo.y + a.y, lo.z + a.z, lo.w);
}

// The record mode's derivatives, out of line: one copy of their double-precision transcendentals.
static __device__ __noinline__ float rec_eval_dlnD(float rough, float3 N, float3 V, float3 L) { return eval_dlnD(rough, N, V, L); }
static __device__ __noinline__ float rec_sample_dlnD(float rough, float3 N, float3 V, float3 L) {
    return sample_dlnD(rough, N, V, L);
}

// Three resident 256-thread blocks per SM (85 registers, some spilled) instead of the two that
// its 106 registers allow: 50.7 vs 52.3 ms per 1080p frame.
// kPart selects the entries: SHADE_ALL every queued one; with the queue sorted by bucket,
// SHADE_MATTE the matte bucket alone (its lobe known at compile time, so the glossy lobes'
// code and registers drop out) and SHADE_REST all others. The bucket counts stay in place
// until the next-event stage resets them, after both parts have read them.
enum : int { SHADE_ALL = 0, SHADE_MATTE = 1, SHADE_REST = 2 };
#ifndef AUR_SHADE_MATTE_MINB
#define AUR_SHADE_MATTE_MINB 4
#endif
template <bool kRec, int kPart>
__global__ void __launch_bounds__(256, kPart == SHADE_MATTE ? AUR_SHADE_MATTE_MINB : 3) k_shade(WfPool w, int in_q, int sorted,
                                                                                                 bool sweep) {
    const uint32_t* qin = sorted ? w.q_sort : (in_q ? w.q_ext1 : w.q_ext0);
    const uint32_t n_all = w.ctr[in_q ? C_EXT1 : C_EXT0];
    // the sorted queue holds the misses first, then the matte bucket
    const uint32_t nmiss = kPart == SHADE_ALL ? 0u : w.ctr[C_BUCKET + B_MISS];
    const uint32_t nm = kPart == SHADE_ALL ? 0u : w.ctr[C_BUCKET + B_MATTE];
    const uint32_t n = kPart == SHADE_ALL ? n_all : kPart == SHADE_MATTE ? nm : n_all - nm;
    uint32_t* qout = in_q ? w.q_ext0 : w.q_ext1;
    uint32_t* cout = &w.ctr[in_q ? C_EXT0 : C_EXT1];
    __shared__ BlockScan s_scan;
    __shared__ uint32_t s_fetch;
    if (kPart != SHADE_REST) stage_begins(w.st, 3);
    while (true) {
        if (threadIdx.x == 0) s_fetch = atomicAdd(&w.ctr[kPart == SHADE_MATTE ? C_CUR_SHADE2 : C_CUR_SHADE], blockDim.x);
        __syncthreads();
        const uint32_t b = s_fetch;   // rewritten only after block_reserve's barriers below
        if (b >= n) break;
        const uint32_t k = b + threadIdx.x;
        bool push_ext = false, push_sh0 = false, push_sh1 = false, done = false;
        uint32_t slot = 0;
        if (k < n) {
            slot = qin[kPart == SHADE_ALL ? k : kPart == SHADE_MATTE ? nmiss + k : (k < nmiss ? k : k + nm)];
            float4 hh, idf, tpv, lo;
            ld_pair(w.hitid + 2 * (size_t)slot, hh, idf);
            ld_pair(w.tplo + 2 * (size_t)slot, tpv, lo);
            const uint4 id = make_uint4(__float_as_uint(idf.x), __float_as_uint(idf.y), __float_as_uint(idf.z),
                                        __float_as_uint(idf.w));
            const int prim = __float_as_int(hh.w);
            if (prim < 0) {
                const WfScene& S = w.scenes[id.x];
                const int kind = f_kind(id.w), vtx = f_vtx(id.w);
                if (S.sc.sh.nenv && (vtx == 0 || kind == RAY_MIRROR))
                    lo = shade_env_miss(&w, &S, slot, id, vtx, lo);
                done = true;
                w.lo(slot) = lo;
            } else if (f_vtx(id.w) >= w.scenes[id.x].p.max_depth) {
                // the reference's unshaded last ray hit something: the path ends
                done = true;
            } else {
                const WfScene& S = w.scenes[id.x];
                const DevScene& sc = S.sc;
                const uint32_t flags = id.w;
                const int vtx = f_vtx(flags);
                int kind = f_kind(flags);
                bool matte = f_matte(flags);
                int bounces = f_bounces(flags);
                PathRng rng;
                rng.key = S.key;
                rng.base = path_base(id.y, rng_index(S, id.z));
                float4 ro, rd;
                ld_pair(w.ray + 2 * (size_t)slot, ro, rd);
                float3 T = mk(tpv.x, tpv.y, tpv.z);
                float cont = tpv.w;
                float3 Lo = mk(lo.x, lo.y, lo.z);
                if (vtx == 0) lo.w = 1.f;   // camera ray hit: alpha
                const uint32_t rec_at = (id.z * S.npix + id.y) * S.rec_depth + (uint32_t)vtx;
                const Frame f = hit_frame(sc.sh, prim, hh.x, hh.y, hh.z, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), true);
                const Attr at = sc.sh.attrs[f.attr];
                if (kind == RAY_DIFFUSE) matte = true;
                if (collects_emission(kind)) Lo += T * at.emission;
                const float lobe_u = kPart == SHADE_MATTE ? 0.f : rng.u(vertex_dim(vtx, kDimLobe));
                const Brdf brdf = kPart == SHADE_MATTE ? matte_brdf(sc.sh, sc.sh.mats[at.material], f)
                                                       : get_brdf(sc.sh, at.material, f, matte, lobe_u);
                ParamRef pr;
                if (kRec) pr = param_of(sc.sh, at.material, brdf, f, matte, lobe_u);
                const float3 pre = Lo;       // record: the radiance before the next-event estimate
                bool nee_rec = false;
                // next-event estimation: rays and their unoccluded contributions
                if (brdf.lobe == LOBE_MATTE || brdf.lobe == LOBE_SPEC) {
                    int nvis;
                    const int li = pick_visible_light(sc.sh, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightPick)), &nvis);
                    if (li >= 0) {
                        const Light& L = sc.sh.lights[li];   // global: the env paths take its address
                        const LightSample ls = light_sample(sc.sh, L, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightSample)),
                                                            rng.u(vertex_dim(vtx, kDimLightSample + 1)));
                        float cost = dot(f.N, ls.dir);
                        float3 c0 = mk(0.f, 0.f, 0.f), c1 = c0;
                        float3 d0 = ls.dir, d1 = ls.dir;
                        float m0 = ls.maxt, m1 = 0.f;
                        bool r0 = false, r1 = false;
                        float g0 = 0.f, g1 = 0.f;   // record: d ln c / d roughness
                        if (brdf.lobe == LOBE_MATTE) {
                            if (cost >= 0.f && ls.pdf > 0.f) {
                                r0 = true;
                                c0 = cdiv((ls.color * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                                if (kRec && cost > 0.f) c1 = cdiv((ls.color * kInvPiMacro) * cost, ls.pdf);   // d c0 / d colour
                            }
                        } else {
                            if (cost > 0.f && ls.pdf > 0.f) {
                                const float bp = brdf_pdf(brdf, ls.dir, f.V, f.N);
                                if (bp > 0.f) {
                                    r0 = true;
                                    const float wgt = power_heuristic(ls.pdf, bp);
                                    c0 = cdiv(((ls.color * wgt) * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                                    if (kRec && pr.kind == 3) g0 = rec_eval_dlnD(brdf.rough, f.N, f.V, ls.dir) * pr.dr;
                                }
                            }
                            const BrdfSample bs = brdf_sample(brdf, f.V, f.N, rng.u(vertex_dim(vtx, kDimMisBrdf)),
                                                              rng.u(vertex_dim(vtx, kDimMisBrdf + 1)));
                            cost = dot(f.N, bs.dir);
                            if (cost > 0.f) {
                                float maxt = bs.maxt;
                                const float lp = light_pdf(sc.sh, L, f.P, bs.dir, kRayBias, &maxt);
                                if (lp > 0.f && bs.pdf > 0.f) {
                                    r1 = true;
                                    d1 = bs.dir;
                                    m1 = maxt;
                                    const float wgt = power_heuristic(bs.pdf, lp);
                                    c1 = cdiv(((bs.color * wgt) * light_eval(sc.sh, L, bs.dir)) * cost, bs.pdf);
                                    if (kRec && pr.kind == 3) g1 = rec_sample_dlnD(brdf.rough, f.N, f.V, bs.dir) * pr.dr;
                                }
                            }
                        }
                        if (r0 || r1) {
                            if (kRec) {
                                w.rec_cur[slot] = pr.kind == 0 ? kNoRec : (rec_at << 1) | (pr.kind == 3 ? 1u : 0u);
                                nee_rec = true;
                            }
                            st_pair(w.neeA + 2 * (size_t)slot, make_float4(f.P.x, f.P.y, f.P.z, 0.f),
                                    make_float4(d0.x, d0.y, d0.z, m0));
                            if (kRec || r1)   // nothing else reads the second ray's pair
                                st_pair(w.neeB + 2 * (size_t)slot, make_float4(d1.x, d1.y, d1.z, m1),
                                        make_float4(c1.x, c1.y, c1.z, g1));
                            st_pair(w.neeC + 2 * (size_t)slot, make_float4(c0.x, c0.y, c0.z, g0),
                                    make_float4(T.x, T.y, T.z, (float)nvis));
                            w.sh_vis[slot] = 0u;
                            push_sh0 = r0;
                            push_sh1 = r1;
                        }
                    }
                }
                // continuation (integrator.cpp:208-261)
                bool alive = false;
                const BrdfSample bs = brdf_sample(brdf, f.V, f.N, rng.u(vertex_dim(vtx, kDimBrdf)),
                                                  rng.u(vertex_dim(vtx, kDimBrdf + 1)));
                if (kRec) {
                    // the vertex's record; regen completes it where next-event rays are in flight
                    float4* r = S.rec + (size_t)rec_at * S.rec_stride;
                    float3 q = mk(0.f, 0.f, 0.f);
                    if (pr.kind != 0) {
                        if (bs.pdf > 0.f) {
                            if (pr.kind == 3) {
                                const float g = rec_sample_dlnD(brdf.rough, f.N, f.V, bs.dir) * pr.dr;   // dw/w = d ln f
                                q = mk(g, g, g);
                            } else {
                                const float cosl = dot(f.N, bs.dir);
                                const float3 wt = cdiv(bs.color * cosl, bs.pdf);
                                const float dw = kInvPiMacro * cosl / bs.pdf;   // d w_c / d diffuse_c
                                q = mk(wt.x != 0.f ? dw / wt.x : 0.f, wt.y != 0.f ? dw / wt.y : 0.f,
                                       wt.z != 0.f ? dw / wt.z : 0.f);
                            }
                        }
                        float score = 0.f;
                        if (kPart != SHADE_MATTE) {
                            const Material& m = sc.sh.mats[at.material];
                            if (m.type == MAT_KELEMEN && m.refl < 1.f && m.rough_tex < 0)
                                score = kelemen_score(sc.sh, m, f, brdf, matte);
                        }
                        if (nee_rec) {
                            r->w = __int_as_float(at.material);
                        } else {
                            r[0] = make_float4(pre.x, pre.y, pre.z, __int_as_float(at.material));
                            r[1] = make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                        r[2] = make_float4(pre.x, pre.y, pre.z, score);
                        if (S.rec_stride > kVertexRec && pr.kind == 2) {
                            r[4] = make_float4(__int_as_float(pr.taps.idx[0]), __int_as_float(pr.taps.idx[1]),
                                               __int_as_float(pr.taps.idx[2]), 0.f);
                            r[5] = make_float4(pr.taps.w[0], pr.taps.w[1], pr.taps.w[2], 0.f);
                        }
                    }
                    const uint32_t index = (uint32_t)(pr.kind == 2 ? pr.taps.idx[0] : pr.index);
                    r[3] = make_float4(q.x, q.y, q.z, __uint_as_float((uint32_t)pr.kind | (index << 2)));
                }
                // after the last vertex the reference traces one more ray, which only an
                // escaping mirror ray in a scene with an environment light turns into radiance
                // (integrator.cpp:256-274): that ray is queued and its hit is not shaded
                if (continue_path(brdf, bs, f.N, S.p.min_depth, rng, vtx, T, cont, kind, bounces) &&
                    (vtx + 1 < S.p.max_depth || (kind == RAY_MIRROR && sc.sh.nenv))) {
                    alive = true;
                    st_pair(w.ray + 2 * (size_t)slot, make_float4(f.P.x, f.P.y, f.P.z, kRayBias),
                            make_float4(bs.dir.x, bs.dir.y, bs.dir.z, bs.maxt));
                    w.id(slot).w = pack_flags(vtx + 1, bounces, kind, matte);
                }
                st_pair(w.tplo + 2 * (size_t)slot, make_float4(T.x, T.y, T.z, cont), make_float4(Lo.x, Lo.y, Lo.z, lo.w));
                // a finished path's flags count its recorded vertices (a missed ray's vertex is not recorded)
                if (kRec && !alive) w.id(slot).w = pack_flags(vtx + 1, bounces, kind, matte);
                done = !alive;
                push_ext = alive;
            }
        }
        {
            const bool nee = push_sh0 || push_sh1;
            const uint32_t todo = (done ? kDone : 0u) | (nee ? kPending : 0u);
            const bool pp[4] = {push_ext, push_sh0, push_sh1, todo && !sweep};
            uint32_t* const cp[4] = {cout, &w.ctr[C_SHADOW], &w.ctr[C_SHADOW], &w.ctr[C_LIST]};
            uint32_t pos[4];
            block_reserve(s_scan, pp, cp, pos);
            if (push_ext) qout[pos[0]] = slot;
            if (push_sh0) w.q_shadow[pos[1]] = slot << 1;
            if (push_sh1) w.q_shadow[pos[2]] = (slot << 1) | 1u;
            if (todo) w.q_regen[sweep ? slot : pos[3]] = sweep ? todo : slot | todo;
        }
    }
}

// ------------------------------------------------------------------ shadow
// Occlusion of the next-event rays (entries slot << 1 | ray); lanes are refilled as in
// k_extend. An unoccluded ray sets its bit in sh_vis; the next regen adds the light.
template <int kTree>
__global__ void __launch_bounds__(256, AUR_TRAV_MINB) k_shadow(WfPool w) {
    using Tree = TreeTypes<kTree, true>;
    const uint32_t n = w.ctr[C_SHADOW];
    stage_begins(w.st, 4);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.st->rays[1] += n;
        // extend, scatter and shade are finished: reset their fetch and bucket counters
        w.ctr[C_CUR_EXT] = 0;
        for (int k = 0; k < kBuckets; ++k) { w.ctr[C_BUCKET + k] = 0; w.ctr[C_FILL + k] = 0; }
    }
    extern __shared__ int s_stack[];
    typename Tree::Stack stack;
    stack.col = s_stack + threadIdx.x;
    stack.stride = blockDim.x;
    typename Tree::Trace ts;
    const typename Tree::Node* nodes = nullptr;
    const BvhTri* tris = nullptr;
    uint32_t entry = 0;
    bool has = false, exhausted = false;
    while (true) {
        const bool need = !has && !exhausted;
        const uint32_t m = __ballot_sync(0xffffffffu, need);
        const uint32_t act = __ballot_sync(0xffffffffu, has);
        if (m && (__popc(m) >= kRefill || act == 0)) {
            const int leader = __ffs(m) - 1;
            uint32_t b = 0;
            if ((int)lane_id() == leader) b = atomicAdd(&w.ctr[C_CUR_SHADOW], (uint32_t)__popc(m));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (need) {
                const uint32_t k = b + __popc(m & lanemask_lt());
                if (k < n) {
                    entry = w.q_shadow[k];
                    const uint32_t slot = entry >> 1;
                    const WfScene& S = w.scenes[w.id(slot).x];
                    nodes = Tree::nodes(S.sc);
                    tris = S.sc.tris;
                    const float4 p = w.sh_p(slot);
                    const float4 d = (entry & 1u) ? w.sh_d1(slot) : w.sh_d0(slot);
                    ts.begin(mk(p.x, p.y, p.z), mk(d.x, d.y, d.z), kRayBias, d.w);
                    has = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, has || !exhausted) == 0) break;
        for (int k = 0; k < kRounds; ++k) ts.round(nodes, tris, stack);
        if (has && ts.finished()) {
            if (!ts.hit_any) atomicOr(&w.sh_vis[entry >> 1], 1u << (entry & 1u));
            has = false;
        }
    }
}

// ------------------------------------------------------------------ resolve
// Adds this pass's samples of every pixel of every scene (blockIdx.y), in sample order, to the
// pixel's compensated sum (the plain kernel's accumulation order), and after a scene's last pass
// writes its film. A render of one pass keeps no sums in memory. It ends the pass's last stage.
__global__ void k_resolve(const WfScene* scenes, WfState* st) {
    if (blockIdx.y == 0) stage_begins(st, -1);
    const WfScene& S = scenes[blockIdx.y];
    if (S.p.spp == 0) return;
    for (uint32_t pixel = blockIdx.x * blockDim.x + threadIdx.x; pixel < S.npix; pixel += gridDim.x * blockDim.x) {
        Kahan3 k;
        k.init();
        float alpha = 0.f;
        if (!S.first_pass) {
            const float4 a = S.acc_s[pixel], c = S.acc_c[pixel];
            k.s = mk(a.x, a.y, a.z);
            k.c = mk(c.x, c.y, c.z);
            alpha = a.w;
        }
        if (S.lsub <= 1) {
            const float4* v = S.samples + pixel;
            const int n = S.p.spp;
            const size_t step = S.npix;
#pragma unroll 8
            for (int j = 0; j < n; ++j) {
                const float4 x = __ldg(v + j * step);
                k.add(mk(x.x, x.y, x.z));
                alpha += x.w;
            }
        } else {
            // a camera sample with light samples is the mean of its n sub-samples, added in their
            // order as Lo / n (integrate_camera_sample); n = 1 for the render's sample 0
            for (int sl = 0; sl < S.p.spp; ++sl) {
                const float4* sub = S.samples + (size_t)sl * S.lsub * S.npix + pixel;
                const float4 v0 = sub[0];
                if (v0.w == 2.f) {               // the camera ray saw the environment
                    k.add(mk(v0.x, v0.y, v0.z));
                    alpha += 1.f;
                    continue;
                }
                const int n = S.p.sample_offset + sl == 0 ? 1 : (int)S.lsub;
                float3 sum = mk(v0.x, v0.y, v0.z);
                if (n > 1) {
                    sum = cdiv(sum, (float)n);
                    for (int j = 1; j < n; ++j) {
                        const float4 v = sub[(size_t)j * S.npix];
                        sum += cdiv(mk(v.x, v.y, v.z), (float)n);
                    }
                }
                k.add(sum);
                alpha += v0.w;
            }
        }
        if (S.last_pass) {
            const float inv = 1.f / (float)S.total_spp;
            const float3 t = k.total();
            S.film[pixel] = make_float4(t.x * inv, t.y * inv, t.z * inv, alpha * inv);
        } else {
            S.acc_s[pixel] = make_float4(k.s.x, k.s.y, k.s.z, alpha);
            S.acc_c[pixel] = make_float4(k.c.x, k.c.y, k.c.z, 0.f);
        }
    }
}

}  // namespace

constexpr uint32_t kMinPool = 1u << 16;   // no pool smaller than this in the place of one that does not fit

struct WfConfig {
    uint32_t pool = 1u << 21;
    int block = 128;
    int sort = 1;
    int record = 0;   // record mode: vertex records + unclamped radiance per item instead of samples
    bool fixed_pool = false;   // the caller's size: no smaller pool in its place where it does not fit
    // the trees traversed by closest-hit and any-hit rays (TREE_*; the 4-wide ones only when every
    // scene has them), chosen by tree_for
    int tree = TREE_BINARY, tree_any = TREE_BINARY;
};

// The 4-wide traversal is used when every scene of a batch has a 4-wide tree.
#ifndef AUR_WIDE_TRAVERSAL
#define AUR_WIDE_TRAVERSAL 1
#endif
struct BatchItem;
static void tree_for(const std::vector<BatchItem>& items, WfConfig* cfg);

static auto extend_kernel(const WfConfig& c) -> void (*)(WfPool, int) {
    if (c.tree == TREE_QUANT) return c.sort ? k_extend<true, TREE_QUANT> : k_extend<false, TREE_QUANT>;
    if (c.tree == TREE_WIDE) return c.sort ? k_extend<true, TREE_WIDE> : k_extend<false, TREE_WIDE>;
    return c.sort ? k_extend<true, TREE_BINARY> : k_extend<false, TREE_BINARY>;
}
static auto shadow_kernel(const WfConfig& c) -> void (*)(WfPool) {
    return c.tree_any == TREE_QUANT ? k_shadow<TREE_QUANT>
         : c.tree_any == TREE_WIDE ? k_shadow<TREE_WIDE> : k_shadow<TREE_BINARY>;
}

// ------------------------------------------------------------------ host driver
struct WfRun {
    // one wavefront engine: pool buffers + captured graphs of 1 to kItersPerGraph iterations
    WfConfig cfg;
    WfPool w{};
    void* mem = nullptr;
    WfScene* d_scenes = nullptr;
    int cap_scenes = 0;
    float4* samples = nullptr;                 // per-sample buffer, grown on demand
    size_t samples_bytes = 0;
    float4* acc = nullptr;                     // per-pixel compensated sums, grown on demand
    size_t acc_bytes = 0;
    cudaStream_t stream = nullptr;
    int grid_regen = 0, grid_shade = 0, grid_shade_m = 0, grid_shade_r = 0, grid_sort = 0;
    int grid_ext[3] = {}, grid_shadow[3] = {};   // by tree
    size_t stack_smem = 0;                     // shared traversal stack of one block
    WfState* h_state = nullptr;                // pinned: [0] as read back, [1] as uploaded
    WfScene* h_scenes = nullptr;               // pinned scene table
    static constexpr int kItersPerGraph = 8;
    static constexpr int kStages = 5;          // regen, extend, sort, shade, shadow
    cudaEvent_t e0 = nullptr, e1 = nullptr;    // around a whole render
    // by iterations and kind of pass: one that refills its slots, one that fits the pool, and one of
    // at most kSmallPass paths, whose launches need few blocks (box scene at depth 5, 128 x 128 with 1 / 4 samples
    // 334 / 359 us against 346 / 371 without it, 256 x 256 with 2 / 4 samples 384 / 468 against 395 / 460;
    // 20,480 triangles, the same four 700 / 761 / 817 / 901 against 716 / 778 / 828 / 900)
    enum Kind : int { REFILL = 0, FITS = 1, SMALL = 2 };
    // and by the trees traversed: scenes on either side of their limits share an engine and its pool
    cudaGraphExec_t exec[kItersPerGraph + 1][3][3][3] = {};
    static constexpr uint32_t kSmallPass = 1u << 18;

    int launches_per_iteration() const { return cfg.sort ? 6 : 4; }

    cudaError_t init(const WfConfig& c, int nscenes, cudaStream_t s) {
        cfg = c;
        stream = s;
        const size_t P = c.pool;
        const size_t bytes = P * (12 * sizeof(float4) + 8 * sizeof(uint32_t) + 1) + 21 * 256 + sizeof(WfState);
        cudaError_t e = cudaMalloc(&mem, bytes);
        if (e != cudaSuccess) return e;
        char* p = (char*)mem;
        auto take = [&](size_t n) { char* r = p; p += (n + 255) & ~(size_t)255; return (void*)r; };
        float4** pairs[] = {&w.ray, &w.hitid, &w.tplo, &w.neeA, &w.neeB, &w.neeC};
        for (float4** q : pairs) *q = (float4*)take(2 * P * sizeof(float4));
        w.q_regen = (uint32_t*)take(P * 4);
        w.q_ext0 = (uint32_t*)take(P * 4);
        w.q_ext1 = (uint32_t*)take(P * 4);
        w.q_sort = (uint32_t*)take(P * 4);
        w.q_shadow = (uint32_t*)take(2 * P * 4);   // up to two next-event rays per slot
        w.sh_vis = (uint32_t*)take(P * 4);
        w.rec_cur = (uint32_t*)take(P * 4);
        w.bucket = (uint8_t*)take(P);
        w.st = (WfState*)take(sizeof(WfState));
        w.ctr = w.st->ctr;
        if ((size_t)(p - (char*)mem) > bytes) return cudaErrorMemoryAllocation;
        cap_scenes = std::max(nscenes, 64);
        e = cudaMalloc(&d_scenes, sizeof(WfScene) * cap_scenes);
        if (e != cudaSuccess) return e;
        w.scenes = d_scenes;
        w.P = (uint32_t)P;
        e = cudaMallocHost(&h_state, 2 * sizeof(WfState));
        if (e == cudaSuccess) e = cudaMallocHost(&h_scenes, sizeof(WfScene) * cap_scenes);
        if (e == cudaSuccess) e = cudaEventCreate(&e0);
        if (e == cudaSuccess) e = cudaEventCreate(&e1);
        if (e != cudaSuccess) return e;
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        stack_smem = (size_t)kSharedDepth * c.block * sizeof(int);
        auto persist = [&](const void* fn, size_t smem) {
            int nb = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, c.block, smem);
            return std::max(1, nb) * sms;
        };
        for (int t = TREE_BINARY; t <= TREE_QUANT; ++t) {
            WfConfig ct = c;
            ct.tree = ct.tree_any = t;
            grid_ext[t] = persist((const void*)extend_kernel(ct), stack_smem);
            grid_shadow[t] = persist((const void*)shadow_kernel(ct), stack_smem);
        }
        grid_shade = persist(c.record ? (const void*)k_shade<true, SHADE_ALL> : (const void*)k_shade<false, SHADE_ALL>, 0);
        grid_shade_m = persist(c.record ? (const void*)k_shade<true, SHADE_MATTE> : (const void*)k_shade<false, SHADE_MATTE>, 0);
        grid_shade_r = persist(c.record ? (const void*)k_shade<true, SHADE_REST> : (const void*)k_shade<false, SHADE_REST>, 0);
        grid_sort = persist((const void*)k_sort_scatter, 0);
        grid_regen = (int)std::min<size_t>((P + c.block - 1) / c.block, (size_t)sms * 64);
        return cudaSuccess;
    }

    Kind kind_of(uint32_t total) const { return total > w.P ? REFILL : total > kSmallPass ? FITS : SMALL; }

    void regen(int in_q, Kind kind) {
        const int grid = kind == SMALL ? std::min(grid_regen, (int)(kSmallPass / 4 / cfg.block)) : grid_regen;
        auto kern = kind == REFILL ? (cfg.record ? k_regen<true, true> : k_regen<false, true>)
                                   : (cfg.record ? k_regen<true, false> : k_regen<false, false>);
        kern<<<grid, cfg.block, 0, stream>>>(w, in_q);
    }

    void enqueue_iteration(int in_q, Kind kind) {
        const int cap = kind == SMALL ? (int)(kSmallPass / cfg.block) : INT_MAX;
        const bool sweep = kind == REFILL;
        regen(in_q, kind);
        extend_kernel(cfg)<<<std::min(grid_ext[cfg.tree], cap), cfg.block, stack_smem, stream>>>(w, in_q);
        if (cfg.sort) {   // the matte bucket, then the others
            k_sort_scatter<<<std::min(grid_sort, cap), cfg.block, 0, stream>>>(w, in_q);
            auto matte = cfg.record ? k_shade<true, SHADE_MATTE> : k_shade<false, SHADE_MATTE>;
            auto rest = cfg.record ? k_shade<true, SHADE_REST> : k_shade<false, SHADE_REST>;
            matte<<<std::min(grid_shade_m, cap), cfg.block, 0, stream>>>(w, in_q, 1, sweep);
            rest<<<std::min(grid_shade_r, cap), cfg.block, 0, stream>>>(w, in_q, 1, sweep);
        } else {
            auto all = cfg.record ? k_shade<true, SHADE_ALL> : k_shade<false, SHADE_ALL>;
            all<<<std::min(grid_shade, cap), cfg.block, 0, stream>>>(w, in_q, 0, sweep);
        }
        shadow_kernel(cfg)<<<std::min(grid_shadow[cfg.tree_any], cap), cfg.block, stack_smem, stream>>>(w);
    }

    cudaError_t launch_graph(int iters, Kind kind) {
        cudaGraphExec_t& x = exec[iters][kind][cfg.tree][cfg.tree_any];
        if (!x) {
            cudaGraph_t g;
            cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
            if (e != cudaSuccess) return e;
            for (int it = 0; it < iters; ++it) enqueue_iteration(it & 1, kind);
            if (iters == kItersPerGraph) k_stage_end<<<1, 1, 0, stream>>>(w);
            e = cudaStreamEndCapture(stream, &g);
            if (e != cudaSuccess) return e;
            e = cudaGraphInstantiate(&x, g, 0);
            cudaGraphDestroy(g);
            if (e != cudaSuccess) { x = nullptr; return e; }
        }
        return cudaGraphLaunch(x, stream);
    }

    // Uploads the first n entries of h_scenes and the pass's counters; `reset` also clears what a
    // render sums over its passes.
    cudaError_t begin_pass(uint32_t total, int n, bool reset) {
        WfState& h = h_state[1];
        memset(&h, 0, sizeof(h));
        h.ctr[C_TOTAL] = total;
        h.ctr[C_FRESH] = 1;
        h.ctr[C_SCENES] = (uint32_t)n;
        h.stage = -1;
        cudaError_t e = cudaMemcpyAsync(d_scenes, h_scenes, sizeof(WfScene) * n, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(w.st, &h, reset ? sizeof(WfState) : offsetof(WfState, rays), cudaMemcpyHostToDevice, stream);
        // the sweep reads every slot's flags: none set from a pass before
        if (e == cudaSuccess && kind_of(total) == REFILL) e = cudaMemsetAsync(w.q_regen, 0, (size_t)w.P * 4, stream);
        return e;
    }
    cudaError_t read_state() {
        return cudaMemcpyAsync(&h_state[0], w.st, sizeof(WfState), cudaMemcpyDeviceToHost, stream);
    }

    // Runs one pass over `total` work items of the uploaded scene table, whose paths have at most
    // `depth` rays. A pass that fits the pool starts all its paths in its first iteration and is
    // done after `depth` of them: one graph of that many, nothing to wait for. A larger one runs
    // graphs of kItersPerGraph iterations and reads the counters between them. The stream is not
    // synchronised at the end; drained() tells after that, and after read_state(), whether the
    // pass finished.
    cudaError_t run_pass(uint32_t total, int depth, uint64_t* launches) {
        const Kind kind = kind_of(total);
        cudaError_t e = cudaSuccess;
        if (kind != REFILL && depth <= kItersPerGraph) {   // as graph_iters
            e = launch_graph(depth, kind);
            if (e != cudaSuccess) return e;
            *launches += depth * launches_per_iteration() + (depth == kItersPerGraph ? 1 : 0);
        } else {
            // Bound on graph launches: each launch advances every live path by 8 bounces
            // and refills the pool, so a pass needs about total / P * depth / 8 launches.
            const uint64_t max_launches = (uint64_t)total * 64ull / ((uint64_t)w.P) + 4096ull;
            bool done = false;
            for (uint64_t it = 0; it < max_launches && !done; ++it) {
                e = launch_graph(kItersPerGraph, kind);
                if (e == cudaSuccess) e = read_state();
                if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
                if (e != cudaSuccess) return e;
                *launches += kItersPerGraph * launches_per_iteration() + 1;
                done = drained(total, kItersPerGraph);
            }
            if (!done) return cudaErrorLaunchTimeout;
        }
        regen(0, kind);   // writes the last finished samples
        *launches += 1;
        return cudaGetLastError();
    }
    // By the counters as last read, after `iters` iterations of the last graph: no work left and
    // no ray in the queue that the next iteration would take.
    bool drained(uint32_t total, int iters) const {
        const uint32_t* c = h_state[0].ctr;
        return c[C_WORK] >= total && c[iters & 1 ? C_EXT1 : C_EXT0] == 0;
    }
    int graph_iters(uint32_t total, int depth) const {
        return total <= w.P && depth <= kItersPerGraph ? depth : kItersPerGraph;
    }

    cudaError_t ensure_samples(size_t bytes) {
        if (bytes <= samples_bytes) return cudaSuccess;
        if (samples) cudaFree(samples);
        samples = nullptr;
        samples_bytes = 0;
        cudaError_t e = cudaMalloc(&samples, bytes);
        if (e == cudaSuccess) samples_bytes = bytes;
        return e;
    }

    cudaError_t ensure_acc(size_t bytes) {
        if (bytes <= acc_bytes) return cudaSuccess;
        if (acc) cudaFree(acc);
        acc = nullptr;
        acc_bytes = 0;
        cudaError_t e = cudaMalloc(&acc, bytes);
        if (e == cudaSuccess) acc_bytes = bytes;
        return e;
    }

    void release() {
        if (acc) cudaFree(acc);
        acc = nullptr;
        acc_bytes = 0;
        for (cudaGraphExec_t* x = &exec[0][0][0][0]; x != &exec[0][0][0][0] + sizeof(exec) / sizeof(*x); ++x) {
            if (*x) cudaGraphExecDestroy(*x);
            *x = nullptr;
        }
        if (mem) cudaFree(mem);
        if (d_scenes) cudaFree(d_scenes);
        if (samples) cudaFree(samples);
        samples = nullptr;
        samples_bytes = 0;
        if (h_state) cudaFreeHost(h_state);
        if (h_scenes) cudaFreeHost(h_scenes);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        mem = nullptr; d_scenes = nullptr; h_state = nullptr; h_scenes = nullptr; e0 = e1 = nullptr;
    }
};

struct BatchItem {
    aur_scene* scene;
    PathParams p;
    uint32_t npix;
    float4* film;
    float4* acc_s;
    float4* acc_c;
    uint32_t lsub() const { return p.light_samples > 1 ? (uint32_t)p.light_samples : 1u; }
    // sub-samples of one camera sample of every pixel (the sample buffer's unit)
    uint64_t items_per_sample() const { return (uint64_t)npix * lsub(); }
    // paths traced for spp samples from sample_offset (the render's sample 0 traces one): the
    // work items of a pass
    uint64_t paths(int spp, int offset) const {
        return (uint64_t)npix * ((uint64_t)spp * lsub() - (offset == 0 && spp > 0 ? lsub() - 1 : 0));
    }
    // rays on the longest path: one per vertex, and with an environment light the one after the last
    int depth() const {
        int rays = p.max_depth;
        for (const Light& l : scene->h_lights) if (l.type == LIGHT_ENV) return rays + 1;
        return rays;
    }
};
static int max_rays(const std::vector<BatchItem>& items) {
    int d = 1;
    for (const BatchItem& it : items) d = std::max(d, it.depth());
    return d;
}

// Fills the scene table of one pass: samples [s0, s0 + chunk) of every scene. Returns the
// number of work items.
static uint32_t fill_table(std::vector<BatchItem>& items, int s0, int chunk, float4* samples, WfScene* tab) {
    uint32_t base = 0;
    size_t off = 0;
    for (size_t i = 0; i < items.size(); ++i) {
        WfScene& t = tab[i];
        const BatchItem& it = items[i];
        memset(&t, 0, sizeof(t));
        t.sc = it.scene->dev();
        t.p = it.p;
        const int pass_spp = std::max(0, std::min(chunk, it.p.spp - s0));
        t.p.spp = pass_spp;
        t.p.sample_offset = it.p.sample_offset + s0;
        t.key = seed_key(it.p.seed);
        t.npix = it.npix;
        t.lsub = it.lsub();
        t.rng_offset = (uint32_t)t.p.sample_offset * t.lsub;
        t.item_base = base;
        t.items = (uint32_t)it.paths(pass_spp, t.p.sample_offset);
        t.samples = samples ? samples + off : nullptr;
        t.film = it.film;
        t.acc_s = it.acc_s;
        t.acc_c = it.acc_c;
        t.total_spp = it.p.spp;
        t.first_pass = s0 == 0;
        t.last_pass = s0 + pass_spp >= it.p.spp;
        base += t.items;
        off += (size_t)it.items_per_sample() * chunk;
    }
    return base;
}

// Engines (pool buffers, captured graphs, events, sample buffer) are cached per (context,
// configuration) and reused by later calls; aur_ctx_destroy releases them, and so does a call
// that finds no memory for its own. A context's engines are used by one call at a time (wf_mutex).
static std::mutex g_engine_mutex;
using EngineKey = std::tuple<aur_ctx*, uint32_t, int, int, int>;
static std::map<EngineKey, std::unique_ptr<WfRun>> g_engines;
static EngineKey engine_key(aur_ctx* ctx, const WfConfig& c) { return EngineKey(ctx, c.pool, c.block, c.sort, c.record); }

// Gives back what the context holds for later calls: its engines but `keep`, and the free blocks of the
// device's stream-ordered pool.
static void wf_reclaim(aur_ctx* ctx, const WfRun* keep) {
    {
        std::lock_guard<std::mutex> lock(g_engine_mutex);
        for (auto it = g_engines.begin(); it != g_engines.end();) {
            if (std::get<0>(it->first) == ctx && it->second.get() != keep) { it->second->release(); it = g_engines.erase(it); }
            else ++it;
        }
    }
    cudaStreamSynchronize(ctx->stream);
    cudaStreamSynchronize(ctx->work_stream);
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, ctx->device) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
    cudaGetLastError();
}

static WfRun* engine_for(aur_ctx* ctx, const WfConfig& cfg, int nscenes, cudaError_t* err) {
    const EngineKey key = engine_key(ctx, cfg);
    {
        std::lock_guard<std::mutex> lock(g_engine_mutex);
        auto it = g_engines.find(key);
        if (it != g_engines.end() && it->second->cap_scenes >= nscenes) {
            it->second->cfg = cfg;                    // its trees are this call's
            return it->second.get();
        }
        if (it != g_engines.end()) { it->second->release(); g_engines.erase(it); }
    }
    std::unique_ptr<WfRun> r(new WfRun());
    *err = r->init(cfg, nscenes, ctx->work_stream);
    if (*err == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        r->release();
        wf_reclaim(ctx, nullptr);
        *err = r->init(cfg, nscenes, ctx->work_stream);
    }
    if (*err != cudaSuccess) { r->release(); return nullptr; }
    std::lock_guard<std::mutex> lock(g_engine_mutex);
    return (g_engines[key] = std::move(r)).get();
}

// The engine of a configuration, or where its pool does not fit the device and the caller did not ask for
// it, of the largest halving that does (cfg->pool; the films are the same).
static WfRun* engine_that_fits(aur_ctx* ctx, WfConfig* cfg, int nscenes, cudaError_t* err) {
    WfRun* r = engine_for(ctx, *cfg, nscenes, err);
    while (!r && *err == cudaErrorMemoryAllocation && !cfg->fixed_pool && cfg->pool > kMinPool) {
        cudaGetLastError();
        cfg->pool /= 2;
        r = engine_for(ctx, *cfg, nscenes, err);
    }
    return r;
}

static void wf_drop_engine(aur_ctx* ctx, const WfConfig& cfg) {
    std::lock_guard<std::mutex> lock(g_engine_mutex);
    auto it = g_engines.find(engine_key(ctx, cfg));
    if (it != g_engines.end()) { it->second->release(); g_engines.erase(it); }
}

// Autotuner: times candidates (pool size, material sort, block size) on the same probe, the first
// `limit` work items of the real workload (at most 2^25), and keeps the fastest: first the pool
// sizes with the sort on and blocks of 256, then the best pool without the sort, then the better of
// those with blocks of 128. (All twenty combinations take twice the time and chose one of these
// on every workload here.) Pools larger than twice the probe are not tried. More paths in flight hide
// more of the traversal's fetch latency, 1080p terrain frame at 2^21 / 2^22 / 2^23 / 2^24 / 2^25 slots:
// 204.6 / 196.1 / 189.6 / 185.2 / 183.3 ms. The largest (7.5 GB) is tried only where all paths fit
// it and not the next smaller: a batch of 25.6 M paths 25.6 -> 22.9 ms.
// Returns the chosen configuration.
static aur_status autotune(aur_ctx* ctx, std::vector<BatchItem>& items, WfConfig* best_out) {
    cudaStream_t s = ctx->work_stream;
    size_t per_sample = 0;
    uint64_t total = 0;
    for (auto& it : items) {
        per_sample += (size_t)it.items_per_sample() * sizeof(float4);
        total += it.items_per_sample() * it.p.spp;
    }
    uint32_t limit = (uint32_t)std::min<uint64_t>(total, 1ull << 25);
    int chunk = 1;   // samples buffer large enough for the probe's first `limit` items
    {
        uint64_t covered = 0;
        while (covered < limit) {
            covered = 0;
            for (auto& it : items) covered += it.items_per_sample() * std::min(chunk, it.p.spp);
            ++chunk;
        }
    }
    float4* samples = nullptr;
    cudaError_t e = cudaMallocAsync(&samples, per_sample * chunk, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        wf_reclaim(ctx, nullptr);
        e = cudaMallocAsync(&samples, per_sample * chunk, s);
    }
    if (e != cudaSuccess) return cuda_fail(e, "wavefront autotune");
    std::vector<WfScene> tab(items.size());
    limit = std::min(limit, fill_table(items, 0, chunk, samples, tab.data()));
    const int depth = max_rays(items), n = (int)items.size();
    double best = -1.0;
    WfConfig bestc;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto probe = [&](uint32_t pool, int sort, int block) {
        if (e != cudaSuccess) return;
        WfConfig c;
        c.pool = pool;
        c.block = block;
        c.sort = sort;
        tree_for(items, &c);
        WfRun run;
        e = run.init(c, n, s);
        if (e == cudaSuccess) memcpy(run.h_scenes, tab.data(), sizeof(WfScene) * n);
        uint64_t l = 0;
        auto pass = [&](uint32_t items_in_pass) {
            cudaError_t pe = run.begin_pass(items_in_pass, n, true);
            if (pe == cudaSuccess) pe = cudaEventRecord(e0, s);
            if (pe == cudaSuccess) pe = run.run_pass(items_in_pass, depth, &l);
            if (pe == cudaSuccess) pe = cudaEventRecord(e1, s);
            const cudaError_t se = cudaStreamSynchronize(s);
            return pe != cudaSuccess ? pe : se;
        };
        // a short probe runs twice: the first pass also builds its graph
        if (e == cudaSuccess && limit <= (1u << 22)) e = pass(limit);
        if (e == cudaSuccess) e = pass(limit);
        float ms = 0.f;
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        run.release();
        if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); e = cudaSuccess; return; }
        const double rate = ms > 0.f ? limit / ms : 0.0;
        if (e == cudaSuccess && rate > best) { best = rate; bestc = c; }
    };
    for (uint32_t pool = 1u << 20; pool <= (1u << 24); pool <<= 1) {
        if (pool > (1u << 20) && (uint64_t)pool > 2ull * limit) break;   // a pool that would stay mostly empty
        probe(pool, 1, 256);
    }
    if (total > (1ull << 24) && total <= (1ull << 25)) probe(1u << 25, 1, 256);
    if (best >= 0) probe(bestc.pool, 0, 256);
    if (best >= 0) probe(bestc.pool, bestc.sort, 128);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFreeAsync(samples, s);
    cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "wavefront autotune");
    if (best < 0) return fail(AUR_ERR_OOM, "wavefront autotune: no configuration fits in device memory");
    *best_out = bestc;
    return AUR_OK;
}

void wf_release_context(aur_ctx* ctx) {
    std::lock_guard<std::mutex> lock(g_engine_mutex);
    for (auto it = g_engines.begin(); it != g_engines.end();) {
        if (std::get<0>(it->first) == ctx) { it->second->release(); it = g_engines.erase(it); }
        else ++it;
    }
}

static void tree_for(const std::vector<BatchItem>& items, WfConfig* cfg) {
    int largest = 0;
    cfg->tree = cfg->tree_any = TREE_BINARY;
    for (const BatchItem& it : items) {
        if (!AUR_WIDE_TRAVERSAL || !it.scene->bvh.bvh.nodes4) return;
        largest = std::max(largest, it.scene->bvh.bvh.num_nodes4);
    }
    cfg->tree = largest >= kQuantMinNodes4 ? TREE_QUANT : TREE_WIDE;
    cfg->tree_any = largest >= kQuantMinNodes4Any ? TREE_QUANT : TREE_WIDE;
}

// Renders a batch of scenes with the wavefront engine into items[i].film (device float4[npix]).
static aur_status wavefront_batch(aur_ctx* ctx, std::vector<BatchItem>& items, const WfConfig& cfg_in,
                                  aur_render_stats* stats) {
    const int n = (int)items.size();
    WfConfig cfg = cfg_in;
    tree_for(items, &cfg);
    // The engine runs on the context's own non-blocking stream (graph capture is not
    // allowed on the legacy default stream), ordered after the caller's stream.
    cudaStream_t s = ctx->work_stream;
    cudaEventRecord(ctx->ev_order, ctx->stream);
    cudaStreamWaitEvent(s, ctx->ev_order, 0);
    cudaError_t e = cudaSuccess;
    WfRun* engine = engine_that_fits(ctx, &cfg, n, &e);
    if (!engine) return cuda_fail(e, "wavefront: pool allocation");
    WfRun& run = *engine;
    // sample-buffer budget: passes over the spp range when all samples do not fit
    const size_t budget = (size_t)3 << 30;
    size_t per_sample = 0;
    int max_spp = 0;
    uint32_t max_pix = 0;
    for (auto& it : items) {
        per_sample += (size_t)it.items_per_sample() * sizeof(float4);
        max_spp = std::max(max_spp, it.p.spp);
        max_pix = std::max(max_pix, it.npix);
    }
    const int chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)max_spp, budget / std::max<size_t>(per_sample, 1)));
    e = run.ensure_samples(per_sample * chunk);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        wf_reclaim(ctx, &run);
        e = run.ensure_samples(per_sample * chunk);
    }
    if (chunk < max_spp) {   // several passes: two float4 sums per pixel between them
        size_t pixels = 0;
        for (auto& it : items) pixels += it.npix;
        if (e == cudaSuccess) e = run.ensure_acc(2 * pixels * sizeof(float4));
        size_t off = 0;
        for (auto& it : items) {
            it.acc_s = run.acc + off;
            it.acc_c = run.acc + off + it.npix;
            off += 2 * (size_t)it.npix;
        }
    }
    if (e != cudaSuccess) return cuda_fail(e, "wavefront: sample buffers");
    const int depth = max_rays(items);
    uint64_t launches = 0;
    cudaEventRecord(run.e0, s);
    for (int s0 = 0; s0 < max_spp && e == cudaSuccess; s0 += chunk) {
        const uint32_t total = fill_table(items, s0, chunk, run.samples, run.h_scenes);
        e = run.begin_pass(total, n, s0 == 0);
        if (e == cudaSuccess) e = run.run_pass(total, depth, &launches);
        if (e != cudaSuccess) break;
        for (int i = 0; i < n; i += 65535) {
            const dim3 grid((unsigned)std::min<uint32_t>((max_pix + 255) / 256, 1u << 20), (unsigned)std::min(n - i, 65535));
            k_resolve<<<grid, 256, 0, s>>>(run.d_scenes + i, run.w.st);
            ++launches;
        }
        e = cudaGetLastError();
        const bool last = s0 + chunk >= max_spp;
        if (e == cudaSuccess && last) e = cudaEventRecord(run.e1, s);
        if (e == cudaSuccess) e = run.read_state();
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // the scene table is rewritten next pass
        if (e == cudaSuccess && !run.drained(total, run.graph_iters(total, depth))) e = cudaErrorLaunchTimeout;
    }
    float ms = 0.f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, run.e0, run.e1);
    const WfState& hs = run.h_state[0];
    const unsigned long long rays[2] = {hs.rays[0], hs.rays[1]};
    cudaEventRecord(ctx->ev_order, s);              // the caller's stream continues after this work
    cudaStreamWaitEvent(ctx->stream, ctx->ev_order, 0);
    double stage[WfRun::kStages];
    for (int k = 0; k < WfRun::kStages; ++k) stage[k] = 1e-6 * (double)hs.stage_ns[k];
    if (e != cudaSuccess) wf_drop_engine(ctx, cfg);   // never reuse an engine left in an unknown state
    if (e == cudaErrorLaunchTimeout) return fail(AUR_ERR_TIMEOUT, "wavefront: the path pool did not drain");
    if (e != cudaSuccess) return cuda_fail(e, "wavefront");
    if (stats) {
        uint64_t paths = 0, cams = 0;
        for (auto& it : items) { paths += it.paths(it.p.spp, it.p.sample_offset); cams += (uint64_t)it.npix * it.p.spp; }
        stats->paths = paths;
        stats->camera_rays = cams;   // camera samples; with light samples every path retraces its camera ray
        stats->closest_rays = rays[0];
        stats->shadow_rays = rays[1];
        stats->launches = launches;
        stats->kernel_ms = ms;
        for (int k = 0; k < WfRun::kStages; ++k) stats->stage_ms[k] = stage[k];
        stats->wf_pool = (int32_t)cfg.pool;
        stats->wf_block = cfg.block;
        stats->wf_sort = cfg.sort;
        stats->node_bytes = (int32_t)(cfg.tree == TREE_QUANT ? sizeof(BvhNode4Q) : cfg.tree == TREE_WIDE ? sizeof(BvhNode4) : sizeof(BvhNode));
    }
    return AUR_OK;
}

// Record pass of the path-replay adjoint: traces samples [s0, s0 + nsamples) of every
// pixel with the wavefront engine in record mode and writes, per item (sample-major:
// sl * npix + pixel), the records of its vertices (p.max_depth of `stride` float4s) and its
// unclamped radiance. Ordered after the caller's stream and before its later work.
aur_status wf_record_pass(aur_scene* sc, const PathParams& p, int s0, int nsamples, float4* rec, int stride,
                          float4* lo_raw, uint64_t* launches, unsigned long long* rays) {
    aur_ctx* ctx = sc->ctx;
    std::lock_guard<std::mutex> lock(ctx->wf_mutex);
    WfConfig cfg;
    if (sc->wf_tuned) { cfg.pool = (uint32_t)sc->wf_pool; cfg.block = sc->wf_block; cfg.sort = sc->wf_sort; }
    cfg.record = 1;
    std::vector<BatchItem> items(1);
    items[0] = {sc, p, (uint32_t)sc->cam.w * (uint32_t)sc->cam.h, nullptr, nullptr, nullptr};
    tree_for(items, &cfg);
    cudaStream_t s = ctx->work_stream;
    cudaEventRecord(ctx->ev_order, ctx->stream);
    cudaStreamWaitEvent(s, ctx->ev_order, 0);
    cudaError_t e = cudaSuccess;
    WfRun* engine = engine_that_fits(ctx, &cfg, 1, &e);
    if (!engine) return cuda_fail(e, "adjoint record pass: pool allocation");
    WfRun& run = *engine;
    const uint32_t total = fill_table(items, s0, nsamples, nullptr, run.h_scenes);
    run.h_scenes[0].rec = rec;
    run.h_scenes[0].lo_raw = lo_raw;
    run.h_scenes[0].rec_depth = (uint32_t)p.max_depth;
    run.h_scenes[0].rec_stride = (uint32_t)stride;
    e = run.begin_pass(total, 1, true);
    if (e == cudaSuccess) e = run.run_pass(total, max_rays(items), launches);
    if (e == cudaSuccess) e = run.read_state();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // the host table and counters are reused
    if (e == cudaSuccess && !run.drained(total, run.graph_iters(total, max_rays(items)))) e = cudaErrorLaunchTimeout;
    const unsigned long long r[2] = {run.h_state[0].rays[0], run.h_state[0].rays[1]};
    cudaEventRecord(ctx->ev_order, s);
    cudaStreamWaitEvent(ctx->stream, ctx->ev_order, 0);
    if (e != cudaSuccess) wf_drop_engine(ctx, cfg);
    if (e == cudaErrorLaunchTimeout) return fail(AUR_ERR_TIMEOUT, "adjoint record pass: the path pool did not drain");
    if (e != cudaSuccess) return cuda_fail(e, "adjoint record pass");
    rays[0] += r[0];
    rays[1] += r[1];
    return AUR_OK;
}

static bool wants_tuning(const aur_render_opts* o) { return o->wf_pool == 0 && o->wf_block == 0 && o->wf_sort < 0; }

static WfConfig config_from(const aur_render_opts* o, const WfConfig& base) {
    WfConfig c = base;
    if (o->wf_pool > 0) { c.pool = (uint32_t)o->wf_pool; c.fixed_pool = true; }
    if (o->wf_block > 0) c.block = o->wf_block;
    if (o->wf_sort >= 0) c.sort = o->wf_sort;
    return c;
}

static aur_status check_config(const WfConfig& c) {
    if (c.pool < 1024 || c.pool > (1u << 26) || (c.pool & 31))
        return fail(AUR_ERR_INVALID_ARG, "wavefront: pool must be a multiple of 32 in [1024, 2^26]");
    if (c.block != 64 && c.block != 128 && c.block != 256)   // the stage kernels take at most 256
        return fail(AUR_ERR_INVALID_ARG, "wavefront: block must be 64, 128 or 256");
    return AUR_OK;
}

aur_status render_wavefront(aur_scene* sc, const aur_render_opts* o, float* film, aur_render_stats* stats) {
    if (!sc || !o || !film) return fail(AUR_ERR_INVALID_ARG, "aur_render: NULL argument");
    PathParams p;
    aur_status st = render_options(sc, o, &p);
    if (st != AUR_OK) return st;
    if (o->count_work) return fail(AUR_ERR_UNSUPPORTED, "aur_render: count_work is implemented by the plain renderer");
    WfConfig cfg = config_from(o, WfConfig());
    if ((st = check_config(cfg)) != AUR_OK) return st;
    DeviceGuard g(sc->ctx->device);
    std::lock_guard<std::mutex> lock(sc->ctx->wf_mutex);
    cudaStream_t s = sc->ctx->stream;
    const uint32_t npix = (uint32_t)sc->cam.w * sc->cam.h;
    if ((uint64_t)npix * o->spp * (uint64_t)p.light_samples >= (1ull << 31))
        return fail(AUR_ERR_INVALID_ARG, "aur_render: more than 2^31 paths");
    DevOut fo;
    cudaError_t e = fo.init(film, sizeof(float4) * npix, 16, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // film staging allocated on the caller's stream
    if (e != cudaSuccess) return cuda_fail(e, "aur_render(wavefront)");
    std::vector<BatchItem> items(1);
    items[0] = {sc, p, npix, (float4*)fo.ptr, nullptr, nullptr};
    if (wants_tuning(o)) {
        // Tuned once per render shape (triangles, materials, lights, resolution, spp, light samples,
        // depths) on this context: a scene rendered at another spp or depth is tuned for that too,
        // and a new scene of the same shape reuses the configuration. The first sample of a render
        // has one path whatever the light samples, so a render that has it is another shape.
        uint64_t sig = 1469598103934665603ull;
        const uint64_t parts[10] = {sc->ntri, sc->h_mats.size(), sc->h_lights.size(), (uint64_t)sc->cam.w,
                                    (uint64_t)sc->cam.h, (uint64_t)o->spp, (uint64_t)o->max_depth,
                                    (uint64_t)(int64_t)o->min_depth, (uint64_t)p.light_samples,
                                    (uint64_t)(p.light_samples > 1 && p.sample_offset == 0)};
        for (uint64_t v : parts) sig = (sig ^ v) * 1099511628211ull;
        auto it = sc->ctx->wf_scene_tuned.find(sig);
        if (it == sc->ctx->wf_scene_tuned.end()) {
            WfConfig t;
            if ((st = autotune(sc->ctx, items, &t)) != AUR_OK) return st;
            it = sc->ctx->wf_scene_tuned.emplace(sig, std::array<int, 3>{(int)t.pool, t.block, t.sort}).first;
        }
        sc->wf_pool = it->second[0]; sc->wf_block = it->second[1]; sc->wf_sort = it->second[2];
        sc->wf_tuned = true;
        cfg.pool = sc->wf_pool; cfg.block = sc->wf_block; cfg.sort = sc->wf_sort;
    }
    st = wavefront_batch(sc->ctx, items, cfg, stats);
    if (st == AUR_OK) {
        e = fo.finish();
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) st = cuda_fail(e, "aur_render(wavefront download)");
    }
    return st;
}

}  // namespace aur

extern "C" aur_status aur_render_batch(aur_scene* const* scenes, const aur_render_opts* opts, uint32_t n,
                                       float* const* films, aur_render_stats* stats) {
    using namespace aur;
    if (!scenes || !opts || !films || n == 0) return fail(AUR_ERR_INVALID_ARG, "aur_render_batch: NULL argument");
    aur_ctx* ctx = scenes[0] ? scenes[0]->ctx : nullptr;
    if (!ctx) return fail(AUR_ERR_INVALID_ARG, "aur_render_batch: NULL scene");
    for (uint32_t i = 0; i < n; ++i)
        if (!scenes[i] || scenes[i]->ctx != ctx || !films[i])
            return fail(AUR_ERR_INVALID_ARG, "aur_render_batch: scenes must share one context and have films");
    WfConfig cfg = config_from(&opts[0], WfConfig());
    aur_status st = check_config(cfg);
    if (st != AUR_OK) return st;
    DeviceGuard g(ctx->device);
    std::lock_guard<std::mutex> lock(ctx->wf_mutex);
    cudaStream_t s = ctx->stream;
    std::vector<BatchItem> items(n);
    std::vector<DevOut> outs(n);
    uint64_t total = 0;
    for (uint32_t i = 0; i < n; ++i) {
        PathParams p;
        if ((st = render_options(scenes[i], &opts[i], &p)) != AUR_OK) return st;
        const uint32_t npix = (uint32_t)scenes[i]->cam.w * scenes[i]->cam.h;
        total += (uint64_t)npix * p.spp * (uint64_t)p.light_samples;
        items[i] = {scenes[i], p, npix, nullptr, nullptr, nullptr};
    }
    if (total >= (1ull << 31)) return fail(AUR_ERR_INVALID_ARG, "aur_render_batch: more than 2^31 paths");
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < n && e == cudaSuccess; ++i) {
        e = outs[i].init(films[i], sizeof(float4) * items[i].npix, 16, s);
        items[i].film = (float4*)outs[i].ptr;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && wants_tuning(&opts[0])) {
        // tuned once per (scene count, path count) on this context
        const uint64_t key = ((uint64_t)n << 40) ^ total;
        auto it = ctx->wf_batch_tuned.find(key);
        if (it == ctx->wf_batch_tuned.end()) {
            WfConfig t;
            st = autotune(ctx, items, &t);
            if (st == AUR_OK) it = ctx->wf_batch_tuned.emplace(key, std::array<int, 3>{(int)t.pool, t.block, t.sort}).first;
        }
        if (st == AUR_OK) { cfg.pool = (uint32_t)it->second[0]; cfg.block = it->second[1]; cfg.sort = it->second[2]; }
    }
    if (e == cudaSuccess && st == AUR_OK) st = wavefront_batch(ctx, items, cfg, stats);
    else if (e != cudaSuccess) st = cuda_fail(e, "aur_render_batch");
    for (uint32_t i = 0; i < n && st == AUR_OK; ++i) {
        e = outs[i].finish();
        if (e != cudaSuccess) st = cuda_fail(e, "aur_render_batch(download)");
    }
    cudaStreamSynchronize(s);
    return st;
}
