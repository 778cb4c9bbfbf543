// render_paths.cu — the plain renderer with one lane per path (aur_render in plain mode,
// aur_render_f64): the estimator of Integrator::integrateCameraSample
// (Aurora/src/frontend/integrator.cpp:152-300) for every (pixel, sample), and the film's sums.
//
// The transcendentals are out of line here: this kernel is bound by instruction fetch.
#define AUR_MATH_OUT_OF_LINE 1
#include "aur_kernels.h"
#include <algorithm>
#include <type_traits>

namespace aur {
namespace {

// A resident grid of warps whose lanes take the next (pixel, sample) as soon as theirs is finished,
// one vertex of every lane's path per step: the closest-hit rays together, shading, the
// next-event rays (a lane's two in turn), continuation. The rays use the resumable while-while
// rounds, so the kernel holds one closest-hit and one any-hit traversal where the pixel loop
// inlines five. Every sample goes to a buffer and is summed per pixel in sample order
// (k_sum_samples), so the film is the pixel loop's bit for bit; rays that meet two triangles at
// exactly the same distance are traced again in the binary tree's order, which the pixel loop
// follows.
// A thread per pixel ran as many warps as the film has pixels / 32 however many samples there are,
// at 4.9 lanes an instruction: 26.0 ms for 201 x 149 x 64 samples of the shader scene. Lanes per
// path alone: 12.7 ms, warps waiting for instructions of a body much larger than the instruction
// caches, each somewhere else in it. Out-of-line transcendentals and BRDF sampling: 10.9 ms. A
// block-wide barrier between the phases, so that a block's warps run the same code together:
// 6.9 ms with 128 threads a block, 5.8 with 256, 5.6 with 512, 4.95 with two blocks of 512 (64
// registers, some spilled). 640 x 480 x 8 terrain: 20.6 -> 8.6 ms; 128 x 128 x 4: 1.6 -> 0.7 ms.
constexpr int kPathBlock = 512;

static __device__ __noinline__ bool retrace_binary(const BvhNode* nodes, const BvhTri* tris, float3 o, float3 d, float mint,
                                                   float maxt, Hit* h) {
    TraceWork w;
    return bvh_trace<false>(nodes, tris, o, d, mint, maxt, h, w);
}

// one copy for the next-event and the continuation sample
static __device__ __noinline__ BrdfSample path_brdf_sample(int lobe, float3 color, float rough, float3 V, float3 N, float r1,
                                                           float r2) {
    Brdf b;
    b.lobe = lobe;
    b.color = color;
    b.rough = rough;
    return brdf_sample(b, V, N, r1, r2);
}

// A barrier between two phases; the warp is converged first.
__device__ __forceinline__ void phase() { __syncwarp(); __syncthreads(); }

// kQuant: closest-hit rays walk the quantised tree (any-hit rays always do). kMulti: light samples.
template <bool kQuant, bool kMulti>
__global__ void __launch_bounds__(kPathBlock, 2) k_render_paths(DevScene sc, PathParams p, int s0, uint32_t items,
                                                                            float4* __restrict__ samples,
                                                                            unsigned long long* counters) {
    using Node = std::conditional_t<kQuant, BvhNode4Q, BvhNode4>;
    extern __shared__ int s_stack[];
    LaneStack4 stack;
    stack.col = s_stack + threadIdx.x;
    stack.stride = blockDim.x;
    const Node* nodes;
    if constexpr (kQuant) nodes = sc.nodes4q;
    else nodes = sc.nodes4;
    const uint32_t npix = (uint32_t)(sc.cam.w * sc.cam.h);
    const uint64_t key = seed_key(p.seed);
    const int lmax = kMulti ? p.light_samples : 1;
    uint32_t* cursor = reinterpret_cast<uint32_t*>(counters + kPathCursor);
    uint32_t closest = 0, shadow = 0;
    bool active = false, exhausted = false;
    // the lane's path
    uint32_t item = 0;
    PathRng rng;
    rng.key = key;
    rng.base = 0;
    RayF ray{};
    float3 T = mk(1.f, 1.f, 1.f), Lo = mk(0.f, 0.f, 0.f);
    float cont = 1.f;
    int kind = RAY_CAMERA, bounces = 0, vtx = 0;
    bool matte = false;
    // light samples: the camera sample's first hit, its paths so far
    Hit first{};
    float3 sum = mk(0.f, 0.f, 0.f);
    int sub = 0, nsub = 1;

    auto camera = [&]() {
        const uint32_t pixel = item % npix;
        PathRng c;
        c.key = key;
        c.base = path_base(pixel, (uint32_t)(p.sample_offset + s0 + (int)(item / npix)) * (uint32_t)lmax);
        return camera_ray(sc.cam, (int)(pixel % (uint32_t)sc.cam.w), (int)(pixel / (uint32_t)sc.cam.w), c.u(kDimCamera),
                          c.u(kDimCamera + 1));
    };
    auto begin_path = [&]() {
        T = mk(1.f, 1.f, 1.f);
        Lo = mk(0.f, 0.f, 0.f);
        cont = 1.f;
        kind = RAY_CAMERA;
        bounces = vtx = 0;
        matte = false;
        rng.base = path_base(item % npix, (uint32_t)(p.sample_offset + s0 + (int)(item / npix)) * (uint32_t)lmax + (uint32_t)sub);
    };
    while (true) {
        const uint32_t want = __ballot_sync(0xffffffffu, !active && !exhausted);
        if (want) {
            uint32_t b = 0;
            const int leader = __ffs(want) - 1, lane = threadIdx.x & 31;
            if (lane == leader) b = atomicAdd(cursor, (uint32_t)__popc(want));
            b = __shfl_sync(0xffffffffu, b, leader);
            if (!active && !exhausted) {
                item = b + __popc(want & ((1u << lane) - 1u));
                if (item < items) {
                    active = true;
                    sub = 0;
                    nsub = kMulti && p.sample_offset + s0 + (int)(item / npix) > 0 ? lmax : 1;
                    sum = mk(0.f, 0.f, 0.f);
                    begin_path();
                    ray = camera();
                } else {
                    exhausted = true;
                }
            }
        }
        __syncwarp();
        if (!__syncthreads_or(active)) break;
        // closest hits; a later path of a camera sample starts from its first hit
        Hit h;
        bool hit = false;
        {
            TraceState4<false, Node> ts;
            const bool trace = active && !(kMulti && vtx == 0 && sub > 0);
            if (trace) { ts.begin(ray.o, ray.d, ray.mint, ray.maxt); ++closest; }
            while (__ballot_sync(0xffffffffu, !ts.finished())) ts.round(nodes, sc.tris, stack);
            if (trace) {
                h.t = ts.tbest; h.u = ts.bu; h.v = ts.bv; h.prim = ts.best;
                hit = ts.best >= 0;
                if (ts.tie) hit = retrace_binary(sc.nodes, sc.tris, ray.o, ray.d, ray.mint, ray.maxt, &h);
            } else if (kMulti && active) {
                h = first;
                hit = true;
            }
        }
        phase();
        bool done = false;                 // the path is finished
        float3 L = mk(0.f, 0.f, 0.f);      // with this radiance
        float alpha = 1.f;
        bool env_sample = false;           // the camera ray saw the environment: the sample is that radiance
        // this vertex's next-event rays and what they add if unoccluded
        bool r0 = false, r1 = false;
        float3 c0 = mk(0.f, 0.f, 0.f), c1 = c0, d0 = c0, d1 = c0;
        float m0 = 0.f, m1 = 0.f;
        int nvis = 0;
        Frame f;
        Brdf brdf;
        brdf.lobe = LOBE_CONSTANT;
        bool shade = false;
        if (active && !hit) {
            done = true;
            if (vtx == 0) {
                alpha = sc.sh.nenv ? 1.f : 0.f;
                if (sc.sh.nenv) { L = env_radiance(sc.sh, ray.d); env_sample = true; }   // not firefly-filtered
            } else {
                if (kind == RAY_MIRROR && sc.sh.nenv) Lo += env_radiance(sc.sh, camera().d) * T;
                L = firefly_clamp(Lo);
            }
        } else if (active && vtx >= p.max_depth) {
            done = true;                   // the unshaded last ray hit something
            L = firefly_clamp(Lo);
        } else if (active) {
            shade = true;
            if (kMulti && vtx == 0) first = h;
            f = hit_frame(sc.sh, h.prim, h.t, h.u, h.v, ray.o, ray.d, true);
            const Attr at = sc.sh.attrs[f.attr];
            if (kind == RAY_DIFFUSE) matte = true;
            if (collects_emission(kind)) Lo += T * at.emission;
            brdf = get_brdf(sc.sh, at.material, f, matte, rng.u(vertex_dim(vtx, kDimLobe)));
        }
        // light sampling
        const bool nee = shade && (brdf.lobe == LOBE_MATTE || brdf.lobe == LOBE_SPEC);
        int li = -1;
        if (nee) li = pick_visible_light(sc.sh, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightPick)), &nvis);
        if (li >= 0) {
            const Light& light = sc.sh.lights[li];   // global: the env paths take its address
            const LightSample ls = light_sample(sc.sh, light, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightSample)),
                                                rng.u(vertex_dim(vtx, kDimLightSample + 1)));
            const float cost = dot(f.N, ls.dir);
            d0 = ls.dir;
            m0 = ls.maxt;
            if (brdf.lobe == LOBE_MATTE) {
                if (cost >= 0.f && ls.pdf > 0.f) {
                    r0 = true;
                    c0 = cdiv((ls.color * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                }
            } else if (cost > 0.f && ls.pdf > 0.f) {
                const float bp = brdf_pdf(brdf, ls.dir, f.V, f.N);
                if (bp > 0.f) {
                    r0 = true;
                    c0 = cdiv(((ls.color * power_heuristic(ls.pdf, bp)) * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                }
            }
        }
        // BRDF sampling of the light (specular lobes)
        if (li >= 0 && brdf.lobe == LOBE_SPEC) {
            const Light& light = sc.sh.lights[li];
            const BrdfSample bs = path_brdf_sample(brdf.lobe, brdf.color, brdf.rough, f.V, f.N,
                                                   rng.u(vertex_dim(vtx, kDimMisBrdf)), rng.u(vertex_dim(vtx, kDimMisBrdf + 1)));
            const float cost = dot(f.N, bs.dir);
            if (cost > 0.f) {
                float maxt = bs.maxt;
                const float lp = light_pdf(sc.sh, light, f.P, bs.dir, kRayBias, &maxt);
                if (lp > 0.f && bs.pdf > 0.f) {
                    r1 = true;
                    d1 = bs.dir;
                    m1 = maxt;
                    c1 = cdiv(((bs.color * power_heuristic(bs.pdf, lp)) * light_eval(sc.sh, light, bs.dir)) * cost, bs.pdf);
                }
            }
        }
        phase();
        float3 res = mk(0.f, 0.f, 0.f);
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            const bool r = k == 0 ? r0 : r1;
            if (__ballot_sync(0xffffffffu, r) == 0) continue;
            TraceState4<true, BvhNode4Q> ts;
            if (r) { ts.begin(f.P, k == 0 ? d0 : d1, kRayBias, k == 0 ? m0 : m1); ++shadow; }
            while (__ballot_sync(0xffffffffu, !ts.finished())) ts.round(sc.nodes4q, sc.tris, stack);
            if (r && !ts.hit_any) res += k == 0 ? c0 : c1;
        }
        phase();
        if (shade) {
            const bool lit = brdf.lobe == LOBE_MATTE || brdf.lobe == LOBE_SPEC;
            Lo += (lit && nvis ? res * (float)nvis : mk(0.f, 0.f, 0.f)) * T;
            const BrdfSample bs = path_brdf_sample(brdf.lobe, brdf.color, brdf.rough, f.V, f.N,
                                                   rng.u(vertex_dim(vtx, kDimBrdf)), rng.u(vertex_dim(vtx, kDimBrdf + 1)));
            // after the last vertex only an escaping mirror ray in a scene with an environment light is traced
            if (!continue_path(brdf, bs, f.N, p.min_depth, rng, vtx, T, cont, kind, bounces) ||
                (vtx + 1 >= p.max_depth && !(kind == RAY_MIRROR && sc.sh.nenv))) {
                done = true;
                L = firefly_clamp(Lo);
            } else {
                ray.o = f.P;
                ray.d = bs.dir;
                ray.mint = kRayBias;
                ray.maxt = bs.maxt;
                ++vtx;
            }
        }
        if (done) {
            bool whole = true;
            if (kMulti && nsub > 1 && !env_sample && !(vtx == 0 && !hit)) {
                sum += cdiv(L, (float)nsub);
                if (++sub < nsub) {
                    whole = false;
                    begin_path();
                    ray = camera();
                }
                L = sum;
            }
            if (whole) {
                samples[item] = make_float4(L.x, L.y, L.z, alpha);
                active = false;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        closest += __shfl_xor_sync(0xffffffffu, closest, o);
        shadow += __shfl_xor_sync(0xffffffffu, shadow, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&counters[1], (unsigned long long)closest);
        atomicAdd(&counters[2], (unsigned long long)shadow);
    }
}

// Adds a chunk's samples of every pixel in sample order to its sum (acc: what is kept between the
// chunks of a render, 32 bytes a pixel; null for a render of one chunk) and writes the film after
// the last one: the pixel loop's arithmetic.
template <bool kFp64>
__global__ void k_sum_samples(const float4* __restrict__ samples, int npix, int count, int spp, bool first, bool last,
                              void* acc, float4* film, double* film64) {
    const int pixel = blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= npix) return;
    Kahan3 k;
    k.init();
    double d[3] = {0.0, 0.0, 0.0};
    float alpha = 0.f;
    if (!first) {
        if (kFp64) {
            const double* a = (const double*)acc + 4 * (size_t)pixel;
            d[0] = a[0]; d[1] = a[1]; d[2] = a[2];
            alpha = (float)a[3];
        } else {
            const float4 a = ((const float4*)acc)[2 * (size_t)pixel], c = ((const float4*)acc)[2 * (size_t)pixel + 1];
            k.s = mk(a.x, a.y, a.z);
            k.c = mk(c.x, c.y, c.z);
            alpha = a.w;
        }
    }
#pragma unroll 8
    for (int s = 0; s < count; ++s) {
        const float4 v = __ldg(&samples[(size_t)s * npix + pixel]);
        if (kFp64) { d[0] += v.x; d[1] += v.y; d[2] += v.z; }
        else k.add(mk(v.x, v.y, v.z));
        alpha += v.w;
    }
    if (!last) {
        if (kFp64) {
            double* a = (double*)acc + 4 * (size_t)pixel;
            a[0] = d[0]; a[1] = d[1]; a[2] = d[2]; a[3] = (double)alpha;
        } else {
            ((float4*)acc)[2 * (size_t)pixel] = make_float4(k.s.x, k.s.y, k.s.z, alpha);
            ((float4*)acc)[2 * (size_t)pixel + 1] = make_float4(k.c.x, k.c.y, k.c.z, 0.f);
        }
        return;
    }
    const float inv = 1.f / (float)spp;
    if (kFp64) {
        if (film64) {
            film64[4 * (size_t)pixel + 0] = d[0] / spp;
            film64[4 * (size_t)pixel + 1] = d[1] / spp;
            film64[4 * (size_t)pixel + 2] = d[2] / spp;
            film64[4 * (size_t)pixel + 3] = (double)alpha / spp;
        }
        if (film) film[pixel] = make_float4((float)(d[0] / spp), (float)(d[1] / spp), (float)(d[2] / spp), alpha * inv);
    } else {
        const float3 t = k.total();
        film[pixel] = make_float4(t.x * inv, t.y * inv, t.z * inv, alpha * inv);
    }
}

}  // namespace

size_t paths_scratch_bytes(const DevScene& sc, const PathParams& p, size_t budget, int* chunk) {
    const size_t npix = (size_t)sc.cam.w * sc.cam.h;
    *chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)p.spp, budget / (npix * sizeof(float4))));
    *chunk = (int)std::min<size_t>((size_t)*chunk, std::max<size_t>(1, 0x7fffffffull / npix));
    return npix * ((size_t)*chunk * sizeof(float4) + (*chunk < p.spp ? 32 : 0));
}

cudaError_t launch_render_paths(const DevScene& sc, const PathParams& p, bool quantised, bool fp64, int chunk, void* scratch,
                                float4* film, double* film64, unsigned long long* counters, uint64_t* launches, cudaStream_t s) {
    const int npix = sc.cam.w * sc.cam.h;
    float4* samples = (float4*)scratch;
    void* acc = samples + (size_t)npix * chunk;
    const bool multi = p.light_samples > 1;
    auto kern = quantised ? (multi ? k_render_paths<true, true> : k_render_paths<true, false>)
                          : (multi ? k_render_paths<false, true> : k_render_paths<false, false>);
    const size_t smem = sizeof(int) * kSharedDepth * kPathBlock;
    int dev = 0, sms = 0, nb = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kPathBlock, smem);
    for (int s0 = 0; s0 < p.spp; s0 += chunk) {
        const int n = std::min(chunk, p.spp - s0);
        const uint32_t items = (uint32_t)npix * (uint32_t)n;
        if (s0 > 0) {
            const cudaError_t e = cudaMemsetAsync(counters + kPathCursor, 0, sizeof(unsigned long long), s);
            if (e != cudaSuccess) return e;
        }
        const int grid = (int)std::min<uint32_t>((items + kPathBlock - 1) / kPathBlock, (uint32_t)(std::max(1, nb) * sms));
        kern<<<grid, kPathBlock, smem, s>>>(sc, p, s0, items, samples, counters);
        auto sum = fp64 ? k_sum_samples<true> : k_sum_samples<false>;
        sum<<<(npix + 127) / 128, 128, 0, s>>>(samples, npix, n, p.spp, s0 == 0, s0 + n >= p.spp, acc, film, film64);
        *launches += 2;
    }
    return cudaGetLastError();
}

}  // namespace aur
