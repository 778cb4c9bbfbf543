// adjoint.cu — path-replay backpropagation (Vicini, Speierer, Jakob, "Path Replay
// Backpropagation", SIGGRAPH 2021) for the Aurora path loop. No reference counterpart.
//
// Given dLoss/dFilm, every pixel replays its spp camera paths with the same
// counter-based random numbers as the forward renderer:
//   pass 1  the forward estimator of Integrator::integrateCameraSample
//           (integrator.cpp:152-300) with identical arithmetic; it records each
//           vertex's hit (prim, t, u, v) and the visibility of its next-event
//           rays in thread-local arrays, and yields the path radiance Lo;
//   pass 2  re-shades the recorded vertices (no ray tracing) and accumulates
//             dL/dtheta += delta . [ T_k dD_k/dtheta + L_after,k (dw_k/dtheta) / w_k ]
//           where D_k is the vertex's next-event estimate, w_k = f cos / pdf its
//           continuation weight, T_k the throughput and L_after,k = Lo minus the
//           radiance collected up to and including vertex k.
// Sampling decisions are detached: pdfs, MIS weights, the Kelemen/metal lobe
// choice, roulette probabilities and the firefly clamp factor are constants of
// the derivative (the discrete choices and the clamp make the estimator biased;
// the continuous parts are unbiased). Memory: O(pixels) — nothing is stored per path.
//
// Parameters: per material (diffuse rgb, roughness) and all texels. Diffuse
// colour drives Lambert lobes (matte, Kelemen's diffuse lobe); roughness drives
// Cook-Torrance lobes (Kelemen, Cook-Torrance, metal roughnessA); a diffuse
// texture receives the diffuse gradient of the texel the lookup used. Gradients
// are summed in FP32 with TwoSum-compensated atomics (shared, then global) by the megakernel,
// in FP64 by the wavefront form, which computes a vertex's derivative factors where the wavefront
// engine shades it (record mode) instead of shading it again.
#define AUR_MATH_OUT_OF_LINE 1
#include "aur_capi_internal.h"
#include "aur_adjoint.cuh"
#include <algorithm>

namespace aur {
namespace {

constexpr int kAdjBlock = 128;
constexpr int kAdjMaxDepth = 16;
constexpr int kAdjMaxMat = 64;
constexpr size_t kRecBudget = (size_t)4 << 30;   // bytes of vertex records in one record pass

// float4s per vertex record: the three texels of a triplanar diffuse shader take two more
int record_stride(const aur_scene* sc) {
    for (const Material& m : sc->h_mats)
        if ((m.type == MAT_MATTE || m.type == MAT_KELEMEN) && m.diff_tex >= 0 && sc->h_texs[m.diff_tex].tri_scale != 0.f)
            return kVertexRec + 2;
    return kVertexRec;
}

// hit record of one vertex: (t, u, v, prim | visibility of its next-event rays << 30)
__device__ __forceinline__ float4 pack_rec(const Hit& h, uint32_t vis) {
    return make_float4(h.t, h.u, h.v, __int_as_float(h.prim | (int)(vis << 30)));
}

// atomic add with the exact rounding error of that addition sent to a compensation slot
__device__ __forceinline__ void comp_add(float* sum, float* comp, float x) {
    if (x == 0.f) return;
    const float old = atomicAdd(sum, x);
    const float t = old + x;                        // what the atomic stored
    const float bp = t - old;
    const float err = (old - (t - bp)) + (x - bp);  // TwoSum(old, x) error
    if (err != 0.f) atomicAdd(comp, err);
}

// TwoSum step of a thread-local compensated sum
__device__ __forceinline__ void two_sum_add(float& sum, float& comp, float x) {
    const float t = sum + x;
    const float bp = t - sum;
    comp += (sum - (t - bp)) + (x - bp);
    sum = t;
}

// Per-thread compensated accumulators of the per-material gradients (diffuse rgb,
// roughness) of the two most recently touched materials. A pixel's paths mostly revisit
// the same materials, so the block's shared sums see one flush per eviction instead of
// one atomic per vertex (11% faster). Register-resident: slots resolved by selects.
struct MatCache {
    int tag0 = -1, tag1 = -1;
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, c0[4] = {0.f, 0.f, 0.f, 0.f};
    float s1[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};

    __device__ __forceinline__ static void flush_slot(int tag, const float* s, const float* c, float* s_g, float* s_c) {
        if (tag < 0) return;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (s[q] != 0.f) comp_add(&s_g[4 * tag + q], &s_c[4 * tag + q], s[q]);
            if (c[q] != 0.f) comp_add(&s_g[4 * tag + q], &s_c[4 * tag + q], c[q]);
        }
    }
    __device__ __forceinline__ void flush(float* s_g, float* s_c) {
        flush_slot(tag0, s0, c0, s_g, s_c);
        flush_slot(tag1, s1, c1, s_g, s_c);
        tag0 = tag1 = -1;
    }
    // makes `mat` the tag of slot 0 (evicting slot 1 to the shared sums if needed)
    __device__ __forceinline__ bool slot0(int mat, float* s_g, float* s_c) {
        if (tag0 == mat) return true;
        if (tag1 == mat) return false;
        flush_slot(tag1, s1, c1, s_g, s_c);
        tag1 = tag0;
#pragma unroll
        for (int q = 0; q < 4; ++q) { s1[q] = s0[q]; c1[q] = c0[q]; s0[q] = 0.f; c0[q] = 0.f; }
        tag0 = mat;
        return true;
    }
    template <int Q>
    __device__ __forceinline__ void add(int mat, float x, float* s_g, float* s_c) {
        if (x == 0.f) return;
        if (slot0(mat, s_g, s_c)) two_sum_add(s0[Q], c0[Q], x);
        else two_sum_add(s1[Q], c1[Q], x);
    }
    __device__ __forceinline__ void add3(int mat, float3 v, float* s_g, float* s_c) {
        if (v.x == 0.f && v.y == 0.f && v.z == 0.f) return;
        if (slot0(mat, s_g, s_c)) { two_sum_add(s0[0], c0[0], v.x); two_sum_add(s0[1], c0[1], v.y); two_sum_add(s0[2], c0[2], v.z); }
        else { two_sum_add(s1[0], c1[0], v.x); two_sum_add(s1[1], c1[1], v.y); two_sum_add(s1[2], c1[2], v.z); }
    }
};

// Next-event estimation of one vertex (integrateDirect with integrateDirectLight /
// integrateDirectMIS). kTrace: traces the shadow rays and records their visibility
// in *vis; otherwise replays `vis`. With kGrad it also returns dD/dtheta of the lobe's
// parameter: per channel d/d(diffuse_c) for a Lambert lobe, d/d(roughness_eff) for a
// Cook-Torrance lobe (replicated in all channels).
template <bool kTrace, bool kGrad>
__device__ __forceinline__ float3 direct(const DevScene& sc, const Frame& f, const Brdf& brdf, const PathRng& rng,
                                         int vtx, RayCounts& rc, uint32_t* vis, float3* dD) {
    float3 res = mk(0.f, 0.f, 0.f), dres = res;
    if (kGrad) *dD = res;
    if (brdf.lobe != LOBE_MATTE && brdf.lobe != LOBE_SPEC) return res;
    int nvis;
    const int li = pick_visible_light(sc.sh, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightPick)), &nvis);
    if (li < 0) return res;
    const Light& L = sc.sh.lights[li];   // global: the env paths take its address
    const LightSample ls = light_sample(sc.sh, L, f.P, f.N, rng.u(vertex_dim(vtx, kDimLightSample)),
                                        rng.u(vertex_dim(vtx, kDimLightSample + 1)));
    float cost = dot(f.N, ls.dir);
    if (brdf.lobe == LOBE_MATTE) {
        if (cost >= 0.f && ls.pdf > 0.f) {
            bool open;
            if (kTrace) { ++rc.shadow; open = !bvh_occluded(sc.nodes, sc.tris, f.P, ls.dir, kRayBias, ls.maxt, rc.shadow_work); if (open) *vis |= 1u; }
            else open = (*vis & 1u) != 0;
            if (open) {
                res += cdiv((ls.color * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                if (kGrad && dot(ls.dir, f.N) > 0.f) dres += cdiv((ls.color * kInvPiMacro) * cost, ls.pdf);
            }
        }
    } else {
        if (cost > 0.f && ls.pdf > 0.f) {
            const float bp = brdf_pdf(brdf, ls.dir, f.V, f.N);
            if (bp > 0.f) {
                bool open;
                if (kTrace) { ++rc.shadow; open = !bvh_occluded(sc.nodes, sc.tris, f.P, ls.dir, kRayBias, ls.maxt, rc.shadow_work); if (open) *vis |= 1u; }
                else open = (*vis & 1u) != 0;
                if (open) {
                    const float w = power_heuristic(ls.pdf, bp);
                    const float3 c0 = cdiv(((ls.color * w) * brdf_eval(brdf, ls.dir, f.V, f.N)) * cost, ls.pdf);
                    res += c0;
                    if (kGrad) dres += c0 * eval_dlnD(brdf.rough, f.N, f.V, ls.dir);
                }
            }
        }
        const BrdfSample bs = brdf_sample(brdf, f.V, f.N, rng.u(vertex_dim(vtx, kDimMisBrdf)),
                                          rng.u(vertex_dim(vtx, kDimMisBrdf + 1)));
        cost = dot(f.N, bs.dir);
        if (cost > 0.f) {
            float maxt = bs.maxt;
            const float lp = light_pdf(sc.sh, L, f.P, bs.dir, kRayBias, &maxt);
            if (lp > 0.f && bs.pdf > 0.f) {
                bool open;
                if (kTrace) { ++rc.shadow; open = !bvh_occluded(sc.nodes, sc.tris, f.P, bs.dir, kRayBias, maxt, rc.shadow_work); if (open) *vis |= 2u; }
                else open = (*vis & 2u) != 0;
                if (open) {
                    const float w = power_heuristic(bs.pdf, lp);
                    const float3 c1 = cdiv(((bs.color * w) * light_eval(sc.sh, L, bs.dir)) * cost, bs.pdf);
                    res += c1;
                    if (kGrad) dres += c1 * sample_dlnD(brdf.rough, f.N, f.V, bs.dir);
                }
            }
        }
    }
    if (kGrad) *dD = dres * (float)nvis;
    return res * (float)nvis;
}

// The firefly clamp's factor of a path of radiance c (detached).
__device__ __forceinline__ float firefly_factor(float3 c) {
    float f = 1.f;
    for (int k = 0; k < 64 && (c.x > kFirefly || c.y > kFirefly || c.z > kFirefly); ++k) { c *= 0.2f; f *= 0.2f; }
    return f;
}

// Pass 2 of one camera path: re-shades the recorded vertices rec[0, nv) (no ray
// tracing) and accumulates dL/dtheta with delta = dLoss/dpixel / spp (/ n for one of the
// n paths of a camera sample with light samples). Lo is the path's unclamped radiance
// from pass 1; cam_rng draws the camera ray (the path's own rng but for light samples,
// whose paths share their sample's camera ray).
__device__ __forceinline__ void replay_path(const DevScene& sc, const PathParams& p, int px, int py,
                                            const PathRng& cam_rng, const PathRng& rng, const float4* rec, int nv,
                                            float3 Lo, float3 delta, MatCache& mc, float* s_g, float* s_c, float* g_tex,
                                            float* g_tex_c, RayCounts& rc) {
    if (nv == 0 || !isfinite(Lo.x) || !isfinite(Lo.y) || !isfinite(Lo.z)) return;
    const float3 dp = delta * firefly_factor(Lo);
    RayF ray = camera_ray(sc.cam, px, py, cam_rng.u(kDimCamera), cam_rng.u(kDimCamera + 1));
    float3 T = mk(1.f, 1.f, 1.f), collected = mk(0.f, 0.f, 0.f);
    float cont = 1.f;
    bool matte = false;
    int kind = RAY_CAMERA, bounces = 0;
    for (int vtx = 0; vtx < nv; ++vtx) {
        const float4 r = rec[vtx];
        const uint32_t bits = __float_as_uint(r.w);
        const int prim = (int)(bits & 0x3fffffffu);
        uint32_t vis = bits >> 30;
        const Frame f = hit_frame(sc.sh, prim, r.x, r.y, r.z, ray.o, ray.d, true);
        const Attr at = sc.sh.attrs[f.attr];
        if (kind == RAY_DIFFUSE) matte = true;
        if (collects_emission(kind)) collected += T * at.emission;
        const float lobe_u = rng.u(vertex_dim(vtx, kDimLobe));
        const Brdf brdf = get_brdf(sc.sh, at.material, f, matte, lobe_u);
        const ParamRef pr = param_of(sc.sh, at.material, brdf, f, matte, lobe_u);
        float3 dD;
        const float3 D = direct<false, true>(sc, f, brdf, rng, vtx, rc, &vis, &dD);
        collected += D * T;
        const float3 gdir = T * dD;
        const BrdfSample bs = brdf_sample(brdf, f.V, f.N, rng.u(vertex_dim(vtx, kDimBrdf)),
                                          rng.u(vertex_dim(vtx, kDimBrdf + 1)));
        float3 gcont = mk(0.f, 0.f, 0.f);
        float3 w = mk(0.f, 0.f, 0.f);
        const bool cont_ok = bs.pdf > 0.f;
        const float3 after = Lo - collected;
        const Material mat = sc.sh.mats[at.material];
        if (mat.type == MAT_KELEMEN && mat.refl < 1.f && mat.rough_tex < 0) {
            // the lobe choice depends on roughness: score-function term on the subtree radiance
            const float score = kelemen_score(sc.sh, mat, f, brdf, matte);
            const float3 sub = dp * (D * T + after);
            mc.add<3>(at.material, score * (sub.x + sub.y + sub.z), s_g, s_c);
        }
        if (cont_ok && pr.kind != 0) {
            const float cosl = dot(f.N, bs.dir);
            w = cdiv(bs.color * cosl, bs.pdf);
            if (pr.kind == 3) {
                const float g = sample_dlnD(brdf.rough, f.N, f.V, bs.dir);   // dw/w = d ln f
                gcont = after * g;
            } else {
                const float dw = kInvPiMacro * cosl / bs.pdf;  // d w_c / d diffuse_c
                gcont = mk(w.x != 0.f ? after.x * dw / w.x : 0.f, w.y != 0.f ? after.y * dw / w.y : 0.f,
                           w.z != 0.f ? after.z * dw / w.z : 0.f);
            }
        }
        if (pr.kind == 1 || pr.kind == 2) {
            const float3 g = dp * (gdir + gcont);
            if (pr.kind == 1) {
                mc.add3(pr.index, g, s_g, s_c);
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int i = pr.taps.idx[k];
                    const float wk = pr.taps.w[k];
                    if (!(wk > 0.f)) continue;
                    comp_add(&g_tex[3 * i + 0], &g_tex_c[3 * i + 0], g.x * wk);
                    comp_add(&g_tex[3 * i + 1], &g_tex_c[3 * i + 1], g.y * wk);
                    comp_add(&g_tex[3 * i + 2], &g_tex_c[3 * i + 2], g.z * wk);
                }
            }
        } else if (pr.kind == 3) {
            const float3 g = dp * (gdir * pr.dr + gcont * pr.dr);
            mc.add<3>(pr.index, g.x + g.y + g.z, s_g, s_c);
        }
        // the forward update, identical to pass 1
        if (!continue_path(brdf, bs, f.N, p.min_depth, rng, vtx, T, cont, kind, bounces)) break;
        ray.o = f.P; ray.d = bs.dir; ray.mint = kRayBias; ray.maxt = bs.maxt;
    }
}

// the block's material gradients (sum and compensation) go to the global ones
__device__ __forceinline__ void flush_block(const float* s_g, const float* s_c, int nmat, float* g_mat, float* g_mat_c) {
    __syncthreads();
    for (int i = threadIdx.x; i < nmat * 4; i += blockDim.x) {
        comp_add(&g_mat[i], &g_mat_c[i], s_g[i]);
        comp_add(&g_mat[i], &g_mat_c[i], s_c[i]);
    }
}

// The environment seen by a mirror ray traced after the last shaded vertex (zero when the ray
// hits anything in [RAY_BIAS, maxt]); out of line, as the case is rare.
__device__ __noinline__ float3 escape_after_last(const BvhNode* nodes, const BvhTri* tris, const Light* lights,
                                                 int nlights, const Texture* texs, const float* texels, float3 P,
                                                 float3 dir, float maxt, float3 cam_d) {
    TraceWork w;
    if (bvh_occluded(nodes, tris, P, dir, kRayBias, maxt, w)) return mk(0.f, 0.f, 0.f);
    return env_radiance_of(lights, nlights, texs, texels, cam_d);
}

// Megakernel form: one thread per pixel runs, for each of its camera samples, pass 1
// (forward with tracing, records in thread-local memory) and pass 2 of each path. With
// light samples a camera sample's n paths start at its camera ray's first hit (traced
// once) and draw from sample indices s * L + j (integrate_camera_sample). kMulti: light
// samples above one; the one-path form keeps a single path per sample (no inner loop), whose
// code is smaller and faster. kEnv: the scene has an environment light; only then is the ray
// after the last vertex traced (any code for it in the loop made the kernel 8% slower on
// scenes without one).
template <bool kMulti, bool kEnv>
__global__ void __launch_bounds__(kAdjBlock) k_adjoint(DevScene sc, PathParams p, const float4* __restrict__ dfilm,
                                                       int nmat, float* g_mat, float* g_mat_c, float* g_tex,
                                                       float* g_tex_c, unsigned long long* counters) {
    __shared__ float s_g[kAdjMaxMat * 4], s_c[kAdjMaxMat * 4];
    for (int i = threadIdx.x; i < nmat * 4; i += blockDim.x) { s_g[i] = 0.f; s_c[i] = 0.f; }
    __syncthreads();
    const int npix = sc.cam.w * sc.cam.h;
    const int pixel = blockIdx.x * blockDim.x + threadIdx.x;
    const int lmax = kMulti && p.light_samples > 1 ? p.light_samples : 1;
    RayCounts rc;
    MatCache mc;
    // paths traced for this pixel: the render's sample 0 has one, every other sample lmax
    const uint32_t paths = pixel < npix ? (uint32_t)(p.spp * lmax - (p.sample_offset == 0 ? lmax - 1 : 0)) : 0u;
    if (pixel < npix) {
        const float4 df = dfilm[pixel];
        const float inv = 1.f / (float)p.spp;
        const float3 delta = mk(df.x * inv, df.y * inv, df.z * inv);
        const int px = pixel % sc.cam.w, py = pixel / sc.cam.w;
        PathRng cam_rng;
        cam_rng.key = seed_key(p.seed);
        const bool any = delta.x != 0.f || delta.y != 0.f || delta.z != 0.f;
        for (int s = 0; any && s < p.spp; ++s) {
            const int pass = p.sample_offset + s;
            const int n = kMulti ? (pass == 0 ? 1 : lmax) : 1;
            cam_rng.base = path_base((uint32_t)pixel, (uint32_t)(pass * lmax));
            RayF ray0 = camera_ray(sc.cam, px, py, cam_rng.u(kDimCamera), cam_rng.u(kDimCamera + 1));
            const float3 cam_d = ray0.d;
            Hit h0;
            ++rc.closest;
            if (!bvh_closest(sc.nodes, sc.tris, ray0.o, ray0.d, ray0.mint, ray0.maxt, &h0, rc.work)) continue;
            const float3 dn = n > 1 ? delta * (1.f / (float)n) : delta;
            for (int j = 0; j < n; ++j) {
                PathRng rng = cam_rng;
                rng.base = path_base((uint32_t)pixel, (uint32_t)(pass * lmax + j));
                // ---------------- pass 1: forward, recording hits and visibility
                float4 rec[kAdjMaxDepth];
                int nv = 0;
                float3 Lo = mk(0.f, 0.f, 0.f);
                {
                    RayF ray = ray0;
                    Hit h = h0;
                    float3 T = mk(1.f, 1.f, 1.f);
                    float cont = 1.f;
                    bool matte = false;
                    int kind = RAY_CAMERA, bounces = 0;
                    for (int vtx = 0; vtx < p.max_depth; ++vtx) {
                        nv = vtx + 1;
                        const Frame f = hit_frame(sc.sh, h.prim, h.t, h.u, h.v, ray.o, ray.d, true);
                        const Attr at = sc.sh.attrs[f.attr];
                        if (kind == RAY_DIFFUSE) matte = true;
                        if (collects_emission(kind)) Lo += T * at.emission;
                        const Brdf brdf = get_brdf(sc.sh, at.material, f, matte,
                                                   rng.u(vertex_dim(vtx, kDimLobe)));
                        uint32_t vis = 0;
                        Lo += direct<true, false>(sc, f, brdf, rng, vtx, rc, &vis, nullptr) * T;
                        rec[vtx] = pack_rec(h, vis);
                        const BrdfSample bs = brdf_sample(brdf, f.V, f.N, rng.u(vertex_dim(vtx, kDimBrdf)),
                                                          rng.u(vertex_dim(vtx, kDimBrdf + 1)));
                        if (!continue_path(brdf, bs, f.N, p.min_depth, rng, vtx, T, cont, kind, bounces)) break;
                        if (vtx + 1 >= p.max_depth) {
                            // the reference's unshaded last ray: only an escaping mirror ray adds
                            // anything, the environment (integrator.cpp:256-274); replay sees it in Lo
                            if constexpr (kEnv) {
                                if (kind == RAY_MIRROR) {
                                    ++rc.closest;
                                    Lo += escape_after_last(sc.nodes, sc.tris, sc.sh.lights, sc.sh.nlights,
                                                            sc.sh.texs, sc.sh.texels, f.P, bs.dir, bs.maxt, cam_d) * T;
                                }
                            }
                            break;
                        }
                        ray.o = f.P; ray.d = bs.dir; ray.mint = kRayBias; ray.maxt = bs.maxt;
                        ++rc.closest;
                        if (!bvh_closest(sc.nodes, sc.tris, ray.o, ray.d, ray.mint, ray.maxt, &h, rc.work)) {
                            if (kEnv && kind == RAY_MIRROR) Lo += env_radiance(sc.sh, cam_d) * T;
                            break;
                        }
                    }
                }
                // ---------------- pass 2: re-shade the recorded vertices, accumulate gradients
                // one path per sample: its own generator drew the camera ray (cam_rng is no longer live)
                replay_path(sc, p, px, py, kMulti ? cam_rng : rng, rng, rec, nv, Lo, dn, mc, s_g, s_c, g_tex,
                            g_tex_c, rc);
            }
        }
    }
    mc.flush(s_g, s_c);
    flush_block(s_g, s_c, nmat, g_mat, g_mat_c);
    unsigned long long v[3] = {rc.closest, rc.shadow, paths};
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; ++k) atomicAdd(&counters[k], v[k]);
}

// Replay form (pass 2 over a record pass): one thread per path walks the vertex records that the
// wavefront engine's record mode wrote (VertexRec; the derivative factors of a vertex were computed
// where it was shaded), and needs nothing but the path's radiance to finish them. Items are
// sub-sample-major: q * npix + pixel with q = sl * L + j, L = max(1, light_samples), camera sample
// p.sample_offset + s0 + sl; the sub-samples j > 0 of the render's sample 0 were not traced.
// Re-shading every vertex here instead took 28 of the 62 ms of a 256 x 256, 256 sample texture
// adjoint, its warps waiting for instructions (28 per issue) of a large body that ran 8 of 32
// lanes. What is left is bound by the records' 64 B per vertex and the texels' atomics.
// Sums are in FP64: per thread column of shared memory and then one global add per block for the
// materials (`cols` columns; threads share one where all of them do not fit), one reduction to the
// L2 per texel channel.
__global__ void __launch_bounds__(kAdjBlock) k_adjoint_replay(PathParams p, uint32_t npix, int s0, uint32_t items,
                                                              const float4* __restrict__ rec, int stride,
                                                              const float4* __restrict__ lo_raw,
                                                              const float4* __restrict__ dfilm, int nmat, int cols,
                                                              double* g_mat, double* g_tex) {
    extern __shared__ double s_acc[];   // [4 nmat][cols]
    for (int i = threadIdx.x; i < 4 * nmat * cols; i += blockDim.x) s_acc[i] = 0.0;
    __syncthreads();
    double* col = s_acc + threadIdx.x % cols;
    auto add = [&](int param, float x) {
        if (x == 0.f) return;
        if (cols == kAdjBlock) col[(size_t)param * cols] += (double)x;   // the thread's own column
        else atomicAdd(&col[(size_t)param * cols], (double)x);
    };
    const uint32_t lsub = p.light_samples > 1 ? (uint32_t)p.light_samples : 1u;
    const float inv = 1.f / (float)p.spp;
    for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < items; item += gridDim.x * blockDim.x) {
        const uint32_t pixel = item % npix, q = item / npix;
        const uint32_t j = q % lsub, sample = (uint32_t)(p.sample_offset + s0) + q / lsub;
        const uint32_t n = sample == 0 ? 1u : lsub;
        if (j >= n) continue;
        const float4 df = dfilm[pixel], lo = lo_raw[item];
        const int nv = __float_as_int(lo.w);
        float3 delta = mk(df.x * inv, df.y * inv, df.z * inv);
        if (n > 1) delta = delta * (1.f / (float)n);
        if (delta.x == 0.f && delta.y == 0.f && delta.z == 0.f) continue;
        const float3 Lo = mk(lo.x, lo.y, lo.z);
        if (!isfinite(Lo.x) || !isfinite(Lo.y) || !isfinite(Lo.z)) continue;
        const float3 dp = delta * firefly_factor(Lo);
        const float4* r = rec + (size_t)item * p.max_depth * stride;
        for (int v = 0; v < nv; ++v, r += stride) {
            const float4 r3 = __ldg(r + 3);
            const uint32_t meta = __float_as_uint(r3.w);
            const int kind = (int)(meta & 3u), index = (int)(meta >> 2);
            if (kind == 0) continue;
            const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
            const float3 after = Lo - mk(r0.x, r0.y, r0.z);
            const float3 g = dp * (mk(r1.x, r1.y, r1.z) + after * mk(r3.x, r3.y, r3.z));
            if (r2.w != 0.f) {   // the lobe choice depends on roughness: score-function term on the subtree radiance
                const float3 sub = dp * (Lo - mk(r2.x, r2.y, r2.z));
                add(4 * __float_as_int(r0.w) + 3, r2.w * (sub.x + sub.y + sub.z));
            }
            if (kind == 1) {
                add(4 * index, g.x);
                add(4 * index + 1, g.y);
                add(4 * index + 2, g.z);
            } else if (kind == 3) {
                add(4 * index + 3, g.x + g.y + g.z);
            } else {
                auto tap = [&](int t, float w) {
                    if (!(w > 0.f)) return;
                    if (g.x != 0.f) atomicAdd(&g_tex[3 * (size_t)t], (double)(g.x * w));
                    if (g.y != 0.f) atomicAdd(&g_tex[3 * (size_t)t + 1], (double)(g.y * w));
                    if (g.z != 0.f) atomicAdd(&g_tex[3 * (size_t)t + 2], (double)(g.z * w));
                };
                if (stride == kVertexRec) {
                    tap(index, 1.f);
                } else {
                    const float4 ti = __ldg(r + 4), tw = __ldg(r + 5);
                    tap(__float_as_int(ti.x), tw.x);
                    tap(__float_as_int(ti.y), tw.y);
                    tap(__float_as_int(ti.z), tw.z);
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * nmat; i += blockDim.x) {
        double sum = 0.0;
        for (int c = 0; c < cols; ++c) sum += s_acc[(size_t)i * cols + (c + i) % cols];
        if (sum != 0.0) atomicAdd(&g_mat[i], sum);
    }
}

__global__ void k_to_float(const double* g, float* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)g[i];
}

__global__ void k_add_comp(float* g, const float* c, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) g[i] += c[i];
}

}  // namespace
}  // namespace aur

using namespace aur;

extern "C" aur_status aur_render_adjoint(aur_scene* sc, const aur_render_opts* o, const float* dfilm, float* grad_mat,
                                         float* grad_tex, aur_render_stats* stats) {
    if (!sc || !o || !dfilm || !grad_mat) return fail(AUR_ERR_INVALID_ARG, "aur_render_adjoint: NULL argument");
    if (sc->ntexel_floats && !grad_tex) return fail(AUR_ERR_INVALID_ARG, "aur_render_adjoint: grad_tex is NULL");
    PathParams p;
    aur_status st = render_options(sc, o, &p);
    if (st != AUR_OK) return st;
    if (o->mode != AUR_RENDER_PLAIN && o->mode != AUR_RENDER_WAVEFRONT)
        return fail(AUR_ERR_INVALID_ARG, "aur_render_adjoint: unknown mode");
    const bool wavefront = o->mode == AUR_RENDER_WAVEFRONT;
    // the megakernel keeps a path's hit records in registers / local memory; the wavefront
    // form records them in device memory and takes any depth
    if (!wavefront && o->max_depth > kAdjMaxDepth)
        return fail(AUR_ERR_UNSUPPORTED, "aur_render_adjoint: max_depth above 16 needs mode AUR_RENDER_WAVEFRONT");
    if (sc->ntri >= (1u << 30)) return fail(AUR_ERR_UNSUPPORTED, "aur_render_adjoint: 2^30 triangles or more");
    const int nmat = (int)sc->h_mats.size();
    if (nmat > kAdjMaxMat) return fail(AUR_ERR_UNSUPPORTED, "aur_render_adjoint: more than 64 materials");
    DeviceGuard g(sc->ctx->device);
    cudaStream_t s = sc->ctx->stream;
    const size_t npix = (size_t)sc->cam.w * sc->cam.h;
    const int ntex = (int)sc->ntexel_floats;
    DevIn din;
    DevOut gm, gt;
    DevBuf counters, records;              // this call's own
    // the sums beside the outputs: compensation terms (megakernel) or the FP64 sums themselves
    const int nsum = 4 * nmat + ntex;
    const size_t sum_bytes = (wavefront ? sizeof(double) : sizeof(float)) * nsum;
    void* sums = nullptr;
    cudaError_t e = din.init(dfilm, sizeof(float4) * npix, 16, s);
    if (e == cudaSuccess) e = gm.init(grad_mat, sizeof(float) * 4 * nmat, 4, s);
    if (e == cudaSuccess && ntex) e = gt.init(grad_tex, sizeof(float) * ntex, 4, s);
    if (e == cudaSuccess) e = cudaMallocAsync(&sums, sum_bytes, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(sums, 0, sum_bytes, s);
    if (e == cudaSuccess && !wavefront) e = cudaMemsetAsync(gm.ptr, 0, sizeof(float) * 4 * nmat, s);
    if (e == cudaSuccess && !wavefront && ntex) e = cudaMemsetAsync(gt.ptr, 0, sizeof(float) * ntex, s);
    if (e == cudaSuccess) e = counters.init(sizeof(unsigned long long) * 8, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(counters.ptr, 0, sizeof(unsigned long long) * 8, s);
    float* cm = (float*)sums;
    float* ct = cm ? cm + 4 * nmat : nullptr;
    double* dm = (double*)sums;
    double* dt = dm ? dm + 4 * nmat : nullptr;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    cudaEvent_t er0, er1;   // replay kernels alone (wavefront mode)
    cudaEventCreate(&er0);
    cudaEventCreate(&er1);
    double replay_ms = 0.0;
    uint64_t launches = 0;
    unsigned long long rays[2] = {0, 0};
    if (wavefront) {
        // record passes (wavefront engine) + replay kernels over chunks of the samples, sized so that
        // the records stay within kRecBudget and their indices within 2^31; where the device has less
        // memory left, the chunk is halved until its records fit
        const size_t lsub = (size_t)p.light_samples;   // items per pixel and camera sample
        const int stride = record_stride(sc);
        const size_t per_item = sizeof(float4) * ((size_t)p.max_depth * stride + 1);
        const size_t per_spp = npix * lsub;
        int chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)p.spp, kRecBudget / (per_item * per_spp)));
        while (chunk > 1 && (size_t)chunk * per_spp * (p.max_depth + 1) >= (1ull << 31)) chunk /= 2;
        if ((size_t)chunk * per_spp * (p.max_depth + 1) >= (1ull << 31)) e = cudaErrorInvalidValue;
        // as many passes as the budget needs, of equal size
        chunk = (p.spp + (p.spp + chunk - 1) / chunk - 1) / ((p.spp + chunk - 1) / chunk);
        while (e == cudaSuccess) {
            e = records.init(per_item * per_spp * chunk, s);
            if (e != cudaErrorMemoryAllocation || chunk == 1) break;
            cudaGetLastError();
            e = cudaSuccess;
            chunk = (chunk + 1) / 2;
        }
        float4* rec = (float4*)records.ptr;
        float4* lo_raw = rec ? rec + per_spp * chunk * p.max_depth * stride : nullptr;
        // a column of shared sums per thread, or as many as fit 48 KB
        const int cols = std::min<int>(kAdjBlock, (int)(48 * 1024 / (sizeof(double) * 4 * nmat)));
        const size_t smem = sizeof(double) * 4 * nmat * cols;
        int sms = 0, nb = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, sc->ctx->device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_adjoint_replay, kAdjBlock, smem);
        for (int s0 = 0; s0 < p.spp && e == cudaSuccess; s0 += chunk) {
            const int n = std::min(chunk, p.spp - s0);
            aur_status rs = wf_record_pass(sc, p, s0, n, rec, stride, lo_raw, &launches, rays);
            if (rs != AUR_OK) {
                if (sums) cudaFreeAsync(sums, s);
                cudaEventDestroy(e0);
                cudaEventDestroy(e1);
                cudaEventDestroy(er0);
                cudaEventDestroy(er1);
                return rs;
            }
            const uint32_t items = (uint32_t)(per_spp * (size_t)n);
            const unsigned grid = std::min<unsigned>((items + kAdjBlock - 1) / kAdjBlock, (unsigned)(std::max(1, nb) * sms));
            cudaEventRecord(er0, s);
            k_adjoint_replay<<<grid, kAdjBlock, smem, s>>>(p, (uint32_t)npix, s0, items, rec, stride, lo_raw,
                                                           (const float4*)din.ptr, nmat, cols, dm, dt);
            ++launches;
            e = cudaGetLastError();
            cudaEventRecord(er1, s);
            if (e == cudaSuccess) e = cudaEventSynchronize(er1);
            float rms = 0.f;
            if (e == cudaSuccess && cudaEventElapsedTime(&rms, er0, er1) == cudaSuccess) replay_ms += rms;
        }
    } else if (e == cudaSuccess) {
        const unsigned grid = (unsigned)((npix + kAdjBlock - 1) / kAdjBlock);
        const DevScene dsc = sc->dev();
        auto kern = p.light_samples > 1 ? (dsc.sh.nenv ? k_adjoint<true, true> : k_adjoint<true, false>)
                                        : (dsc.sh.nenv ? k_adjoint<false, true> : k_adjoint<false, false>);
        kern<<<grid, kAdjBlock, 0, s>>>(dsc, p, (const float4*)din.ptr, nmat, (float*)gm.ptr, cm,
                                        ntex ? (float*)gt.ptr : nullptr, ct, (unsigned long long*)counters.ptr);
        ++launches;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && wavefront) {
        k_to_float<<<(4 * nmat + 255) / 256, 256, 0, s>>>(dm, (float*)gm.ptr, 4 * nmat);
        ++launches;
        if (ntex) { k_to_float<<<(ntex + 255) / 256, 256, 0, s>>>(dt, (float*)gt.ptr, ntex); ++launches; }
        e = cudaGetLastError();
    } else if (e == cudaSuccess) {
        k_add_comp<<<(4 * nmat + 255) / 256, 256, 0, s>>>((float*)gm.ptr, cm, 4 * nmat);
        ++launches;
        if (ntex) { k_add_comp<<<(ntex + 255) / 256, 256, 0, s>>>((float*)gt.ptr, ct, ntex); ++launches; }
        e = cudaGetLastError();
    }
    cudaEventRecord(e1, s);
    if (e == cudaSuccess) e = gm.finish();
    if (e == cudaSuccess && ntex) e = gt.finish();
    // paths traced: the render's sample 0 traces one path, every other camera sample L
    const unsigned long long lpaths = (unsigned long long)p.light_samples;
    unsigned long long cnt[3] = {rays[0], rays[1],
                                 (unsigned long long)npix * ((unsigned long long)p.spp * lpaths -
                                                             (p.sample_offset == 0 ? lpaths - 1 : 0))};
    if (e == cudaSuccess && !wavefront)
        e = cudaMemcpyAsync(cnt, counters.ptr, sizeof(cnt), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    float ms = 0.f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaEventDestroy(er0);
    cudaEventDestroy(er1);
    if (sums) cudaFreeAsync(sums, s);
    if (e != cudaSuccess) return cuda_fail(e, "aur_render_adjoint");
    if (stats) {
        *stats = aur_render_stats{};
        stats->closest_rays = cnt[0];
        stats->shadow_rays = cnt[1];
        stats->paths = cnt[2];
        stats->camera_rays = (unsigned long long)npix * p.spp;
        stats->launches = launches;
        stats->kernel_ms = ms;
        if (wavefront) {   // stage_ms[0]: record passes (and the rest), stage_ms[1]: replay kernels
            stats->stage_ms[1] = replay_ms;
            stats->stage_ms[0] = ms - replay_ms;
            std::lock_guard<std::mutex> lock(sc->ctx->wf_mutex);
            if (sc->wf_tuned) { stats->wf_pool = sc->wf_pool; stats->wf_block = sc->wf_block; stats->wf_sort = sc->wf_sort; }
        }
    }
    return AUR_OK;
}
