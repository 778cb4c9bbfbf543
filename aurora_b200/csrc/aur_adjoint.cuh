// aur_adjoint.cuh — the derivatives of one path vertex that both forms of the path-replay adjoint
// use: which parameter a vertex's lobe depends on, and the logarithmic derivatives of the
// Cook-Torrance lobe and of Kelemen's lobe choice (adjoint.cu has the estimator).
#pragma once
#include "aur_integrator.cuh"

namespace aur {

// ln D derivative w.r.t. roughness r of the Beckmann term, with tan^2(alpha) given
// and the reference's max(0.001, r^2) floor (eval uses r^2 unfloored).
__device__ __forceinline__ float dlnD_dr(float r, float tan2, bool floored) {
    const float r2 = r * r;
    if (floored && r2 <= 0.001f) return 0.f;
    return 2.f * tan2 / (r2 * r) - 2.f / r;
}
__device__ __forceinline__ float tan2_of(float ndoth) {
    const float t = xtan_acosf(ndoth);
    return t * t;
}

// d ln f / d roughness of the Cook-Torrance lobe's value towards L (cookTorrance.cpp:125-144).
__device__ __forceinline__ float eval_dlnD(float rough, float3 N, float3 V, float3 L) {
    const float3 H = normalize(L + V);
    return dlnD_dr(rough, tan2_of(dot(H, N)), false);
}

// d ln f / d roughness of a Cook-Torrance sample (cookTorrance.cpp:47-99): the sampled
// half vector is normalize(L + V); a clamped D (>= 1000) or the 0.001 floor on r^2
// makes the sample's colour independent of roughness.
__device__ __forceinline__ float sample_dlnD(float rough, float3 N, float3 V, float3 L) {
    const float3 H = normalize(L + V);
    const float ndoth = dot(N, H);
    const float tana = ndoth > 0.999f ? 0.f : xtan_acosf(ndoth);
    if (ct_d(rough, ndoth, tana) >= 1000.f) return 0.f;
    return dlnD_dr(rough, tana * tana, true);
}

// d A / d roughness of the Kelemen directional-albedo lookup (kelemen_albedo): the
// lookup is linear in roughness * 31 between the two columns it reads.
__device__ __forceinline__ float kelemen_dalbedo_dr(const float* table, float costheta, float roughness) {
    int i = aur_floor(costheta * (kAlbedoCos - 1));
    int ra = aur_floor(roughness * (kAlbedoRough - 1));
    int rb = ra + 1 > kAlbedoRough - 1 ? ra + 1 : kAlbedoRough - 1;
    i = i < 0 ? 0 : (i > kAlbedoCos - 1 ? kAlbedoCos - 1 : i);
    ra = ra < 0 ? 0 : (ra > kAlbedoRough - 1 ? kAlbedoRough - 1 : ra);
    rb = rb > kAlbedoRough - 1 ? kAlbedoRough - 1 : rb;
    const int i1 = i + 1 < kAlbedoCos - 1 ? i + 1 : kAlbedoCos - 1;
    const float mixc = costheta * (kAlbedoCos - 1) - (float)i;
    const float resA = (1.f - mixc) * table[i * kAlbedoRough + ra] + mixc * table[i1 * kAlbedoRough + ra];
    const float resB = (1.f - mixc) * table[i * kAlbedoRough + rb] + mixc * table[i1 * kAlbedoRough + rb];
    return (resB - resA) * (float)(kAlbedoRough - 1);
}

// Score-function factor d ln P(chosen lobe) / d roughness of Kelemen's lobe choice
// (kelemenMaterial.cpp:236-253): P(spec) = min(1, A(cos, r_eff)), P(diffuse) = 1 - A.
__device__ __forceinline__ float kelemen_score(const ShadeScene& sh, const Material& m, const Frame& f, const Brdf& b,
                                               bool matte) {
    float r = m.rough;
    if (matte) r = caustic_blur(r);
    float c = dot(f.N, f.V);
    c = c < 0.f ? 0.f : (c > 1.f ? 1.f : c);
    const float* table = sh.albedo + (size_t)m.table * (kAlbedoCos * kAlbedoRough);
    const float A = kelemen_albedo(table, c, r);
    const float dA = kelemen_dalbedo_dr(table, c, r) * (matte ? (float)(1.0 - 0.2) : 1.f);
    if (b.lobe == LOBE_SPEC) return A < 1.f && A > 0.f ? dA / A : 0.f;
    return A < 1.f ? -dA / (1.f - A) : 0.f;
}

// Which parameter a vertex's lobe depends on.
struct ParamRef {
    int kind;        // 0 none, 1 diffuse colour of material `index`, 2 texels `taps`, 3 roughness
    int index;
    float dr;        // roughness: d r_eff / d r (caustic blur on matte paths)
    Taps taps;       // kind 2: texel blocks (3 floats each, index from the texel array start) and
                     // the weights the shader blends them with (1 for the uv lookup; 0 = unused)
};

__device__ __forceinline__ ParamRef param_of(const ShadeScene& sh, int mat_id, const Brdf& b, const Frame& f,
                                             bool matte, float lobe_u) {
    ParamRef p;
    p.kind = 0; p.index = 0; p.dr = 0.f;
    for (int k = 0; k < 3; ++k) { p.taps.idx[k] = 0; p.taps.w[k] = 0.f; }
    const Material m = sh.mats[mat_id];
    if (b.lobe == LOBE_MATTE) {
        if (m.type != MAT_MATTE && m.type != MAT_KELEMEN) return p;
        if (m.diff_tex >= 0) {
            const Texture t = sh.texs[m.diff_tex];
            p.kind = 2;
            if (t.tri_scale == 0.f) {
                p.taps.idx[0] = uv_texel_index(t, f.su, f.sv);
                p.taps.w[0] = 1.f;
            } else {
                p.taps = triplanar_taps(sh.attr_c2o + (size_t)f.attr * 16, t, f.P, f.Ng, false);
            }
            for (int k = 0; k < 3; ++k) p.taps.idx[k] += t.offset / 3;
        } else {
            p.kind = 1;
            p.index = mat_id;
        }
        return p;
    }
    if (b.lobe == LOBE_SPEC && m.rough_tex < 0 &&
        (m.type == MAT_KELEMEN || m.type == MAT_COOKTORRANCE || (m.type == MAT_METAL && lobe_u > m.mix))) {
        p.kind = 3;
        p.index = mat_id;
        p.dr = matte ? (float)(1.0 - 0.2) : 1.f;
    }
    return p;
}

}  // namespace aur
