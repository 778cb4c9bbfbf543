// accel.cu — the full contract of EmbreeAccelerator::intersect for arrays of rays
// (Aurora/src/geometry/embreeAccelerator.cpp:41-91): closest hit, then the hit's
// post-process with the per-corner normals and uvs the mesh retains
// (EmbreeMesh::normals / uvs, geometry/embreeMesh.h:62-63):
//   w = 1. - u - v (in double, rounded to float)
//   hitP = org + dir * t
//   hitN = normalize(w n0 + u n1 + v n2), negated first when it faces along dir
//   st   = w st0 + u st1 + v st2
//   barCoords = (u, v, w); ray.maxt = t on a hit (embreeAccelerator.cpp:56)
// The arithmetic is the shading frame's (hit_frame), so a hit reported here and the
// same hit shaded by the renderers agree bit for bit.
#include "aur_capi_internal.h"

namespace aur {
namespace {

constexpr int kIsectBlock = 128;

__global__ void k_pack_tri_shade(const float* __restrict__ cn, const float* __restrict__ cu, const int* __restrict__ attr,
                                 size_t ntri, TriShade* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntri) return;
    TriShade r;
    for (int k = 0; k < 9; ++k) r.n[k] = cn[9 * i + k];
    for (int k = 0; k < 6; ++k) r.uv[k] = cu ? cu[6 * i + k] : 0.f;
    r.attr = attr ? attr[i] : 0;
    float4* o = reinterpret_cast<float4*>(out + i);
    o[0] = make_float4(r.n[0], r.n[1], r.n[2], r.n[3]);
    o[1] = make_float4(r.n[4], r.n[5], r.n[6], r.n[7]);
    o[2] = make_float4(r.n[8], __int_as_float(r.attr), r.uv[0], r.uv[1]);
    o[3] = make_float4(r.uv[2], r.uv[3], r.uv[4], r.uv[5]);
}

__global__ void __launch_bounds__(kIsectBlock) k_intersect(const BvhNode* __restrict__ nodes,
                                                           const BvhNode4* __restrict__ nodes4,
                                                           const BvhTri* __restrict__ tris,
                                                           const TriShade* __restrict__ tri, float4* rays,
                                                           aur_isect* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = rays[2 * i];
    const float4 b = rays[2 * i + 1];
    const float3 o = mk(a.x, a.y, a.z), d = mk(b.x, b.y, b.z);
    Hit h;
    TraceWork work;
    aur_isect r;
    if (!bvh_closest(nodes, nodes4, tris, o, d, a.w, b.w, &h, work)) {
        r.t = b.w; r.u = r.v = 0.f; r.prim = -1; r.attr = -1;
        for (int k = 0; k < 3; ++k) { r.hitP[k] = 0.f; r.hitN[k] = 0.f; r.bar[k] = 0.f; }
        r.st[0] = r.st[1] = 0.f;
        out[i] = r;
        return;
    }
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
    const float s = w * uv[0] + h.u * uv[2] + h.v * uv[4];
    const float t = w * uv[1] + h.u * uv[3] + h.v * uv[5];
    r.t = h.t; r.u = h.u; r.v = h.v; r.prim = h.prim;
    r.attr = ts.attr;
    r.hitP[0] = P.x; r.hitP[1] = P.y; r.hitP[2] = P.z;
    r.hitN[0] = N.x; r.hitN[1] = N.y; r.hitN[2] = N.z;
    r.st[0] = s; r.st[1] = t;
    r.bar[0] = h.u; r.bar[1] = h.v; r.bar[2] = w;
    out[i] = r;
    rays[2 * i + 1].w = h.t;                 // ray->maxt = t
}

__global__ void k_tri_type(const int* __restrict__ attr, const Attr* __restrict__ attrs, const Material* __restrict__ mats,
                           size_t ntri, uint8_t* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntri) out[i] = (uint8_t)mats[attrs[attr[i]].material].type;
}

}  // namespace

cudaError_t make_tri_type(const int* tri_attr, const Attr* attrs, const Material* mats, size_t ntri, uint8_t** out,
                          cudaStream_t s) {
    const cudaError_t e = cudaMallocAsync((void**)out, ntri, s);
    if (e != cudaSuccess) { *out = nullptr; return e; }
    k_tri_type<<<(unsigned)((ntri + 255) / 256), 256, 0, s>>>(tri_attr, attrs, mats, ntri, *out);
    return cudaGetLastError();
}

cudaError_t pack_tri_shade(const float* corner_n, const float* corner_uv, const int* tri_attr, size_t ntri, TriShade** out,
                           cudaStream_t s) {
    cudaError_t e = cudaMallocAsync((void**)out, sizeof(TriShade) * ntri, s);
    if (e != cudaSuccess) { *out = nullptr; return e; }
    // records are read in 256-bit loads: the allocator's alignment, checked rather than assumed
    if ((uintptr_t)*out % sizeof(TriShade) != 0) return cudaErrorMisalignedAddress;
    k_pack_tri_shade<<<(unsigned)((ntri + 255) / 256), 256, 0, s>>>(corner_n, corner_uv, tri_attr, ntri, *out);
    return cudaGetLastError();
}
}  // namespace aur

using namespace aur;

extern "C" aur_status aur_bvh_set_shading(aur_bvh* b, const float* corner_normals, const float* corner_uvs) {
    if (!b || !corner_normals) return fail(AUR_ERR_INVALID_ARG, "aur_bvh_set_shading: NULL argument");
    if (b->owned_by_scene) return fail(AUR_ERR_INVALID_ARG, "aur_bvh_set_shading: the BVH belongs to a scene, "
                                                            "which provides its normals and uvs");
    DeviceGuard g(b->ctx->device);
    cudaStream_t s = b->ctx->stream;
    const size_t ntri = (size_t)b->bvh.num_tris;
    if (b->owns_shading && b->tri) cudaFreeAsync(b->tri, s);
    b->tri = nullptr;
    b->owns_shading = false;
    TriShade* tri = nullptr;
    DevIn cn, cu;
    cudaError_t e = cn.init(corner_normals, sizeof(float) * 9 * ntri, 4, s);
    if (e == cudaSuccess) e = cu.init(corner_uvs, sizeof(float) * 6 * ntri, 4, s);
    if (e == cudaSuccess) e = pack_tri_shade((const float*)cn.ptr, (const float*)cu.ptr, b->tri_attr, ntri, &tri, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        if (tri) cudaFreeAsync(tri, s);
        cudaStreamSynchronize(s);
        return cuda_fail(e, "aur_bvh_set_shading");
    }
    b->tri = tri;
    b->owns_shading = true;
    return AUR_OK;
}

extern "C" aur_status aur_bvh_intersect(aur_bvh* b, aur_ray* rays, aur_isect* isects, uint32_t n) {
    if (!b || (n && (!rays || !isects))) return fail(AUR_ERR_INVALID_ARG, "aur_bvh_intersect: NULL argument");
    if (!b->tri)
        return fail(AUR_ERR_INVALID_ARG, "aur_bvh_intersect: no per-corner normals (aur_bvh_set_shading)");
    if (n == 0) return AUR_OK;
    DeviceGuard g(b->ctx->device);
    cudaStream_t s = b->ctx->stream;
    DevOut dr, dh;   // rays are read and written (maxt), hits written
    CUDA_TRY(dr.init(rays, sizeof(aur_ray) * n, 16, s), "aur_bvh_intersect(rays)");
    if (dr.owned)
        CUDA_TRY(cudaMemcpyAsync(dr.ptr, rays, sizeof(aur_ray) * n, cudaMemcpyDefault, s), "aur_bvh_intersect(rays)");
    CUDA_TRY(dh.init(isects, sizeof(aur_isect) * n, 16, s), "aur_bvh_intersect(isects)");
    k_intersect<<<(n + kIsectBlock - 1) / kIsectBlock, kIsectBlock, 0, s>>>(
        b->bvh.nodes, b->bvh.nodes4, b->bvh.tris, b->tri, (float4*)dr.ptr,
        (aur_isect*)dh.ptr, n);
    CUDA_TRY(cudaGetLastError(), "aur_bvh_intersect");
    CUDA_TRY(dr.finish(), "aur_bvh_intersect(download)");
    CUDA_TRY(dh.finish(), "aur_bvh_intersect(download)");
    CUDA_TRY(cudaStreamSynchronize(s), "aur_bvh_intersect");
    return AUR_OK;
}
