// accel.cu — the full contract of EmbreeAccelerator::intersect for arrays of rays
// (Aurora/src/geometry/embreeAccelerator.cpp:41-91): the shading records its post-process reads
// and the entry points; the queries and the post-process are in trace.cu (IsectOut).
#include "aur_capi_internal.h"

namespace aur {
namespace {

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

// A material index out of range can come from a device-resident attribute table, which is not checked; it
// matters only if such a triangle is shaded, so no material is read for it here.
__global__ void k_tri_type(const int* __restrict__ attr, const Attr* __restrict__ attrs, const Material* __restrict__ mats,
                           uint32_t nmat, size_t ntri, uint8_t* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntri) return;
    const uint32_t m = (uint32_t)attrs[attr[i]].material;
    out[i] = (uint8_t)(m < nmat ? mats[m].type : MAT_CONSTANT);
}

}  // namespace

cudaError_t make_tri_type(const int* tri_attr, const Attr* attrs, const Material* mats, uint32_t nmat, size_t ntri,
                          uint8_t** out, cudaStream_t s) {
    const cudaError_t e = cudaMallocAsync((void**)out, ntri, s);
    if (e != cudaSuccess) { *out = nullptr; return e; }
    k_tri_type<<<(unsigned)((ntri + 255) / 256), 256, 0, s>>>(tri_attr, attrs, mats, nmat, ntri, *out);
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
    TraceSlot slot(b->ctx);
    CUDA_TRY(launch_intersect(b->bvh, b->tri, dr.ptr, dh.ptr, n, slot.ptr, s), "aur_bvh_intersect");
    CUDA_TRY(dr.finish(), "aur_bvh_intersect(download)");
    CUDA_TRY(dh.finish(), "aur_bvh_intersect(download)");
    CUDA_TRY(cudaStreamSynchronize(s), "aur_bvh_intersect");
    slot.done();
    return AUR_OK;
}
