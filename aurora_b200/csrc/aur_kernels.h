// aur_kernels.h — host-side launch wrappers of the sm_100a kernels (internal).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "aur_bvh.cuh"
#include "aur_integrator.cuh"

namespace aur {

// trace.cu — batched ray queries (aur_ray / aur_hit layouts of aurora_b200.h). cursor: kCursorWords words of device memory that
// are zero, that the call has to itself until its work is done, and that are zero again then (TraceSlot); without
// them the forms that need none are used.
constexpr int kCursorWords = 2;
cudaError_t launch_trace_closest(const DeviceBvh& bvh, const int* tri_attr, const void* rays, void* hits, uint32_t n,
                                 uint32_t* cursor, cudaStream_t s);
// the whole record of EmbreeAccelerator::intersect (aur_isect); shrinks rays[i].maxt on a hit
cudaError_t launch_intersect(const DeviceBvh& bvh, const TriShade* tri, void* rays, void* isects, uint32_t n, uint32_t* cursor,
                             cudaStream_t s);
cudaError_t launch_trace_occluded(const DeviceBvh& bvh, const void* rays, uint8_t* occ, uint32_t n, uint32_t* cursor, cudaStream_t s);

// kelemen.cu — directional-albedo table for reflectance index 0..20 into out[2048]
cudaError_t launch_kelemen_table(int refl_index, float* out, cudaStream_t s);

// render_plain.cu — one thread per pixel, spp paths per thread: the counting pass, callers without
// scratch memory, scenes without 4-wide trees.
// counters[0..3] = camera rays, closest rays, shadow rays, paths; with count_width (the width of the
// tree walked while counting: 2 binary, 4 four-wide, 8 quantised four-wide; 0 not counting)
// also [4..5] interior-node visits / triangle tests of closest-hit rays and
// [6..7] those of shadow rays (accumulated).
cudaError_t launch_render_plain(const DevScene& sc, const PathParams& p, float4* film, double* film64,
                                unsigned long long* counters, int count_width, cudaStream_t s);

// render_paths.cu — the plain renderer with one lane per path (needs the 4-wide trees): `chunk` samples of every pixel
// at a time through `scratch` (paths_scratch_bytes). counters: [1] closest rays, [2] shadow rays
// (accumulated), [kPathCursor] cleared by the caller. film and film64 may be null (FP64 only).
constexpr int kPathCursor = 7;
size_t paths_scratch_bytes(const DevScene& sc, const PathParams& p, size_t budget, int* chunk);
cudaError_t launch_render_paths(const DevScene& sc, const PathParams& p, bool quantised, bool fp64, int chunk, void* scratch,
                                float4* film, double* film64, unsigned long long* counters, uint64_t* launches, cudaStream_t s);

}  // namespace aur
