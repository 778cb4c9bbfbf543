// aur_trace_split.h — which thread takes which ray of a batch, in the forms with a thread or a warp per ray.
// Plain C++, so that the arithmetic can be compiled and checked without a device.
#pragma once
#include <cstdint>
#ifdef __CUDACC__
#define AUR_SPLIT __host__ __device__ __forceinline__
#else
#define AUR_SPLIT inline
#endif

namespace aur {

constexpr int kTraceBlock = 128;

// Rays per warp of a small batch: the fewest (a power of two) that need at most kSpreadWarps warps per
// SM; 32 once the batch is large. n + r - 1 does not fit 32 bits for the largest batches.
constexpr int kSpreadWarps = 16;
AUR_SPLIT int rays_per_warp(uint32_t n, int sms) {
    int r = 1;
    while (r < 32 && ((uint64_t)n + r - 1) / r > (uint64_t)(kSpreadWarps * sms)) r *= 2;
    return r;
}

AUR_SPLIT uint32_t spread_grid(uint32_t n, int per_warp) {
    const uint64_t warps = ((uint64_t)n + per_warp - 1) / per_warp;
    return (uint32_t)((warps * 32 + kTraceBlock - 1) / kTraceBlock);
}

// The ray of a thread when every warp takes `per_warp` of them; n or more: none. By the warp's number:
// that of the thread passes 2^32 in batches of 2^32 - 96 rays and more.
AUR_SPLIT uint32_t spread_index(uint32_t block, uint32_t thread, int per_warp) {
    const uint32_t lane = thread & 31, warp = block * (kTraceBlock / 32) + (thread >> 5);
    if (lane >= (uint32_t)per_warp) return 0xffffffffu;
    const uint64_t i = (uint64_t)warp * per_warp + lane;
    return i < 0xffffffffu ? (uint32_t)i : 0xffffffffu;
}

}  // namespace aur
