// Every ray of a batch is one thread's, up to the largest batch that the interface takes (2^32 - 1 rays).
#include "aur_trace_split.h"
#include <cstdio>
#include <initializer_list>

using namespace aur;

int main() {
    int bad = 0;
    for (int sms : {1, 148}) {
        for (uint32_t n : {1u, 2u, 31u, 32u, 33u, 1000u, 14208u, 14209u, 75776u, 75777u, 1u << 20, 1u << 31, 0xffffff80u, 0xffffffa0u,
                           0xfffffff0u, 0xfffffff1u, 0xfffffff9u, 0xfffffffcu, 0xfffffffdu, 0xfffffffeu, 0xffffffffu}) {
            const int r = rays_per_warp(n, sms);
            const uint64_t warps = ((uint64_t)n + r - 1) / r;
            if (r < 32 && warps > (uint64_t)(kSpreadWarps * sms)) { std::printf("n %u: %d rays a warp\n", n, r); ++bad; }
            for (int per : {1, r, 32}) {
                const uint64_t threads = (uint64_t)spread_grid(n, per) * kTraceBlock;
                const uint64_t need = ((uint64_t)n + per - 1) / per;
                if (threads / 32 < need) { std::printf("n %u, %d a warp: %llu warps\n", n, per, (unsigned long long)(threads / 32)); ++bad; }
                if (per < 32 && n > (1u << 27)) continue;   // more warps than a launch of this form is used for
                // the first and last warps in full, and one in between: index = its place, or none
                for (uint64_t w : {(uint64_t)0, need / 2, need > 2 ? need - 2 : (uint64_t)0, need - 1, threads / 32 - 1})
                    for (uint32_t lane = 0; lane < 32; ++lane) {
                        const uint64_t t = w * 32 + lane, i = w * per + lane;
                        const uint32_t got = spread_index((uint32_t)(t / kTraceBlock), (uint32_t)(t % kTraceBlock), per);
                        const bool mine = lane < (uint32_t)per && i < n;
                        if (mine ? got != i : got < n) { std::printf("n %u, %d a warp, warp %llu lane %u: %u\n", n, per, (unsigned long long)w, lane, got); ++bad; }
                    }
            }
        }
    }
    return bad ? 1 : 0;
}
