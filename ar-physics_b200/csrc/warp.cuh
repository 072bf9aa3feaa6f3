// warp.cuh -- sums over the lanes of a thread group inside a warp, 32-byte loads.
#pragma once

#include <cstdint>

namespace arp {

// One 32-byte sector in one load (p 32-byte aligned).  load8 is volatile and so
// stays behind the wait of step_begin(); load8_at may be moved and is for
// addresses that depend on memory read after that wait.
__device__ __forceinline__ void load8(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}
__device__ __forceinline__ void load8_at(const float4* p, float4& a, float4& b) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// Sum of v over the LANES consecutive lanes (LANES a power of two, at most
// 32) that share one item: a butterfly of shuffles, the same order on every
// lane, so the result is deterministic and identical on all of them.
template <int LANES>
__device__ __forceinline__ float group_sum(float v) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t mask = (LANES == 32 ? 0xFFFFFFFFu : ((1u << LANES) - 1u)) << (lane & ~(uint32_t)(LANES - 1));
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, LANES);
    return v;
}

}  // namespace arp
