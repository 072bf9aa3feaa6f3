// solid_rec.cuh -- the records the solid kernels keep per solid, in solid-id
// order: what a neighbor needs is read with as few, as wide loads as its size
// allows.
#pragma once

#include "arp_internal.h"
#include "warp.cuh"

namespace arp {

// Position record, 2 float4 (SolidArgs::sx): stage position and density, then
// reference position and rest volume m / rho0 (constant).
struct SolidPos {
    float4 x, X;
};
__device__ __forceinline__ SolidPos load_pos(const float4* sx, uint32_t i) {
    SolidPos r;
    load8(sx + 2 * (size_t)i, r.x, r.X);
    return r;
}
__device__ __forceinline__ SolidPos load_pos_at(const float4* sx, uint32_t j) {  // j read from a reference list
    SolidPos r;
    load8_at(sx + 2 * (size_t)j, r.x, r.X);
    return r;
}

// Stress record, 6 float4 (SolidArgs::AF): the 3 x 3 matrices A = sigma L and F
// by columns, then the packed cell coordinates (18 floats + 2 words, 96 bytes).
constexpr int kStressRec = 6;
struct StressRec {
    float A[3][3], F[3][3];  // [column][row]
    uint2 cell;
};
template <bool AT = false>  // AT: i was read from a reference list
__device__ __forceinline__ StressRec load_stress(const float4* AF, uint32_t i) {
    const float4* const p = AF + kStressRec * (size_t)i;
    float4 a, b, c, d;
    if (AT) {
        load8_at(p, a, b);
        load8_at(p + 2, c, d);
    } else {
        load8(p, a, b);
        load8(p + 2, c, d);
    }
    const float4 e = p[4];
    StressRec r;
    r.A[0][0] = a.x; r.A[0][1] = a.y; r.A[0][2] = a.z;
    r.A[1][0] = a.w; r.A[1][1] = b.x; r.A[1][2] = b.y;
    r.A[2][0] = b.z; r.A[2][1] = b.w; r.A[2][2] = c.x;
    r.F[0][0] = c.y; r.F[0][1] = c.z; r.F[0][2] = c.w;
    r.F[1][0] = d.x; r.F[1][1] = d.y; r.F[1][2] = d.z;
    r.F[2][0] = d.w; r.F[2][1] = e.x; r.F[2][2] = e.y;
    r.cell = make_uint2(__float_as_uint(e.z), __float_as_uint(e.w));
    return r;
}
__device__ __forceinline__ void store_stress(float4* AF, uint32_t i, const StressRec& r) {
    float4* const p = AF + kStressRec * (size_t)i;
    p[0] = make_float4(r.A[0][0], r.A[0][1], r.A[0][2], r.A[1][0]);
    p[1] = make_float4(r.A[1][1], r.A[1][2], r.A[2][0], r.A[2][1]);
    p[2] = make_float4(r.A[2][2], r.F[0][0], r.F[0][1], r.F[0][2]);
    p[3] = make_float4(r.F[1][0], r.F[1][1], r.F[1][2], r.F[2][0]);
    p[4] = make_float4(r.F[2][1], r.F[2][2], __uint_as_float(r.cell.x), __uint_as_float(r.cell.y));
}

// Whether two packed cell coordinates lie in the same 3 x 3 x 3 stencil.
__device__ __forceinline__ bool in_stencil(uint2 a, uint2 b) {
    const int dx = (int)(a.x & 0xFFFFu) - (int)(b.x & 0xFFFFu);
    const int dy = (int)(a.x >> 16) - (int)(b.x >> 16);
    const int dz = (int)a.y - (int)b.y;
    return a.y != 0xFFFFFFFFu && b.y != 0xFFFFFFFFu && dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && dz >= -1 &&
           dz <= 1;
}

}  // namespace arp
