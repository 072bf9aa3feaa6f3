// grid.cuh -- cell hashing shared by the grid build and the force kernels.
#pragma once

#include "arp_internal.h"

namespace arp {

// Cell coordinate along one axis, as fill_buckets hashes it
// (neighbor_list.rs:95): floor(clamp((p - min) / dim, 0, 1) * sub).  An axis
// of zero extent maps to cell 0 (the shader divides 0/0 there) and a
// coordinate exactly on the upper face is clamped into the last cell.  Every
// operation is separately rounded so host and device agree bit for bit.
__host__ __device__ inline uint32_t axis_cell(float p, float mn, float d, uint32_t sub) {
    if (d == 0.0f) return 0u;
#ifdef __CUDA_ARCH__
    float t = __fdiv_rn(__fsub_rn(p, mn), d);
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    uint32_t c = (uint32_t)floorf(__fmul_rn(t, (float)sub));
#else
    volatile float diff = p - mn;
    volatile float t = diff / d;
    float tc = t < 0.0f ? 0.0f : (t > 1.0f ? 1.0f : t);
    volatile float sc = tc * (float)sub;
    uint32_t c = (uint32_t)__builtin_floorf(sc);
#endif
    return c >= sub ? sub - 1u : c;
}

__host__ __device__ inline bool finite3(float4 p) {
#ifdef __CUDA_ARCH__
    return isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
#else
    return __builtin_isfinite(p.x) && __builtin_isfinite(p.y) && __builtin_isfinite(p.z);
#endif
}

struct CellCoord {
    int x, y, z;
};

__host__ __device__ inline CellCoord cell_coord(float4 p, const Grid& g) {
    CellCoord c;
    c.x = (int)axis_cell(p.x, g.min[0], g.dim[0], g.sub[0]);
    c.y = (int)axis_cell(p.y, g.min[1], g.dim[1], g.sub[1]);
    c.z = (int)axis_cell(p.z, g.min[2], g.dim[2], g.sub[2]);
    return c;
}

__host__ __device__ inline uint32_t cell_id(const CellCoord& c, const Grid& g) {
    return (uint32_t)c.x + (uint32_t)c.y * g.sub[0] + (uint32_t)c.z * g.sub[0] * g.sub[1];
}

// Counts slot i, at position p of scene P, into its search cell (the
// non-finite bucket `ncells` for a non-finite position).
__device__ __forceinline__ void bin_particle(float4 p, const SceneP& P, uint32_t ncells, uint32_t i,
                                             const CellBins& b) {
    uint32_t k = ncells;
    uint2 coord = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
    if (finite3(p)) {
        const CellCoord fc = cell_coord(p, P.sgrid);
        k = P.cell_base + cell_id(fc, P.sgrid);
        // reference cell = search cell >> 1 on halved axes (exact, see SceneP)
        coord = make_uint2((uint32_t)fc.x >> P.halved[0] | ((uint32_t)fc.y >> P.halved[1]) << 16,
                           (uint32_t)fc.z >> P.halved[2]);
    }
    b.coord[i] = coord;
    b.key[i] = k;
    b.rank[i] = atomicAdd(&b.count[k], 1u);
}

// ---- quantised positions -------------------------------------------------------
// The fluid kernel tests candidates on positions quantised to h / kCodeUnits,
// one byte per axis modulo 256 (x lowest, the top byte 0): a candidate is 4
// bytes instead of 16, and its test one subtraction, one four-way byte product
// and one compare on integers.
//
// No pair within h may fail the test.  With X = (x - min) 63 / h per axis, a
// candidate's code is rint(X_j); the particle's own code is rint(X_i) in x and
// rint(X_i - 1/2) in y and z.  The codes are subtracted as 32-bit words, so a
// negative lower byte borrows 1 from the next.  The difference then is
// X_j - X_i plus an error of at most 1 in x and 1.5 in y and z (both roundings,
// the half, the borrow), 2.345 in norm; the top byte is 0 or -1.  A pair within
// h therefore has a sum of squares of at most (63 + 2.345)^2 + 1 = 4271.0; the
// bound below leaves 2 for the roundings of X in double precision.  Differences past 127
// wrap, which can only let far candidates through, and the evaluation of a
// pair tests r < h again.  A flat handle (Tables::flat) measures distances in the
// plane whatever z a state set later holds, so its codes leave z out.
constexpr double kCodeUnits = 63.0;
constexpr int kCodeBound = 4273;

__device__ __forceinline__ uint32_t code_axis(float p, float mn, double inv, double shift) {
    return (uint32_t)__double2ll_rn(((double)p - (double)mn) * inv - shift) & 255u;
}
__device__ __forceinline__ uint32_t scan_code(float4 p, const SceneP& P, uint32_t flat) {
    const uint32_t z = flat ? 0u : code_axis(p.z, P.grid.min[2], P.code_inv, 0.0);
    return code_axis(p.x, P.grid.min[0], P.code_inv, 0.0) | code_axis(p.y, P.grid.min[1], P.code_inv, 0.0) << 8 |
           z << 16;
}
template <int DIM>  // 2 for a flat handle
__device__ __forceinline__ uint32_t own_code(float4 p, const SceneP& P) {
    const uint32_t z = DIM == 2 ? 0u : code_axis(p.z, P.grid.min[2], P.code_inv, 0.5);
    return code_axis(p.x, P.grid.min[0], P.code_inv, 0.0) | code_axis(p.y, P.grid.min[1], P.code_inv, 0.5) << 8 |
           z << 16;
}
// Negative when the candidate may lie within h.
__device__ __forceinline__ int code_test(uint32_t candidate, uint32_t own) {
    const int d = (int)(candidate - own);
    return __dp4a(d, d, -kCodeBound - 1);
}

// ---- reference cells ----------------------------------------------------------

// Calls f(c0, c1) for the global search-cell x-rows covering the 3x3(x3)
// reference cells around the reference cell of x (the shaders' neighbor
// stencil, neighbor_list.rs:121-143), ascending.
template <class F>
__device__ __forceinline__ void for_reference_block_rows(float4 x, const SceneP& P, F&& f) {
    const CellCoord c = cell_coord(x, P.grid);
    const int cc[3] = {c.x, c.y, c.z};
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = max(cc[a] - 1, 0) << P.halved[a];
        hi[a] = ((min(cc[a] + 1, (int)P.grid.sub[a] - 1) + 1) << P.halved[a]) - 1;
    }
    const Grid& g = P.sgrid;
    for (int z = lo[2]; z <= hi[2]; ++z)
        for (int y = lo[1]; y <= hi[1]; ++y) {
            const uint32_t row = P.cell_base + (uint32_t)y * g.sub[0] + (uint32_t)z * g.sub[0] * g.sub[1];
            f(row + (uint32_t)lo[0], row + (uint32_t)hi[0] + 1u);
        }
}

}  // namespace arp
