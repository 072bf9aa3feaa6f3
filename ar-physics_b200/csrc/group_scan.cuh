// group_scan.cuh -- the neighbor search of a particle shared by LANES threads
// of a warp: search rows, quantised candidates, hit lists in shared memory.
#pragma once

#include "grid.cuh"

namespace arp {

// The rows of search cells around a particle, 2 cells each way along a halved
// axis and 1 along the others: row q (ascending z, then y) spans `width` cells
// from search_row(q) on.  Every particle within h lies in them (search cells are
// at least h/2 wide on halved axes and h wide on the others).  The rows are not
// clipped to the sphere: the lanes of a warp walk rows of equal length, which a
// clip would only make uneven without shortening the longest.
struct SearchRows {
    int y, z, x0, ry, nrows;
    uint32_t width;
};
template <int DIM>
__device__ __forceinline__ SearchRows search_rows(float4 x, bool scan, const SceneP& P) {
    constexpr int RZ = 1 + (int)(kSearchHalve >> 2 & 1u);
    const Grid& g = P.sgrid;
    const CellCoord c = scan ? cell_coord(x, g) : CellCoord{0, 0, 0};
    const int rx = 1 + (int)P.halved[0];
    SearchRows r;
    r.ry = 1 + (int)P.halved[1];
    r.y = c.y - r.ry;
    r.z = DIM == 3 ? c.z - RZ : c.z;
    r.x0 = max(c.x - rx, 0);
    r.width = (uint32_t)(min(c.x + rx, (int)g.sub[0] - 1) - r.x0) + 1u;
    r.nrows = scan ? (2 * r.ry + 1) * (DIM == 3 ? 2 * RZ + 1 : 1) : 0;
    return r;
}
// First cell of row q, or kInvalid outside the grid.
__device__ __forceinline__ uint32_t search_row(const SearchRows& r, int q, const SceneP& P) {
    const int qz = r.ry == 1 ? q / 3 : q / 5;
    const int y = r.y + q - qz * (2 * r.ry + 1), z = r.z + qz;
    const Grid& g = P.sgrid;
    if (y < 0 || y >= (int)g.sub[1] || z < 0 || z >= (int)g.sub[2]) return kInvalid;
    return P.cell_base + (uint32_t)r.x0 + (uint32_t)y * g.sub[0] + (uint32_t)z * g.sub[0] * g.sub[1];
}

constexpr int kGroupList = 96;  // list entries per particle in the forward kernel

// What a particle's scan reads: the joined arrays of n mobile and then the
// boundary particles (see FluidArgs).
struct ScanArrays {
    const uint32_t *code, *start, *bstart;
    uint32_t n;
};

// Lists the candidates of one particle per LANES threads that pass the
// quantised test, in candidate order (boundary, then mobile, row by row), and
// calls eval(count) on the whole warp whenever lists of it have to be taken:
// entries [0, count) of each particle's list, every entry once, a multiple of
// LANES except the last time.
//   * The bounds of all search rows are read at once, one row per lane, and
//     turned into a list of non-empty segments of consecutive candidates, so
//     the scan is one flat loop with U loads in flight per lane.
//   * Hits are compacted in candidate order by ballots.
// `list` [LIST] and `seg` [2 * MAXROWS] lie in shared memory.
template <int DIM, int LANES, int LIST = kGroupList>
struct GroupScan {
    static constexpr int U = LANES >= 16 ? 2 : 4;  // candidate loads in flight per lane
    static constexpr int RZ = 1 + (int)(kSearchHalve >> 2 & 1u);
    static constexpr int MAXROWS = 5 * (DIM == 3 ? 2 * RZ + 1 : 1);
    static_assert(LIST >= 2 * U * LANES, "the list holds what one scan iteration can add");

    template <class Eval>
    static __device__ __forceinline__ void run(float4 xi, bool scan, const SceneP& P, const ScanArrays& a,
                                               uint32_t* list, uint2* seg, Eval&& eval) {
        constexpr unsigned FULL = 0xFFFFFFFFu;
        constexpr unsigned GM = LANES == 32 ? FULL : (1u << (LANES & 31)) - 1u;
        const uint32_t lane = threadIdx.x % LANES;
        const uint32_t gshift = (threadIdx.x & 31u) & ~(uint32_t)(LANES - 1);
        const uint32_t own = own_code<DIM>(xi, P);
        // segments (end, first index - first number) of candidates, numbered 0 .. total over all rows
        uint32_t total = 0, nseg = 0;
        const SearchRows rows = search_rows<DIM>(xi, scan, P);
#pragma unroll
        for (int q0 = 0; q0 < MAXROWS; q0 += LANES) {
            const int q = q0 + (int)lane;
            const uint32_t c0 = q < rows.nrows ? search_row(rows, q, P) : kInvalid;
            uint32_t bb = 0, lb = 0, jb = 0, lm = 0;
            if (c0 != kInvalid) {
                const uint32_t c1 = c0 + rows.width;
                bb = a.bstart[c0];
                lb = a.bstart[c1] - bb;
                jb = a.start[c0];
                lm = a.start[c1] - jb;
            }
            uint32_t len = lb + lm, cnt = (lb ? 1u : 0u) + (lm ? 1u : 0u);
#pragma unroll
            for (int o = 1; o < LANES; o <<= 1) {
                const uint32_t l2 = __shfl_up_sync(FULL, len, o, LANES), c2 = __shfl_up_sync(FULL, cnt, o, LANES);
                if ((int)lane >= o) {
                    len += l2;
                    cnt += c2;
                }
            }
            const uint32_t first = total + len - lb - lm;
            uint32_t w = nseg + cnt - (lb ? 1u : 0u) - (lm ? 1u : 0u);
            if (lb) seg[w++] = make_uint2(first + lb, a.n + bb - first);
            if (lm) seg[w] = make_uint2(first + lb + lm, jb - first - lb);
            total += __shfl_sync(FULL, len, LANES - 1, LANES);
            nseg += __shfl_sync(FULL, cnt, LANES - 1, LANES);
        }
        __syncwarp();
        uint32_t t0 = 0, cnt = 0, si = 0;  // candidates tested, hits listed, the lane's current segment
        for (;;) {
            while (__any_sync(FULL, t0 < total)) {
                uint32_t jj[U], code[U];
                bool in[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t t = t0 + (uint32_t)(u * LANES) + lane;
                    in[u] = t < total;
                    jj[u] = code[u] = 0u;
                    if (in[u]) {
                        uint2 sg = seg[si];
                        while (t >= sg.x) sg = seg[++si];  // the last segment ends at total > t
                        jj[u] = sg.y + t;
                        code[u] = a.code[jj[u]];
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool h = in[u] && code_test(code[u], own) < 0;
                    const unsigned m = __ballot_sync(FULL, h) >> gshift & GM;
                    if (h) list[cnt + __popc(m & ((1u << lane) - 1u))] = jj[u];
                    cnt += __popc(m);
                }
                t0 += U * LANES;
                if (__any_sync(FULL, cnt > (uint32_t)(LIST - U * LANES))) break;
            }
            __syncwarp();
            const uint32_t ev = t0 < total ? cnt & ~(uint32_t)(LANES - 1) : cnt;
            eval(ev);
            if (!__any_sync(FULL, t0 < total)) break;
            __syncwarp();
            const uint32_t rest = cnt - ev;  // fewer than LANES
            const uint32_t keep = lane < rest ? list[ev + lane] : 0u;
            __syncwarp();
            if (lane < rest) list[lane] = keep;
            cnt = rest;
        }
    }
};

}  // namespace arp
