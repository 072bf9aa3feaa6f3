// neighbor.cu -- uniform-grid neighbor build (replaces reset_buckets +
// fill_buckets, src/soft_body/neighbor_list.rs:37-143 and update_contents
// :224-294).
//
// The reference appends each particle into a fixed 128-slot bucket with
// atomics, so slot order is nondeterministic on a GPU and particles past 128
// are dropped.  Here the grid is a counting sort with no capacity limit:
//   1. cell key + histogram (one atomic per particle; the returned value is
//      the particle's arrival rank inside its cell), by the kernel that writes
//      the state where there is one (CellBins), else by k_cell_keys;
//   2. k_scan_tiles: exclusive prefix of the histogram inside tiles of 4096
//      cells, in place, and the tile totals;
//   3. k_scatter: every block turns the tile totals into tile bases itself,
//      writes its share of the cell starts (prefix + base) and scatters its
//      particles to perm[start[key] + rank];
//   4. k_order_gather: per block of cells, the slots of each cell ascending (so
//      the order is deterministic for every run length) and the state gathered
//      into that order; it also clears the histogram and records the largest
//      occupancy and cells over the reference's 128.
// Memory traffic per particle: 16 B position, 4+4 B key/rank, 4+4 B perm, and
// the state read and written once.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>

#include "grid.cuh"
#include "launch.cuh"

namespace arp {

namespace {

constexpr int kThreads = 256;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // per thread
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t scene_of(const float4* vm, const uint32_t* mat_u32, uint32_t i, const Tables& T) {
    const uint32_t m = vm ? __float_as_uint(vm[i].w) : (mat_u32 ? mat_u32[i] : 0u);
    return T.mats[m].scene;
}

__global__ void k_cell_keys(const float4* pos, const float4* vm,
                            const uint32_t* mat_u32, uint32_t n, Tables T, CellBins bin) {
    step_begin();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bin_particle(pos[i], T.scenes[scene_of(vm, mat_u32, i, T)], T.ncells, i, bin);
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x a multiple
// of 32, at most 1024).  The block total is excl + v of the last thread.
__device__ __forceinline__ void block_excl_scan(uint32_t v, uint32_t& excl) {
    __shared__ uint32_t warp_tot[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (int)(blockDim.x >> 5);
    uint32_t inc = warp_incl_scan(v);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nwarps ? warp_tot[lane] : 0u;
        uint32_t wi = warp_incl_scan(w);
        if (lane < nwarps) warp_tot[lane] = wi - w;
    }
    __syncthreads();
    excl = warp_tot[warp] + inc - v;
}

// Exclusive prefix inside each tile of kScanTile counts and the tile totals.
// `count` and `out` may be the same array, so they are not declared
// __restrict__; with CLEAR (different arrays) the counts are left at zero for
// the next histogram.  `wide`: both arrays are 16-byte aligned (the
// allocation-free build scans a caller's array, which need not be).
template <bool CLEAR>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(uint32_t* count, uint32_t len, uint32_t* out,
                                                             uint32_t* block_sums, bool wide) {
    __shared__ uint32_t last_total;
    step_begin();
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems] = {0u, 0u, 0u, 0u};
    static_assert(kScanItems == 4, "one 16-byte load per thread");
    const bool whole = wide && base + kScanItems <= len;
    if (whole) {
        const uint4 q = *reinterpret_cast<const uint4*>(count + base);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        if (CLEAR) *reinterpret_cast<uint4*>(count + base) = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
        for (int j = 0; j < kScanItems; ++j)
            if (base + j < len) {
                v[j] = count[base + j];
                if (CLEAR) count[base + j] = 0u;
            }
    }
    uint32_t excl;
    const uint32_t s = v[0] + v[1] + v[2] + v[3];
    block_excl_scan(s, excl);
    if (threadIdx.x == blockDim.x - 1) last_total = excl + s;
    const uint4 o = make_uint4(excl, excl + v[0], excl + v[0] + v[1], excl + v[0] + v[1] + v[2]);
    if (whole) {
        *reinterpret_cast<uint4*>(out + base) = o;
    } else {
        const uint32_t w[kScanItems] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int j = 0; j < kScanItems; ++j)
            if (base + j < len) out[base + j] = w[j];
    }
    __syncthreads();
    if (threadIdx.x == 0) block_sums[blockIdx.x] = last_total;
}

// Adds to each tile of the scan the sum of the totals of the tiles before it;
// each block (one tile of kScanTile items) sums those totals itself, a block
// reduction over at most a few hundred values, so no separate pass scans them.
__global__ void k_scan_add(uint32_t* out, uint32_t len, const uint32_t* sums) {
    __shared__ uint32_t warp_part[kScanThreads / 32];
    __shared__ uint32_t prefix;
    step_begin();
    uint32_t part = 0;
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += blockDim.x) part += sums[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t p = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) p += warp_part[w];
        prefix = p;
    }
    __syncthreads();
    const uint32_t add = prefix;
    if (add == 0u) return;
    const uint32_t base = blockIdx.x * kScanTile;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        const uint32_t idx = base + (uint32_t)j * blockDim.x + threadIdx.x;
        if (idx < len) out[idx] += add;
    }
}

// Cell starts and scatter from the tile-local prefix `local` (k_scan_tiles in
// place) and the tile totals, which every block sums up itself: at most
// kBaseTiles of them (4 M cells), so no pass of its own finishes the scan.
constexpr uint32_t kBaseTiles = 1024;
__global__ void __launch_bounds__(kThreads) k_scatter(const uint32_t* key,
                                                      const uint32_t* rank, uint32_t n,
                                                      const uint32_t* local,
                                                      const uint32_t* sums, uint32_t len,
                                                      uint32_t* start, uint32_t* perm,
                                                      uint32_t* zero) {
    __shared__ uint32_t tile_base[kBaseTiles];
    step_begin();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (zero && i < kStageWords) zero[i] = 0u;
    // loads that do not need the bases first
    const bool mine = i < n;
    const uint32_t c = mine ? key[i] : 0u;
    const uint32_t at = mine ? local[c] + rank[i] : 0u;
    const uint32_t q = 4u * i;
    uint4 st = make_uint4(0u, 0u, 0u, 0u);
    if (q + 4u <= len) st = *reinterpret_cast<const uint4*>(local + q);
    const uint32_t tiles = (len + kScanTile - 1) / kScanTile;
    static_assert(kBaseTiles == 4 * kThreads, "four totals per thread");
    {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = 4u * threadIdx.x + j < tiles ? sums[4u * threadIdx.x + j] : 0u;
        uint32_t excl;
        block_excl_scan(v[0] + v[1] + v[2] + v[3], excl);
        tile_base[4u * threadIdx.x] = excl;
        tile_base[4u * threadIdx.x + 1] = excl + v[0];
        tile_base[4u * threadIdx.x + 2] = excl + v[0] + v[1];
        tile_base[4u * threadIdx.x + 3] = excl + v[0] + v[1] + v[2];
    }
    __syncthreads();
    if (mine) perm[at + tile_base[c / kScanTile]] = i;
    if (q < len) {
        const uint32_t b = tile_base[q / kScanTile];  // four entries of one tile
        if (q + 4u <= len) {
            *reinterpret_cast<uint4*>(start + q) = make_uint4(st.x + b, st.y + b, st.z + b, st.w + b);
        } else {
            for (uint32_t j = q; j < len; ++j) start[j] = local[j] + b;
        }
    }
}
// The same scatter from finished cell starts (grids of more tiles).
__global__ void k_scatter_plain(const uint32_t* key, const uint32_t* rank, uint32_t n,
                                const uint32_t* start, uint32_t* perm,
                                uint32_t* zero) {
    step_begin();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (zero && i < kStageWords) zero[i] = 0u;
    if (i < n) perm[start[key[i]] + rank[i]] = i;
}

// Occupancy (mobile + boundary) of the reference cell whose first search
// cell is global cell c, or 0 when c is not the first search cell of its
// reference cell.
__device__ __forceinline__ uint32_t reference_cell_occupancy(uint32_t c, const uint32_t* start, const uint32_t* bstart,
                                                             const Tables& T) {
    uint32_t lo = 0, hi = T.nscenes;  // scene with the largest cell_base <= c
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (T.scenes[mid].cell_base <= c) lo = mid;
        else hi = mid;
    }
    const SceneP& P = T.scenes[lo];
    const Grid& g = P.sgrid;
    const uint32_t l = c - P.cell_base;
    if ((P.halved[1] | P.halved[2]) == 0u) {
        // only x halved: sub[0] is even, so x and l have the same parity
        if (l & P.halved[0]) return 0u;
    } else {
        const uint32_t x = l % g.sub[0], y = (l / g.sub[0]) % g.sub[1], z = l / (g.sub[0] * g.sub[1]);
        if (((x & P.halved[0]) | (y & P.halved[1]) | (z & P.halved[2])) != 0u) return 0u;
    }
    uint32_t occ = 0;
    for (uint32_t dz = 0; dz <= P.halved[2]; ++dz)
        for (uint32_t dy = 0; dy <= P.halved[1]; ++dy) {
            const uint32_t r0 = c + dy * g.sub[0] + dz * g.sub[0] * g.sub[1], r1 = r0 + 1u + P.halved[0];
            occ += start[r1] - start[r0];
            if (bstart) occ += bstart[r1] - bstart[r0];
        }
    return occ;
}

constexpr uint32_t kShortRun = 32;    // runs up to this length: insertion sort by their own thread
constexpr uint32_t kWarpRun = 256;    // up to this length: bitonic sort in shared memory by one warp
constexpr uint32_t kBlockRun = 4096;  // up to this length: bitonic sort in shared memory by the block

// Block-wide reductions (blockDim.x == kThreads); every thread gets the result.
template <class Op>
__device__ __forceinline__ uint32_t block_reduce(uint32_t v, Op op) {
    __shared__ uint32_t part[kThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t r = part[0];
    for (int w = 1; w < kThreads / 32; ++w) r = op(r, part[w]);
    __syncthreads();  // part[] is reused by the next call
    return r;
}

// Sorts one long run perm[b, e) ascending with the whole block: stable
// one-bit LSD radix passes over (v - min), ping-ponging through tmp[b, e).
// The run's values are distinct slots, and a run of a cell-ordered state
// spans few slots, so log2(max - min + 1) passes suffice.
__device__ void block_sort_run(uint32_t* perm, uint32_t* tmp, uint32_t b, uint32_t e) {
    __shared__ uint32_t chunk_zeros;
    const uint32_t L = e - b;
    uint32_t lo = 0xFFFFFFFFu, hi = 0u;
    for (uint32_t i = threadIdx.x; i < L; i += kThreads) {
        const uint32_t v = perm[b + i];
        lo = min(lo, v);
        hi = max(hi, v);
    }
    lo = block_reduce(lo, [](uint32_t x, uint32_t y) { return min(x, y); });
    hi = block_reduce(hi, [](uint32_t x, uint32_t y) { return max(x, y); });
    const uint32_t span = hi - lo;
    const int bits = span ? 32 - __clz(span) : 0;
    uint32_t* src = perm + b;
    uint32_t* dst = tmp + b;
    for (int bit = 0; bit < bits; ++bit) {
        uint32_t z = 0;
        for (uint32_t i = threadIdx.x; i < L; i += kThreads) z += (((src[i] - lo) >> bit) & 1u) ^ 1u;
        z = block_reduce(z, [](uint32_t x, uint32_t y) { return x + y; });
        uint32_t zbase = 0, obase = z;
        for (uint32_t c0 = 0; c0 < L; c0 += kThreads) {
            const uint32_t i = c0 + threadIdx.x;
            const uint32_t v = i < L ? src[i] : 0u;
            const uint32_t f = i < L ? ((((v - lo) >> bit) & 1u) ^ 1u) : 0u;
            uint32_t excl;
            block_excl_scan(f, excl);
            if (threadIdx.x == kThreads - 1) chunk_zeros = excl + f;
            __syncthreads();
            const uint32_t cz = chunk_zeros;
            if (i < L) dst[f ? zbase + excl : obase + (threadIdx.x - excl)] = v;
            zbase += cz;
            obase += min((uint32_t)kThreads, L - c0) - cz;
            __syncthreads();  // chunk_zeros and the scan's shared totals are reused
        }
        __syncthreads();  // dst complete before the next pass reads it
        uint32_t* t = src;
        src = dst;
        dst = t;
    }
    if (src != perm + b)
        for (uint32_t i = threadIdx.x; i < L; i += kThreads) perm[b + i] = src[i];
    __syncthreads();
}

// Sorts one run perm[b, b + L) (L <= kWarpRun) ascending with one warp: a
// bitonic network over the run padded to a power of two in `buf` (shared
// memory, kWarpRun entries of this warp).  The values are distinct slots.
__device__ void warp_sort_run(uint32_t* perm, uint32_t b, uint32_t L, uint32_t* buf) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t P = 32u;
    while (P < L) P <<= 1;
    for (uint32_t i = lane; i < P; i += 32u) buf[i] = i < L ? perm[b + i] : 0xFFFFFFFFu;
    __syncwarp();
    for (uint32_t k = 2u; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j > 0u; j >>= 1) {
            for (uint32_t i = lane; i < P; i += 32u) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const uint32_t x = buf[i], y = buf[ixj];
                    if ((x > y) == ((i & k) == 0u)) {
                        buf[i] = y;
                        buf[ixj] = x;
                    }
                }
            }
            __syncwarp();
        }
    for (uint32_t i = lane; i < L; i += 32u) perm[b + i] = buf[i];
    __syncwarp();
}

// Sorts one run perm[b, b + L) (kWarpRun < L <= kBlockRun) ascending with the
// whole block: a bitonic network in shared memory (`buf`, kBlockRun entries).
__device__ void block_bitonic_run(uint32_t* perm, uint32_t b, uint32_t L, uint32_t* buf) {
    uint32_t P = 2u * kWarpRun;
    while (P < L) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += kThreads) buf[i] = i < L ? perm[b + i] : 0xFFFFFFFFu;
    __syncthreads();
    for (uint32_t k = 2u; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j > 0u; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += kThreads) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const uint32_t x = buf[i], y = buf[ixj];
                    if ((x > y) == ((i & k) == 0u)) {
                        buf[i] = y;
                        buf[ixj] = x;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < L; i += kThreads) perm[b + i] = buf[i];
    __syncthreads();
}

// Sorts the runs of the block's kThreads cells (cells past ncells are the
// non-finite bucket, then nothing) ascending in global memory, so the order
// inside a cell never depends on the arrival order of the histogram's atomics:
// runs of at most kShortRun by an insertion sort on their own thread, runs of
// at most kWarpRun by one warp each (warp_sort_run; the block's warps share its
// runs), runs of at most kBlockRun by the whole block in shared memory
// (block_bitonic_run), and longer ones (cells that gather particles outside the
// box, which are clamped into the edge cells) by the whole block through the
// scratch `tmp`, free once the scatter has run (block_sort_run).
__device__ void sort_block_runs(const uint32_t* start, uint32_t ncells, uint32_t* perm, uint32_t* tmp,
                                uint32_t* wbuf /* [kBlockRun] shared */) {
    __shared__ uint32_t long_cells[kThreads], mid_cells[kThreads];
    __shared__ uint32_t nlong, nmid;
    if (threadIdx.x == 0) nlong = nmid = 0;
    __syncthreads();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= ncells) {  // includes the non-finite bucket at index ncells
        const uint32_t b = start[c], e = start[c + 1];
        const uint32_t len = e - b;
        if (len > kWarpRun) {
            long_cells[atomicAdd(&nlong, 1u)] = c;
        } else if (len > kShortRun) {
            mid_cells[atomicAdd(&nmid, 1u)] = c;
        } else if (len >= 2) {
            for (uint32_t i = b + 1; i < e; ++i) {
                uint32_t v = perm[i];
                uint32_t j = i;
                while (j > b && perm[j - 1] > v) {
                    perm[j] = perm[j - 1];
                    --j;
                }
                perm[j] = v;
            }
        }
    }
    __syncthreads();
    const uint32_t nm = nmid, warp = threadIdx.x >> 5;
    for (uint32_t q = warp; q < nm; q += kThreads / 32) {
        const uint32_t mc = mid_cells[q];
        warp_sort_run(perm, start[mc], start[mc + 1] - start[mc], wbuf + warp * kWarpRun);
    }
    __syncthreads();  // the warps' buffers are the block buffer below
    const uint32_t cnt = nlong;
    for (uint32_t q = 0; q < cnt; ++q) {
        const uint32_t lc = long_cells[q];
        const uint32_t L = start[lc + 1] - start[lc];
        if (L <= kBlockRun) block_bitonic_run(perm, start[lc], L, wbuf);
        else block_sort_run(perm, tmp, start[lc], start[lc + 1]);
    }
    __syncthreads();
}

// The runs of a block's cells ordered without moving data twice: when they
// hold at most kStage slots and none is longer than kWarpRun, the slots are
// staged in shared memory and every thread ranks its slot among its cell's by
// counting the smaller ones (a handful of shared-memory reads for the few
// particles of a search cell); store(position, slot, load(slot)) is called for
// each.  A slot's cell is `key[slot]` or, with key null, marked by the cell's own
// thread at its positions (the allocation-free build, which keeps no keys, read
// the position again: 12.4 us for 1 M particles, 9.6 marked; with the gather the
// marks' shared memory costs 3 us a stage at 1 M, and the key is there).  A
// thread's first slot is loaded before the block's barrier, so those reads
// overlap the wait and the ranking.  Other blocks are sorted in global memory
// first.  Insertion sorts in global memory, one thread per cell, took 14 us per
// stage of the 1 M-particle scene.
constexpr uint32_t kStage = kBlockRun;
template <bool KEYS, class Load, class Store>
__device__ __forceinline__ void order_block(const uint32_t* start, uint32_t ncells, uint32_t* perm, uint32_t* tmp,
                                            const uint32_t* key, Load&& load, Store&& store) {
    __shared__ uint32_t buf[kStage];
    __shared__ uint32_t cstart[kThreads + 1];
    __shared__ uint8_t cell[KEYS ? 4 : kStage];  // of the block's kThreads
    static_assert(kThreads <= 256, "cells in 8 bits");
    const uint32_t c0 = blockIdx.x * kThreads;
    const uint32_t c = c0 + threadIdx.x;
    // cells 0 .. ncells (the last is the non-finite bucket), start has ncells + 2 entries
    const uint32_t s0 = start[min(c, ncells + 1u)], s1 = start[min(c + 1u, ncells + 1u)];
    cstart[threadIdx.x] = s0;
    if (threadIdx.x == kThreads - 1) cstart[kThreads] = s1;
    const int lengthy = __syncthreads_or(s1 - s0 > kWarpRun);
    const uint32_t p0 = cstart[0], m = cstart[kThreads] - p0;
    if (m == 0u) return;
    if (!lengthy && m <= kStage) {
        const uint32_t t0 = threadIdx.x;
        uint32_t q0 = 0;
        decltype(load(0u)) r0{};
        if (t0 < m) {
            const uint32_t v = perm[p0 + t0];
            buf[t0] = v;
            if (KEYS) q0 = key[v];
            r0 = load(v);
        }
        for (uint32_t t = t0 + kThreads; t < m; t += kThreads) buf[t] = perm[p0 + t];
        if (!KEYS)
            for (uint32_t p = s0; p < s1; ++p) cell[p - p0] = (uint8_t)threadIdx.x;
        __syncthreads();
        for (uint32_t t = t0; t < m; t += kThreads) {
            const uint32_t v = buf[t];
            if (t != t0) {
                if (KEYS) q0 = key[v];
                r0 = load(v);
            }
            const uint32_t q = KEYS ? q0 - c0 : cell[t];
            const uint32_t b = cstart[q] - p0, e = cstart[q + 1] - p0;
            uint32_t at = b;
            for (uint32_t j = b; j < e; ++j) at += buf[j] < v ? 1u : 0u;
            store(p0 + at, v, r0);
        }
        return;
    }
    sort_block_runs(start, ncells, perm, tmp, buf);
    for (uint32_t t = threadIdx.x; t < m; t += kThreads) {
        const uint32_t v = perm[p0 + t];
        store(p0 + t, v, load(v));
    }
}

struct Nothing {};

__global__ void __launch_bounds__(kThreads) k_order(const uint32_t* start, uint32_t ncells, uint32_t* perm,
                                                    uint32_t* tmp,
                                                    uint32_t* count) {
    step_begin();
    const uint32_t c = blockIdx.x * kThreads + threadIdx.x;
    if (count && c < ncells + 2u) count[c] = 0u;  // ready for the next histogram
    order_block<false>(start, ncells, perm, tmp, nullptr, [](uint32_t) { return Nothing{}; },
                [&](uint32_t at, uint32_t v, Nothing) { perm[at] = v; });
}

__global__ void k_gather(const uint32_t* __restrict__ perm, uint32_t n, const float4* __restrict__ a_in,
                         float4* __restrict__ a_out, const float4* __restrict__ b_in, float4* __restrict__ b_out,
                         const uint32_t* __restrict__ c_in, uint32_t* __restrict__ c_out,
                         const uint32_t* __restrict__ d_in, uint32_t* __restrict__ d_out) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t s = perm[k];
    if (a_out) a_out[k] = a_in[s];
    if (b_out) b_out[k] = b_in[s];
    if (c_out) c_out[k] = c_in[s];
    if (d_out) d_out[k] = d_in[s];
}

__device__ __forceinline__ float eos_pressure(uint32_t eq, float density, float c, float d0) {
    switch (eq) {  // fluid.rs:45-52, x^7 by products
        case ARP_EOS_CONSTANT: return c * c;
        case ARP_EOS_IDEAL_GAS: return c * c * (density - d0);
        case ARP_EOS_TAIT: {
            const float x = density / d0;
            const float x2 = x * x;
            const float x3 = x2 * x;
            const float x6 = x3 * x3;
            return (c * c * d0 / 7.0f) * (x6 * x - 1.0f);
        }
        default: return 0.0f;
    }
}

// What a gather of a state reads and writes: slot s of the source goes to
// sorted position k.  Null pointers are skipped.
struct GatherArgs {
    const float4 *pd_in, *vm_in;
    float4 *pd_out, *vm_out;
    const uint32_t *a_in, *b_in;
    uint32_t *a_out, *b_out;
    float* ps_out;
    SolidScatter sol;
    DevStats* stats;
    PairOut out;
};
struct Gathered {
    float4 pd, vm;
    float ps;  // p / rho^2
    uint32_t code, local, sid, a, b;
    uint2 coord;
};
__device__ __forceinline__ Gathered gather_load(const GatherArgs& g, const Tables& T, uint32_t s) {
    Gathered r{};
    r.pd = g.pd_in[s];
    r.vm = g.vm_in[s];
    r.sid = g.sol.sx ? g.sol.sid_of_slot[s] : kInvalid;
    if (r.sid != kInvalid) r.coord = g.sol.coord_of_slot[s];
    if (g.a_out) r.a = g.a_in[s];
    if (g.b_out) r.b = g.b_in[s];
    const float4 pd = r.pd;
    const DevMat& m = T.mats[__float_as_uint(r.vm.w)];
    if (g.stats) {
        if (!finite3(pd)) {
            atomicAdd(&g.stats->nonfinite_positions, 1u);
        } else {
            // a coordinate on the upper face would hash one past the last cell
            const Grid& gr = T.scenes[m.scene].grid;
            const bool face = (gr.dim[0] != 0.0f && pd.x == gr.min[0] + gr.dim[0]) ||
                              (gr.dim[1] != 0.0f && pd.y == gr.min[1] + gr.dim[1]) ||
                              (gr.dim[2] != 0.0f && pd.z == gr.min[2] + gr.dim[2]);
            if (face) atomicAdd(&g.stats->clamped_coordinates, 1u);
        }
    }
    const float p = eos_pressure(m.state_eq, pd.w, m.sound_speed, m.target_den);
    r.ps = p / (pd.w * pd.w);
    if (g.out.rec) {
        r.code = scan_code(pd, T.scenes[m.scene], T.flat);
        r.local = m.local;
    }
    return r;
}
__device__ __forceinline__ void gather_store(const GatherArgs& g, uint32_t k, const Gathered& r) {
    if (g.pd_out) g.pd_out[k] = r.pd;
    if (g.vm_out) g.vm_out[k] = r.vm;
    if (r.sid != kInvalid) {
        g.sol.sx[2 * (size_t)r.sid] = r.pd;
        g.sol.sv[r.sid] = r.vm;
        g.sol.sc[r.sid] = r.coord;
        if (g.sol.slot_of) g.sol.slot_of[r.sid] = k;
    }
    if (g.a_out) g.a_out[k] = r.a;
    if (g.b_out) g.b_out[k] = r.b;
    if (g.ps_out) g.ps_out[k] = r.ps;
    if (g.out.rec) {
        g.out.rec[2 * (size_t)k] = r.pd;
        g.out.rec[2 * (size_t)k + 1] = make_float4(r.vm.x, r.vm.y, r.vm.z, r.ps);
        g.out.code[k] = r.code;
        g.out.mat8[k] = (uint8_t)r.local;
        if (g.out.mat) g.out.mat[k] = __float_as_uint(r.vm.w);
    }
}

__global__ void k_gather_state(const uint32_t* __restrict__ perm, uint32_t n, GatherArgs g, Tables T) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) gather_store(g, k, gather_load(g, T, perm ? perm[k] : k));
}

// Orders the block's cells and gathers the state of their particles.  With
// `stats` and up to kCountBeside blocks the grid is twice as long: the second half
// takes the occupancy counters of the reference cells, a chain of reads of its own
// that would double the latency of the ordering in a scene that leaves SMs idle.
// In larger grids, most of whose blocks are empty, each block counts its own
// cells: twice as many blocks cost more than the chain (us a stage, beside / by
// itself: 4,820 blocks of a batch 33 / 37, 8,790 29 / 27, 55,962 161 / 128).
// `count` (null: the scan has done it) is cleared on the way.
constexpr uint32_t kCountBeside = 8192;
__global__ void __launch_bounds__(kThreads) k_order_gather(const uint32_t* start, uint32_t ncells, uint32_t nblocks,
                                                           uint32_t* perm, uint32_t* tmp, const uint32_t* key,
                                                           uint32_t* count,
                                                           const uint32_t* boundary_start, DevStats* stats,
                                                           GatherArgs g, Tables T) {
    step_begin();
    const bool counts = blockIdx.x >= nblocks;
    const uint32_t c = (counts ? blockIdx.x - nblocks : blockIdx.x) * kThreads + threadIdx.x;
    if (counts || (stats && gridDim.x == nblocks)) {
        const uint32_t occ = c < ncells ? reference_cell_occupancy(c, start, boundary_start, T) : 0u;
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, occ);
        const uint32_t over = __popc(__ballot_sync(0xFFFFFFFFu, occ > kBucketSlots));
        if ((threadIdx.x & 31u) == 0u) {
            if (most > 0u) atomicMax(&stats->max_cell_occupancy, most);
            if (over > 0u) atomicAdd(&stats->overflow_cells, over);
        }
        if (counts) return;
    }
    if (count && c < ncells + 2u) count[c] = 0u;  // ready for the next histogram
    order_block<true>(start, ncells, perm, tmp, key, [&](uint32_t v) { return gather_load(g, T, v); },
                [&](uint32_t at, uint32_t v, const Gathered& r) {
                    perm[at] = v;
                    gather_store(g, at, r);
                });
}

// Particle records (48 B, caller order) -> structure of arrays in caller order.
__global__ void k_records_to_soa(const arp_particle* __restrict__ in, uint32_t n, const uint32_t* __restrict__ sid_of,
                                 const uint32_t* __restrict__ mat_of, float4* __restrict__ pd, float4* __restrict__ vm,
                                 uint32_t* __restrict__ orig, uint32_t* __restrict__ sid) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4* r = reinterpret_cast<const float4*>(in + i);
    const float4 h = r[0], p = r[1], v = r[2];  // (den, mat, solid_id, pad), pos, vel
    pd[i] = make_float4(p.x, p.y, p.z, h.x);
    vm[i] = make_float4(v.x, v.y, v.z, __uint_as_float(mat_of[i]));  // batch-wide material id
    orig[i] = i;
    sid[i] = sid_of[i];
}

// Bit 0: a record's material differs from the handle's; bit 1: a w component
// differs from the handle's common w / zero.
__global__ void k_check_records(const arp_particle* __restrict__ in, uint32_t n, const uint32_t* __restrict__ mat_of,
                                const DevMat* __restrict__ mats, float pos_w, uint32_t* __restrict__ flag) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const arp_particle& r = in[i];
    uint32_t bad = (r.mat != mats[mat_of[i]].local) ? 1u : 0u;
    if (r.pos[3] != pos_w || r.vel[3] != 0.0f) bad |= 2u;
    if (bad) atomicOr(flag, bad);
}

// Cell-ordered structure of arrays -> particle records in caller order.
__global__ void k_soa_to_records(const float4* __restrict__ pd, const float4* __restrict__ vm,
                                 const uint32_t* __restrict__ orig, const uint32_t* __restrict__ sid, uint32_t n,
                                 float pos_w, const DevMat* __restrict__ mats, arp_particle* __restrict__ out) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 p = pd[k], v = vm[k];
    float4* r = reinterpret_cast<float4*>(out + orig[k]);
    const DevMat& m = mats[__float_as_uint(v.w)];
    const uint32_t sk = sid[k];
    // the scene's own material index and solid id
    r[0] = make_float4(p.w, __uint_as_float(m.local), __uint_as_float(sk == kInvalid ? sk : sk - m.solid_base), 0.0f);
    r[1] = make_float4(p.x, p.y, p.z, pos_w);
    r[2] = make_float4(v.x, v.y, v.z, 0.0f);
}

__device__ __forceinline__ bool within_h_exact(float4 q, float4 p, float h2) {
    const float rx = __fsub_rn(q.x, p.x), ry = __fsub_rn(q.y, p.y), rz = __fsub_rn(q.z, p.z);
    const float d = __fadd_rn(__fadd_rn(__fmul_rn(rx, rx), __fmul_rn(ry, ry)), __fmul_rn(rz, rz));
    return __fsub_rn(h2, d) > 0.0f;
}

__global__ void k_count_neighbors(const float4* __restrict__ xs, const float4* __restrict__ vs,
                                  const uint32_t* __restrict__ start, uint32_t n, const float4* __restrict__ bxs,
                                  const uint32_t* __restrict__ bstart, Tables T, uint32_t* __restrict__ out) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 p = xs[k];
    uint32_t cnt = 0;
    if (finite3(p)) {
        const SceneP& P = T.scenes[scene_of(vs, nullptr, k, T)];
        // the shader's 3x3(x3) reference cells exactly
        for_reference_block_rows(p, P, [&](uint32_t c0, uint32_t c1) {
            if (bstart)
                for (uint32_t j = bstart[c0]; j < bstart[c1]; ++j) cnt += within_h_exact(bxs[j], p, P.h2);
            for (uint32_t j = start[c0]; j < start[c1]; ++j) cnt += within_h_exact(xs[j], p, P.h2);
        });
    }
    out[k] = cnt;
}

inline uint32_t blocks_for(uint32_t n, int t) { return (n + (uint32_t)t - 1u) / (uint32_t)t; }

// ---- allocation-free grid build ---------------------------------------------
// Scratch of arp_grid_build_noalloc: arrival ranks of up to kNoAllocMaxParticles
// particles, then the scan's tile totals.  The histogram and its scan live in
// the caller's cell_start array, and cell keys are recomputed from the
// positions instead of stored.  4 MiB + 4 KiB per GPU that loads the library.
constexpr uint32_t kNoAllocMaxParticles = 1u << 20;
constexpr uint32_t kNoAllocMaxCells = (1u << 22) - 2;  // cell_start then holds at most 2^22 entries
constexpr uint32_t kNoAllocMaxTiles = (kNoAllocMaxCells + 2 + kScanTile - 1) / kScanTile;
__device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocMaxParticles + kNoAllocMaxTiles];

__global__ void k_rank_noalloc(const float4* pos, uint32_t n, Grid grid, uint32_t* count,
                               uint32_t* rank) {
    step_begin();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const uint32_t k = finite3(p) ? cell_id(cell_coord(p, grid), grid) : grid.ncells;
    rank[i] = atomicAdd(&count[k], 1u);
}

__global__ void k_scatter_noalloc(const float4* pos, uint32_t n, Grid grid,
                                  const uint32_t* start, const uint32_t* rank,
                                  uint32_t* perm) {
    step_begin();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const uint32_t k = finite3(p) ? cell_id(cell_coord(p, grid), grid) : grid.ncells;
    perm[start[k] + rank[i]] = i;
}

// Device address of g_noalloc_scratch, looked up once per device with that
// device current (host code may not use the symbol itself as an address).
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
uint32_t* g_noalloc_ptr[kMaxDevices] = {};

cudaError_t noalloc_scratch(uint32_t** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = static_cast<uint32_t*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

}  // namespace

int bin_cells(const float4* pos, const float4* vm, const uint32_t* mat_u32, uint32_t n, const Tables& T,
              GridBuffers& gb, uint32_t* zero, cudaStream_t st) {
    int launches = 0;
    clear_cells(T, gb, st);
    if (n > 0) {
        // a single scene needs no material to find the scene: skip that read
        const bool one = T.nscenes == 1;
        launch_step(k_cell_keys, blocks_for(n, kThreads), kThreads, 0, st, pos, one ? nullptr : vm, one ? nullptr : mat_u32, n,
                                                                  T, cell_bins(gb));
        ++launches;
    }
    return launches + scatter_cells(n, T, gb, zero, st);
}

void clear_cells(const Tables& T, GridBuffers& gb, cudaStream_t st) {
    // a state that was scattered and then replaced never reached the ordering,
    // which clears the counts
    if (gb.scattered) cudaMemsetAsync(gb.count, 0, (size_t(T.ncells) + 2) * sizeof(uint32_t), st);
    gb.scattered = false;
}

int scatter_cells(uint32_t n, const Tables& T, GridBuffers& gb, uint32_t* zero, cudaStream_t st) {
    const uint32_t len = T.ncells + 2;  // cells, the non-finite bucket, and the total
    const uint32_t tiles = blocks_for(len, kScanTile);
    if (tiles > kBaseTiles) {
        // exclusive_scan clears the counts
        const int l = exclusive_scan(gb.count, len, gb.start, gb.block_sums, st);
        launch_step(k_scatter_plain, std::max(blocks_for(n, kThreads), 1u), kThreads, 0, st, gb.key, gb.rank, n, gb.start,
                                                                                    gb.perm, zero);
        return l + 1;
    }
    gb.scattered = true;
    launch_step(k_scan_tiles<false>, tiles, kScanThreads, 0, st, gb.count, len, gb.count, gb.block_sums, true);
    const uint32_t work = std::max(n, (len + 3u) / 4u);
    launch_step(k_scatter, blocks_for(work, kThreads), kThreads, 0, st, gb.key, gb.rank, n, gb.count, gb.block_sums, len,
                                                               gb.start, gb.perm, zero);
    return 2;
}

// the counts for an ordering to clear: none where the scan has cleared them
static uint32_t* take_counts(GridBuffers& gb) {
    uint32_t* const count = gb.scattered ? gb.count : nullptr;
    gb.scattered = false;
    return count;
}

int order_cells(const Tables& T, GridBuffers& gb, cudaStream_t st) {
    uint32_t* const count = take_counts(gb);
    launch_step(k_order, blocks_for(T.ncells + 2, kThreads), kThreads, 0, st, gb.start, T.ncells, gb.perm, gb.rank,
                count);
    return 1;
}

int order_gather(const Tables& T, GridBuffers& gb, const uint32_t* boundary_start, const float4* pd_in, float4* pd_out,
                 const float4* vm_in, float4* vm_out, const uint32_t* a_in, uint32_t* a_out, const uint32_t* b_in,
                 uint32_t* b_out, cudaStream_t st, const SolidScatter& sol, DevStats* stats, const PairOut& out) {
    uint32_t* const count = take_counts(gb);
    const GatherArgs g{pd_in, vm_in, pd_out, vm_out, a_in, b_in, a_out, b_out, nullptr, sol, stats, out};
    const uint32_t nb = blocks_for(T.ncells + 2, kThreads);
    launch_step(k_order_gather, stats && nb <= kCountBeside ? 2 * nb : nb, kThreads, 0, st, gb.start, T.ncells, nb, gb.perm, gb.rank, gb.key,
                count, boundary_start, stats, g, T);
    return 1;
}

int build_grid(const float4* pos, const float4* vm, const uint32_t* mat_u32, uint32_t n, const Tables& T,
               GridBuffers& gb, cudaStream_t st) {
    const int l = bin_cells(pos, vm, mat_u32, n, T, gb, nullptr, st);
    return l + order_cells(T, gb, st);
}

uint32_t scan_block_sums_needed(uint32_t len) { return blocks_for(len, kScanTile) + 1; }

int exclusive_scan(uint32_t* count, uint32_t len, uint32_t* out, uint32_t* block_sums, cudaStream_t st) {
    const uint32_t tiles = blocks_for(len, kScanTile);
    const bool wide = ((reinterpret_cast<uintptr_t>(count) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0u;
    if (count == out) launch_step(k_scan_tiles<false>, tiles, kScanThreads, 0, st, count, len, out, block_sums, wide);
    else launch_step(k_scan_tiles<true>, tiles, kScanThreads, 0, st, count, len, out, block_sums, wide);
    launch_step(k_scan_add, tiles, kScanThreads, 0, st, out, len, block_sums);
    return 2;
}

int gather_sorted(const uint32_t* perm, uint32_t n, const float4* a_in, float4* a_out, const float4* b_in,
                  float4* b_out, const uint32_t* c_in, uint32_t* c_out, const uint32_t* d_in, uint32_t* d_out,
                  cudaStream_t st) {
    if (n == 0) return 0;
    k_gather<<<blocks_for(n, kThreads), kThreads, 0, st>>>(perm, n, a_in, a_out, b_in, b_out, c_in, c_out, d_in,
                                                           d_out);
    return 1;
}

int gather_state(const uint32_t* perm, uint32_t n, const float4* pd_in, float4* pd_out, const float4* vm_in,
                 float4* vm_out, const uint32_t* a_in, uint32_t* a_out, const uint32_t* b_in, uint32_t* b_out,
                 float* ps_out, const Tables& T, cudaStream_t st, const PairOut& out) {
    if (n == 0) return 0;
    const GatherArgs g{pd_in, vm_in, pd_out, vm_out, a_in, b_in, a_out, b_out, ps_out, SolidScatter{}, nullptr, out};
    k_gather_state<<<blocks_for(n, kThreads), kThreads, 0, st>>>(perm, n, g, T);
    return 1;
}

int records_to_soa(const arp_particle* in, uint32_t n, const uint32_t* sid_of, const uint32_t* mat_of, float4* pd,
                   float4* vm, uint32_t* orig, uint32_t* sid, cudaStream_t st) {
    if (n == 0) return 0;
    k_records_to_soa<<<blocks_for(n, kThreads), kThreads, 0, st>>>(in, n, sid_of, mat_of, pd, vm, orig, sid);
    return 1;
}

int check_records(const arp_particle* in, uint32_t n, const uint32_t* mat_of, const DevMat* mats, float pos_w,
                  uint32_t* flag, cudaStream_t st) {
    if (n == 0) return 0;
    k_check_records<<<blocks_for(n, kThreads), kThreads, 0, st>>>(in, n, mat_of, mats, pos_w, flag);
    return 1;
}

int soa_to_records(const float4* pd, const float4* vm, const uint32_t* orig, const uint32_t* sid, uint32_t n,
                   float pos_w, const DevMat* mats, arp_particle* out, cudaStream_t st) {
    if (n == 0) return 0;
    k_soa_to_records<<<blocks_for(n, kThreads), kThreads, 0, st>>>(pd, vm, orig, sid, n, pos_w, mats, out);
    return 1;
}

int count_neighbors(const float4* xs, const float4* vs, const uint32_t* start, uint32_t n, const float4* bxs,
                    const uint32_t* bstart, const Tables& T, uint32_t* out_sorted, cudaStream_t st) {
    if (n == 0) return 0;
    k_count_neighbors<<<blocks_for(n, kThreads), kThreads, 0, st>>>(xs, vs, start, n, bxs, bstart, T, out_sorted);
    return 1;
}

}  // namespace arp

// ---- C ABI: allocation-free grid build ----------------------------------------
extern "C" arp_status arp_grid_build_noalloc(const void* pos_den, uint32_t n, const arp_aabb* bounds,
                                             float kernel_radius, uint32_t* cell_start,
                                             uint32_t cell_start_capacity, uint32_t* perm, void* stream) {
    using namespace arp;
    if (!bounds) return set_error(ARP_ERR_INVALID_ARG, "bounds is null");
    if (!(kernel_radius > 0.0f)) return set_error(ARP_ERR_INVALID_ARG, "kernel_radius must be positive");
    if (bounds->dim[3] > 0.0f) return set_error(ARP_ERR_UNSUPPORTED, "4-dimensional boxes are not supported");
    if (n > kNoAllocMaxParticles)
        return set_error(ARP_ERR_CAPACITY, "arp_grid_build_noalloc: n exceeds the 1048576-particle maximum");
    if (n > 0 && (!pos_den || !perm)) return set_error(ARP_ERR_INVALID_ARG, "null position or perm pointer");
    if (!cell_start) return set_error(ARP_ERR_INVALID_ARG, "cell_start is null");
    if (reinterpret_cast<uintptr_t>(pos_den) % 16 != 0)
        return set_error(ARP_ERR_INVALID_ARG, "pos_den must be 16-byte aligned (float4 records)");
    Grid g{};
    uint64_t nc = 1;
    for (int a = 0; a < 3; ++a) {
        if (!std::isfinite(bounds->min[a]) || !std::isfinite(bounds->dim[a]) || bounds->dim[a] < 0.0f)
            return set_error(ARP_ERR_INVALID_ARG, "bounds must be finite with non-negative extent");
        g.min[a] = bounds->min[a];
        g.dim[a] = bounds->dim[a];
        // neighbor_list.rs:201-206; the quotient is range-checked in float
        // before the conversion (a huge dim / h would not fit in 32 bits)
        const float q = std::max(1.0f, bounds->dim[a] / kernel_radius);
        if (!(q <= (float)kNoAllocMaxCells))
            return set_error(ARP_ERR_CAPACITY, "arp_grid_build_noalloc: the grid exceeds the 4194302-cell maximum");
        g.sub[a] = (uint32_t)q;
        nc *= g.sub[a];
    }
    if (nc > kNoAllocMaxCells)
        return set_error(ARP_ERR_CAPACITY, "arp_grid_build_noalloc: the grid exceeds the 4194302-cell maximum");
    g.ncells = (uint32_t)nc;
    if ((uint64_t)cell_start_capacity < nc + 2)
        return set_error(ARP_ERR_CAPACITY, "cell_start must hold n_cells + 2 entries (" + std::to_string(nc + 2) +
                                               ")");
    uint32_t* scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) return set_error(ARP_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    uint32_t* rank = scratch;
    uint32_t* tile_sums = scratch + kNoAllocMaxParticles;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t len = g.ncells + 2;
    e = cudaMemsetAsync(cell_start, 0, (size_t)len * sizeof(uint32_t), st);
    if (e != cudaSuccess) return set_error(ARP_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    const float4* pos = static_cast<const float4*>(pos_den);
    if (n > 0) launch_step(k_rank_noalloc, blocks_for(n, kThreads), kThreads, 0, st, pos, n, g, cell_start, rank);
    exclusive_scan(cell_start, len, cell_start, tile_sums, st);  // in place: counts become starts
    if (n > 0) launch_step(k_scatter_noalloc, blocks_for(n, kThreads), kThreads, 0, st, pos, n, g, cell_start, rank, perm);
    if (n > 0) launch_step(k_order, blocks_for(g.ncells + 1, kThreads), kThreads, 0, st, cell_start, g.ncells, perm, rank, nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(ARP_ERR_CUDA, std::string("grid build launch: ") + cudaGetErrorString(e));
    return ARP_OK;
}
