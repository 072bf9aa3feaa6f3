// renderer.cu -- headless point-splat rendering of the particle state.
//
// Replaces the recording path of the reference's demo renderer
// (examples/test_mods/renderer.rs:4-137 shaders, :305-478 frame set-up and
// glReadnPixels) with CUDA rasterisation into an 8-bit RGB frame:
//   * k_rp_project: the vertex shader -- view matrix (renderer.rs:338-349),
//     clip test, viewport mapping, density colour ramp (renderer.rs:45-55);
//   * without lighting, sprites are binned by (16x16 tile, draw-order chunk),
//     each bin is sorted by draw order, and each tile's sprites are composited
//     per pixel in that order with the blend the reference sets
//     (ONE_MINUS_DST_ALPHA, ONE_MINUS_SRC_ALPHA, DST_ALPHA, SRC_ALPHA), the
//     fragment alpha weighted by the poly6 kernel across the disc
//     (renderer.rs:121-128), channels rounded to 8 bits after every blend as a
//     RGBA8 target stores them;
//   * with lighting, a depth pass keeps the nearest sprite of each pixel (depth
//     test LESS, the first drawn on ties) and a shading pass lights it as a
//     sphere (renderer.rs:99-119).
// Fragments sit at pixel centres; a sprite covers the centres inside its
// square [c - S/2, c + S/2) and gl_PointCoord has its origin at the upper left.
#include "grid.cuh"

namespace arp {

namespace {

constexpr int kTile = 16;
constexpr int kChunk = 1024;  // sprites per draw-order chunk

inline uint32_t nblk(uint32_t n, int t) { return (n + (uint32_t)t - 1u) / (uint32_t)t; }

__device__ __forceinline__ float mixf(float x, float y, float a) {
    return __fadd_rn(__fmul_rn(x, __fsub_rn(1.0f, a)), __fmul_rn(y, a));
}

// Vertex stage of one particle: window position, clip w ("depth"), window z,
// colour.  Invalid sprites get alpha 0 (discarded).
__device__ void project(float4 pd, float4 vm, const RenderCfg& c, float4& PR, float4& PC, float4& PP) {
    PR = make_float4(0.f, 0.f, 0.f, 0.f);
    PC = make_float4(0.f, 0.f, 0.f, 0.f);
    PP = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t mat = __float_as_uint(vm.w);
    if (mat >= c.nmat || !finite3(pd)) return;
    // pos2 = trans * (pos, 1), trans columns (cos t, 0, sin t, 0), (0, 1, 0, 0), (-sin t, 0, cos t, 0), (tx, ty, tz, 1)
    const float x2 = __fadd_rn(__fadd_rn(__fmul_rn(c.ca, pd.x), __fmul_rn(-c.sa, pd.z)), c.tx);
    const float y2 = __fadd_rn(pd.y, c.ty);
    const float z2 = __fadd_rn(__fadd_rn(__fmul_rn(c.sa, pd.x), __fmul_rn(c.ca, pd.z)), c.tz);
    const float w = __fadd_rn(z2, 1.0f);
    if (!(w > 0.0f) || x2 < -w || x2 > w || y2 < -w || y2 > w || z2 < -w || z2 > w) return;  // point clipping
    const float xn = __fdiv_rn(x2, w), yn = __fdiv_rn(y2, w), zn = __fdiv_rn(z2, w);
    const float half = 0.5f * c.s2;
    const float xw = __fadd_rn(__fmul_rn(__fadd_rn(xn, 1.0f), half), c.vx0);
    const float yw = __fadd_rn(__fmul_rn(__fadd_rn(yn, 1.0f), half), c.vy0);
    const float zw = __fmul_rn(__fadd_rn(zn, 1.0f), 0.5f);
    // density colour ramp (renderer.rs:45-55)
    const float d0 = c.d0[mat];
    const float dd = __fdiv_rn(__fsub_rn(pd.w, d0), d0);
    const float4 base = c.c2[mat];
    const float4 other = dd < 0.0f ? c.c1[mat] : c.c3[mat];
    const float t = dd < 0.0f ? __fdiv_rn(-dd, 5.0f) : __fdiv_rn(dd, 5.0f);
    float4 col = make_float4(mixf(base.x, other.x, t), mixf(base.y, other.y, t), mixf(base.z, other.z, t),
                             mixf(base.w, other.w, t));
    col.w = fminf(1.0f, col.w);
    PR = make_float4(xw, yw, w, zw);
    PC = col;
    PP = make_float4(x2, y2, z2, 0.0f);
}

__global__ void k_rp_project(const float4* __restrict__ pd, const float4* __restrict__ vm,
                             const uint32_t* __restrict__ orig, uint32_t n, uint32_t prim_base, RenderCfg c,
                             float4* __restrict__ PR, float4* __restrict__ PC, float4* __restrict__ PP) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t prim = prim_base + orig[k];
    float4 r, col, p;
    project(pd[k], vm[k], c, r, col, p);
    PR[prim] = r;
    PC[prim] = col;
    PP[prim] = p;
}

// Half extent of the pixels a sprite can cover: its square, and the disc
// |d| <= 1 with d = 2 (fragment - centre) / S * 2 w.
__device__ __forceinline__ float sprite_reach(const RenderCfg& c, float w) {
    return fminf(0.5f * c.S, __fdiv_rn(c.S, 4.0f * w)) + 1.0f;
}

// d = 2 (fragment - centre) / S * 2 w along x or y at a pixel centre;
// gl_PointCoord (upper-left origin), p = (pc - 0.5) * 2 with p.y negated,
// d = p * 2 * depth
__device__ __forceinline__ float sprite_dx(const RenderCfg& c, float4 r, float fx) {
    const float s = __fadd_rn(0.5f, __fdiv_rn(__fsub_rn(fx, r.x), c.S));
    return __fmul_rn(__fmul_rn(__fmul_rn(__fsub_rn(s, 0.5f), 2.0f), 2.0f), r.z);
}
__device__ __forceinline__ float sprite_dy(const RenderCfg& c, float4 r, float fy) {
    const float t = __fsub_rn(0.5f, __fdiv_rn(__fsub_rn(fy, r.y), c.S));
    return __fmul_rn(__fmul_rn(-__fmul_rn(__fsub_rn(t, 0.5f), 2.0f), 2.0f), r.z);
}
// Whether a pixel centre's coordinate f lies in a sprite's square around r.
__device__ __forceinline__ bool in_square(const RenderCfg& c, float r, float f) {
    const float hs = 0.5f * c.S;
    return !(f < __fsub_rn(r, hs)) && !(f >= __fadd_rn(r, hs));
}

// Coverage of the pixel centre (fx, fy) by a sprite; r2 = dot(d, d) when covered.
__device__ __forceinline__ bool covers(const RenderCfg& c, float4 r, float fx, float fy, float& dx, float& dy,
                                       float& r2) {
    if (!in_square(c, r.x, fx) || !in_square(c, r.y, fy)) return false;
    dx = sprite_dx(c, r, fx);
    dy = sprite_dy(c, r, fy);
    r2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    return r2 <= 1.0f;
}

__device__ __forceinline__ void tile_range(const RenderCfg& c, float4 r, int& tx0, int& tx1, int& ty0, int& ty1) {
    const float R = sprite_reach(c, r.z);
    tx0 = max(0, (int)floorf((r.x - R) / kTile));
    tx1 = min((int)c.tiles_x - 1, (int)floorf((r.x + R) / kTile));
    ty0 = max(0, (int)floorf((r.y - R) / kTile));
    ty1 = min((int)c.tiles_y - 1, (int)floorf((r.y + R) / kTile));
}

// Bin of a sprite in a tile: a tile's bins lie together, in draw order.
__device__ __forceinline__ size_t bin_of(const RenderCfg& c, uint32_t prim, int tx, int ty) {
    const uint32_t nchunks = (c.nprims + kChunk - 1) / kChunk;
    return ((size_t)ty * c.tiles_x + tx) * nchunks + prim / kChunk;
}

// pass 1 of the binning: sprites per (tile, chunk)
__global__ void k_rp_count(const float4* __restrict__ PR, const float4* __restrict__ PC, RenderCfg c,
                           uint32_t* __restrict__ counts) {
    const uint32_t prim = blockIdx.x * blockDim.x + threadIdx.x;
    if (prim >= c.nprims) return;
    const float4 r = PR[prim];
    if (PC[prim].w == 0.0f) return;
    int tx0, tx1, ty0, ty1;
    tile_range(c, r, tx0, tx1, ty0, ty1);
    for (int ty = ty0; ty <= ty1; ++ty)
        for (int tx = tx0; tx <= tx1; ++tx) atomicAdd(&counts[bin_of(c, prim, tx, ty)], 1u);
}

// pass 2: sprite ids into their (tile, chunk) segments (any order inside)
__global__ void k_rp_scatter(const float4* __restrict__ PR, const float4* __restrict__ PC, RenderCfg c,
                             const uint32_t* __restrict__ start, uint32_t* __restrict__ fill,
                             uint32_t* __restrict__ list) {
    const uint32_t prim = blockIdx.x * blockDim.x + threadIdx.x;
    if (prim >= c.nprims) return;
    const float4 r = PR[prim];
    if (PC[prim].w == 0.0f) return;
    int tx0, tx1, ty0, ty1;
    tile_range(c, r, tx0, tx1, ty0, ty1);
    for (int ty = ty0; ty <= ty1; ++ty)
        for (int tx = tx0; tx <= tx1; ++tx) {
            const size_t key = bin_of(c, prim, tx, ty);
            list[start[key] + atomicAdd(&fill[key], 1u)] = prim;
        }
}

// Sprite ids of every bin into draw order.  A warp takes 32 bins; the ids of one
// bin share a chunk, so a bin of two or more is sorted by a bit per sprite of
// the chunk: lane l holds the bits of sprites 32 l .. 32 l + 31 and writes its
// ids after those of the lanes below.  34 us for the 2.5 M bins of a 1920 x 1080
// frame of 314,000 sprites, most of them empty.
constexpr int kSortWarps = 8;
__global__ void __launch_bounds__(kSortWarps * 32) k_rp_sort(const uint32_t* __restrict__ start, uint32_t nbins,
                                                             uint32_t* __restrict__ list) {
    static_assert(kChunk == 1024, "32 bits per lane");
    __shared__ uint32_t s_bits[kSortWarps][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x / 32u;
    uint32_t* const bits = s_bits[warp];
    const uint32_t bin = (blockIdx.x * kSortWarps + warp) * 32u + lane;
    const uint32_t b = bin < nbins ? start[bin] : 0u, e = bin < nbins ? start[bin + 1] : 0u;
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, e - b > 1u); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, b, src), s1 = __shfl_sync(0xFFFFFFFFu, e, src);
        bits[lane] = 0u;
        __syncwarp();
        const uint32_t chunk = list[s0] / kChunk * kChunk;
#pragma unroll 4
        for (uint32_t i = s0 + lane; i < s1; i += 32u) {
            const uint32_t k = list[i] - chunk;
            atomicOr(&bits[k / 32u], 1u << (k & 31u));
        }
        __syncwarp();
        uint32_t w = bits[lane];
        const uint32_t own = __popc(w);
        uint32_t incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += v;
        }
        for (uint32_t at = s0 + incl - own; w; w &= w - 1u) list[at++] = chunk + lane * 32u + __ffs(w) - 1u;
        __syncwarp();
    }
}

// v, clamped to [0, 1], to 8 bits, kept as a float: the floor of v 255 + 0.5 is
// its sum with 2^23 rounded down.
__device__ __forceinline__ float round8(float v) {
    v = __saturatef(v);
    return __fadd_rd(__fadd_rn(__fmul_rn(v, 255.0f), 0.5f), 8388608.0f) - 8388608.0f;
}
__device__ __forceinline__ uint8_t to8(float v) { return (uint8_t)round8(v); }
// q / 255, correctly rounded for every q in 0 .. 255 (checked for all 256): the
// multiplication by a constant held in two floats of Brisebarre and Muller.
__device__ __forceinline__ float from8(float q) {
    return __fmaf_rn(q, 0x1.010102p-8f, __fmul_rn(q, -0x1.fdfdfep-33f));
}

// wk / kconst, correctly rounded likewise for the weight wk of every 1 - r2
// (multiples of 2^-24 in [0, 1]; all checked)
__device__ __forceinline__ float by_kconst(const RenderCfg& c, float wk) {
    return __fmaf_rn(wk, c.kinv_hi, __fmul_rn(wk, c.kinv_lo));
}

// A warp composites 8 x 4 pixels of a tile by itself: it reads the tile's sprites
// in draw order 32 at a time, keeps those that reach its pixels and, for each 32
// kept, computes their squared offsets along its 8 columns and 4 rows once for
// all pixels (lane = sprite); then each lane (= pixel) marks the sprites that
// cover it and blends them in turn, two weights at a time.  Bound by the blends,
// a serial chain per pixel, and by how evenly the tiles' sprites spread (a sixth
// of the lanes a sprite's visit holds are covered, hence a mask per pixel).
// With a block per tile, a chunk at a time (a sort and 4 barriers each), every
// pixel visiting every sprite of the tile, two divisions for its offset and
// three divisions a blend, a 1920 x 1080 frame of 314,000 sprites (631,000
// sprite-tile pairs, 3,289 in the fullest tile) took 2017 us; now 119.
constexpr int kPatchX = 8, kPatchY = 4, kPatches = kTile * kTile / 32;
constexpr int kCompWarps = 4;
struct PatchStage {
    float off[kPatchX + kPatchY][36];  // squared offsets by column / row, then sprite (rows 16-byte aligned)
    float4 col[32];
    uint32_t ids[64];
};
__global__ void __launch_bounds__(kCompWarps * 32) k_rp_composite(const float4* __restrict__ PR,
                                                                   const float4* __restrict__ PC, RenderCfg c,
                                                                   const uint32_t* __restrict__ start,
                                                                   const uint32_t* __restrict__ list,
                                                                   uint8_t* __restrict__ rgb) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    __shared__ __align__(16) PatchStage s_stage[kCompWarps];
    const uint32_t lane = threadIdx.x & 31u;
    PatchStage& st = s_stage[threadIdx.x / 32u];
    const uint32_t patch = blockIdx.x * kCompWarps + threadIdx.x / 32u;
    const uint32_t tile = patch / kPatches, sub = patch % kPatches;
    const uint32_t x0 = tile % c.tiles_x * kTile + sub % (kTile / kPatchX) * kPatchX;
    const uint32_t y0 = tile / c.tiles_x * kTile + sub / (kTile / kPatchX) * kPatchY;
    const uint32_t lx = lane % kPatchX, ly = lane / kPatchX;
    // The target starts white with alpha 0; a blend's alpha sa da + da sa keeps
    // it 0, so its colour is src + dst (1 - sa).
    float q[3] = {255.0f, 255.0f, 255.0f};
    const uint32_t nchunks = (c.nprims + kChunk - 1) / kChunk;
    const uint32_t b = nchunks ? start[(size_t)tile * nchunks] : 0u;
    const uint32_t e = nchunks ? start[(size_t)(tile + 1) * nchunks] : 0u;
    // the patch's pixel centres, and how far from a sprite's centre it reaches
    const float cx = x0 + 0.5f * kPatchX, cy = y0 + 0.5f * kPatchY;

    auto blend = [&](uint32_t m) {  // the first m <= 32 listed sprites, one per lane
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < m) {
            r = PR[st.ids[lane]];
            st.col[lane] = PC[st.ids[lane]];
        }
#pragma unroll
        for (int k = 0; k < kPatchX; ++k) {
            const float f = x0 + k + 0.5f;
            const float d = lane < m && in_square(c, r.x, f) ? sprite_dx(c, r, f) : INFINITY;
            st.off[k][lane] = __fmul_rn(d, d);
        }
#pragma unroll
        for (int k = 0; k < kPatchY; ++k) {
            const float f = y0 + k + 0.5f;
            const float d = lane < m && in_square(c, r.y, f) ? sprite_dy(c, r, f) : INFINITY;
            st.off[kPatchX + k][lane] = __fmul_rn(d, d);
        }
        __syncwarp();
        const float* const ox = st.off[lx];
        const float* const oy = st.off[kPatchX + ly];
        unsigned mask = 0u;
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            const float4 u = *reinterpret_cast<const float4*>(ox + k), v = *reinterpret_cast<const float4*>(oy + k);
            if (__fadd_rn(u.x, v.x) <= 1.0f) mask |= 1u << k;
            if (__fadd_rn(u.y, v.y) <= 1.0f) mask |= 2u << k;
            if (__fadd_rn(u.z, v.z) <= 1.0f) mask |= 4u << k;
            if (__fadd_rn(u.w, v.w) <= 1.0f) mask |= 8u << k;
        }
        while (mask) {
            // a pixel with one sprite left blends a second that adds 0 to all of it
            float4 src[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const bool in = mask != 0u;
                const uint32_t k = in ? __ffs(mask) - 1u : 0u;
                mask &= mask - 1u;
                const float diff = in ? __fsub_rn(1.0f, __fadd_rn(ox[k], oy[k])) : 1.0f;
                const float4 q4 = st.col[k];
                const float wk = __fmul_rn(__fmul_rn(__fmul_rn(c.kconst, diff), diff), diff);
                const float keep = __fsub_rn(1.0f, __fmul_rn(q4.w, by_kconst(c, wk)));
                src[u] = in ? make_float4(q4.x, q4.y, q4.z, keep) : make_float4(0.f, 0.f, 0.f, 1.0f);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                q[0] = round8(__fadd_rn(src[u].x, __fmul_rn(from8(q[0]), src[u].w)));
                q[1] = round8(__fadd_rn(src[u].y, __fmul_rn(from8(q[1]), src[u].w)));
                q[2] = round8(__fadd_rn(src[u].z, __fmul_rn(from8(q[2]), src[u].w)));
            }
        }
        __syncwarp();
    };

    uint32_t kept = 0;
    uint32_t id = b + lane < e ? list[b + lane] : kInvalid;
    float4 r = id != kInvalid ? PR[id] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i = b; i < e; i += 32u) {
        const uint32_t id_now = id;
        const float4 r_now = r;
        id = i + 32u + lane < e ? list[i + 32u + lane] : kInvalid;  // in flight meanwhile
        if (id != kInvalid) r = PR[id];
        bool near = false;
        if (id_now != kInvalid) {
            const float reach = sprite_reach(c, r_now.z);  // a pixel more than the disc and the square
            near = fabsf(r_now.x - cx) <= reach + 0.5f * kPatchX && fabsf(r_now.y - cy) <= reach + 0.5f * kPatchY;
        }
        const unsigned m = __ballot_sync(FULL, near);
        if (near) st.ids[kept + __popc(m & ((1u << lane) - 1u))] = id_now;
        kept += __popc(m);
        __syncwarp();
        if (kept >= 32u) {
            blend(32u);
            kept -= 32u;
            if (lane < kept) st.ids[lane] = st.ids[32u + lane];
            __syncwarp();
        }
    }
    if (kept) blend(kept);
    const uint32_t px = x0 + lx, py = y0 + ly;
    if (px < c.W && py < c.H) {
        const size_t o = ((size_t)py * c.W + px) * 3;
        rgb[o] = (uint8_t)q[0];
        rgb[o + 1] = (uint8_t)q[1];
        rgb[o + 2] = (uint8_t)q[2];
    }
}

// Lighting: the nearest covering sprite of each pixel (depth LESS, the first
// drawn on ties): min over (window depth bits, draw order).  Bound by the
// atomics: with one for every covered pixel, and both offsets divided for every
// pixel, 62 us for 314,000 sprites 64 layers deep; 42 now.
// LANES threads take the rows of one sprite in turn: a thread that walks a large
// sprite alone waits for what its pixels hold row after row.  Frames (ms), 1 / 8
// threads, sprites of 15, 32, 100 and 400 pixels: 314,000 at 1080p 0.41 / 0.45,
// 0.52 / 0.50, 1.6 / 1.2, 17.8 / 11.3; 100 at 720p 0.23 / 0.23, 0.30 / 0.23,
// 1.0 / 0.35, 15.1 / 2.1 (6.4 with an atomic for every covered pixel).  32
// threads: 0.57, 0.65, 1.7, 20.0 and 0.23, 0.23, 0.26, 0.85.
constexpr int kDepthBlock = 128, kDepthLanes = 8;
constexpr float kDepthAlone = 16.0f;  // sprites up to this size: a thread each
template <int LANES>
__global__ void k_rp_depth(const float4* __restrict__ PR, const float4* __restrict__ PC, RenderCfg c,
                           unsigned long long* __restrict__ zkey) {
    const uint32_t prim = blockIdx.x * (kDepthBlock / LANES) + threadIdx.x / LANES;
    if (prim >= c.nprims) return;
    const float4 r = PR[prim];
    if (PC[prim].w == 0.0f || !(r.w < 1.0f) || !(r.w >= 0.0f)) return;
    const float R = sprite_reach(c, r.z);
    const int i0 = max(0, (int)floorf(r.x - R)), i1 = min((int)c.W - 1, (int)ceilf(r.x + R));
    const int j0 = max(0, (int)floorf(r.y - R)), j1 = min((int)c.H - 1, (int)ceilf(r.y + R));
    const unsigned long long key = ((unsigned long long)__float_as_uint(r.w) << 32) | prim;
    constexpr int W = 8;  // columns at a time
    for (int ib = i0; ib <= i1; ib += W) {
        float dx2[W];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const float f = ib + u + 0.5f;
            const float dx = ib + u <= i1 && in_square(c, r.x, f) ? sprite_dx(c, r, f) : INFINITY;
            dx2[u] = __fmul_rn(dx, dx);
        }
        for (int j = j0 + (int)(threadIdx.x % LANES); j <= j1; j += LANES) {
            if (!in_square(c, r.y, j + 0.5f)) continue;
            const float dy = sprite_dy(c, r, j + 0.5f), dy2 = __fmul_rn(dy, dy);
            if (!(dy2 <= 1.0f)) continue;  // no pixel of the row is covered
            unsigned long long* const z = zkey + (size_t)j * c.W + ib;
#pragma unroll
            for (int u = 0; u < W; ++u)  // most sprites lie behind what a pixel already holds
                if (__fadd_rn(dx2[u], dy2) <= 1.0f && key < __ldcg(z + u)) atomicMin(z + u, key);
        }
    }
}

__global__ void k_rp_shade(const float4* __restrict__ PR, const float4* __restrict__ PC,
                           const float4* __restrict__ PP, RenderCfg c, const unsigned long long* __restrict__ zkey,
                           uint8_t* __restrict__ rgb) {
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= c.W * c.H) return;
    const unsigned long long key = zkey[pix];
    uint8_t out[3] = {255, 255, 255};
    const uint32_t prim = (uint32_t)(key & 0xFFFFFFFFull);
    if (prim != 0xFFFFFFFFu) {
        const float4 r = PR[prim], col = PC[prim], p = PP[prim];
        float dx, dy, r2;
        covers(c, r, (pix % c.W) + 0.5f, (pix / c.W) + 0.5f, dx, dy, r2);
        // normal = d.x e_x + d.y e_y + sqrt(1 - n.x^2 - n.y^2) (-e_z)
        const float nz = -sqrtf(1.0f - dx * dx - dy * dy);
        const float sx = p.x + c.render_h * dx, sy = p.y + c.render_h * dy, sz = p.z + c.render_h * nz;
        float lx = c.light[0] - sx, ly = c.light[1] - sy, lz = c.light[2] - sz;
        const float l = rsqrtf(lx * lx + ly * ly + lz * lz);
        const float l3 = l * l * l;
        lx *= l3;
        ly *= l3;
        lz *= l3;
        const float diffuse = lx * dx + ly * dy + lz * nz;
        const float ndl = dx * lx + dy * ly + nz * lz;
        const float rz = lz - 2.0f * ndl * nz;  // reflect(light, normal).z
        float spec = fmaxf(20.0f * rz, 0.0f);
        spec *= spec * spec;
        const float cc[3] = {col.x, col.y, col.z};
        for (int k = 0; k < 3; ++k)
            out[k] = to8(cc[k] * c.amb + diffuse * c.dif * c.lcol[k] + c.lcol[k] * spec * c.spec);
    }
    rgb[(size_t)pix * 3] = out[0];
    rgb[(size_t)pix * 3 + 1] = out[1];
    rgb[(size_t)pix * 3 + 2] = out[2];
}

}  // namespace

int render_project(const float4* pd, const float4* vm, const uint32_t* orig, uint32_t n, uint32_t prim_base,
                   const RenderCfg& c, float4* PR, float4* PC, float4* PP, cudaStream_t st) {
    if (n == 0) return 0;
    k_rp_project<<<nblk(n, 256), 256, 0, st>>>(pd, vm, orig, n, prim_base, c, PR, PC, PP);
    return 1;
}

uint32_t render_chunk_size() { return kChunk; }
uint32_t render_tile_size() { return kTile; }

int render_bin_count(const float4* PR, const float4* PC, const RenderCfg& c, uint32_t* counts, cudaStream_t st) {
    if (c.nprims == 0) return 0;
    k_rp_count<<<nblk(c.nprims, 256), 256, 0, st>>>(PR, PC, c, counts);
    return 1;
}

int render_bin_scatter(const float4* PR, const float4* PC, const RenderCfg& c, const uint32_t* start,
                       uint32_t* fill, uint32_t* list, cudaStream_t st) {
    if (c.nprims == 0) return 0;
    k_rp_scatter<<<nblk(c.nprims, 256), 256, 0, st>>>(PR, PC, c, start, fill, list);
    return 1;
}

int render_composite(const float4* PR, const float4* PC, const RenderCfg& c, const uint32_t* start, uint32_t* list,
                     uint8_t* rgb, cudaStream_t st) {
    const uint32_t nchunks = (c.nprims + kChunk - 1) / kChunk, tiles = c.tiles_x * c.tiles_y;
    int launches = 1;
    if (nchunks) {
        k_rp_sort<<<nblk(tiles * nchunks, kSortWarps * 32), kSortWarps * 32, 0, st>>>(start, tiles * nchunks, list);
        ++launches;
    }
    k_rp_composite<<<tiles * kPatches / kCompWarps, kCompWarps * 32, 0, st>>>(PR, PC, c, start, list, rgb);
    return launches;
}

int render_lit(const float4* PR, const float4* PC, const float4* PP, const RenderCfg& c, unsigned long long* zkey,
               uint8_t* rgb, cudaStream_t st) {
    int launches = 0;
    if (c.nprims) {
        if (c.S <= kDepthAlone)
            k_rp_depth<1><<<nblk(c.nprims, kDepthBlock), kDepthBlock, 0, st>>>(PR, PC, c, zkey);
        else
            k_rp_depth<kDepthLanes><<<nblk(c.nprims, kDepthBlock / kDepthLanes), kDepthBlock, 0, st>>>(PR, PC, c, zkey);
        ++launches;
    }
    k_rp_shade<<<nblk(c.W * c.H, 256), 256, 0, st>>>(PR, PC, PP, c, zkey, rgb);
    return launches + 1;
}

}  // namespace arp
