// fluid.cu -- fluid forces with the Runge-Kutta stage update fused at the tail.
//
// Replaces the reference's `fluid_forces` shader (src/soft_body/shaders/
// fluid.rs:95-251) and the lin_comb stage arithmetic that follows it
// (src/soft_body/particle_state/particles.rs:8-154).  The shader runs one
// 81-invocation workgroup per particle (27 cells x 3 strided lanes) with a
// shared-memory tree reduction; here one thread owns one particle sorted by
// search cell (the reference cell halved along x) and walks 3 (2D) or 9 (3D)
// contiguous x-rows of 5 half-width cells, so neighbor loads are coalesced
// across a warp (consecutive threads sit in the same or adjacent cells) and
// 5/6 of the candidates of the 3x3x3 reference cells are tested; the pair
// terms of the hits are then evaluated by four threads per particle (k_fluid).
// Scenes too small to fill the GPU that way give each particle 4 to 16
// threads throughout (k_fluid_group).
//
// Per pair the math is the shader's, term by term: continuity density rate,
// symmetric pressure force with the equation of state evaluated for both
// particles, contact potential (with the shader's argument order) and
// friction, physical viscosity and artificial viscosity.  Every term carries
// grad_w, which is zero for |r| >= h, so pairs outside the kernel radius are
// skipped before any of it is evaluated.
//
// Epilogue: k = (v, drho/dt, F/rho - g y) (+ the solid term for solid
// particles) is combined into the next stage state y0 + sum c_j k_j and the
// b-weighted accumulator with separately rounded products and sums, the same
// order the oracle uses.
#include <algorithm>

#include "group_scan.cuh"
#include "launch.cuh"
#include "warp.cuh"

namespace arp {

namespace {

__device__ __forceinline__ float pow7(float x) {
    const float x2 = x * x;
    const float x3 = x2 * x;
    const float x6 = x3 * x3;
    return x6 * x;
}

// fluid.rs:54-67 (called with radius and strength in the shader's order)
__device__ __forceinline__ float contact_potential(uint32_t eq, float r, float strength, float r0) {
    switch (eq) {
        case ARP_CONTACT_CONSTANT: return r <= r0 ? strength : 0.0f;
        case ARP_CONTACT_LINEAR: return strength * (r0 - r);
        case ARP_CONTACT_TAIT: return (strength * r / 7.0f) * (pow7(r0 / r) - 1.0f);
        case ARP_CONTACT_LENNARD_JONES: {
            float f = r0 / r;
            f *= f * f;
            f *= f;
            return strength * (f * f - 2.0f * f);
        }
        case ARP_CONTACT_HERTZ: return (strength * r0 / 7.0f) * (pow7(r / r0) - 1.0f);
        default: return 0.0f;
    }
}

// The particle a pair term is evaluated for.
struct Self {
    float3 x, v;
    float d1, m1, pterm1;
    uint32_t mat;       // material id in the scene
    const PairMat* pm;  // pair constants, indexed by the neighbor's material id in the scene (a shared-memory copy for
                        // the block's first scene, the global table otherwise)
};

// The scene scalars the pair terms read, held in registers.
struct PairK {
    float h2, kg, eps_hh;  // kg = -6 kconst
};

struct Acc {
    float den;
    float3 f, c;  // force without and with contact terms only
};

// What the pair terms read of a particle, one 32-byte sector and one load:
// (x, y, z, rho), (vx, vy, vz, p / rho^2).
struct PairRec {
    float4 x, v;
};
__device__ __forceinline__ PairRec load_rec(const float4* rec, uint32_t k) {
    PairRec r;
    load8(rec + 2 * (size_t)k, r.x, r.v);
    return r;
}
__device__ __forceinline__ PairRec load_hit(const float4* rec, uint32_t j) {  // j read from a list or a table
    PairRec r;
    load8_at(rec + 2 * (size_t)j, r.x, r.v);
    return r;
}

// What the terms of one neighbor pair share.  Every force term but the viscous
// one and friction points along r = x_j - x_i, and every term carries
// gws = |grad_w| / |r|, so the shader's sums of vectors
// (pf grad_w - q grad_w + cs grad_w) are coefficients on r.
struct PairGeom {
    float3 r, v;
    float r2, gws, vr;
};
template <int DIM>
__device__ __forceinline__ PairGeom pair_geom(const Self& s, const PairRec& j, const PairK& P) {
    PairGeom g;
    g.r = make_float3(__fsub_rn(j.x.x, s.x.x), __fsub_rn(j.x.y, s.x.y), DIM == 3 ? __fsub_rn(j.x.z, s.x.z) : 0.0f);
    const float rr = fmaf(g.r.y, g.r.y, __fmul_rn(g.r.x, g.r.x));
    g.r2 = DIM == 3 ? fmaf(g.r.z, g.r.z, rr) : rr;
    const float diff = fmaxf(__fsub_rn(P.h2, g.r2), 0.0f);
    g.gws = __fmul_rn(__fmul_rn(P.kg, diff), diff);
    g.v = make_float3(__fsub_rn(j.v.x, s.v.x), __fsub_rn(j.v.y, s.v.y), DIM == 3 ? __fsub_rn(j.v.z, s.v.z) : 0.0f);
    const float vv = fmaf(g.v.y, g.r.y, __fmul_rn(g.v.x, g.r.x));
    g.vr = DIM == 3 ? fmaf(g.v.z, g.r.z, vv) : vv;
    return g;
}

// The terms of one pair inside the kernel radius (the caller has tested it),
// contact aside: (density rate, force).  `ptj` is p_j / rho_j^2 of the
// neighbor, precomputed per particle; v.r is shared by the continuity and the
// artificial viscosity terms (v.grad_w = gws v.r).  Each operation is
// separately rounded or an explicit fma, so every kernel that evaluates a pair
// gets the same bits whatever the number of threads that share a particle.
template <int DIM>
__device__ __forceinline__ float4 pair_terms(const Self& s, const PairGeom& g, float d2, float ptj, bool boundary,
                                             const PairMat& m, const PairK& P) {
    const float mm = __fmul_rn(s.m1, m.mass);
    const float denom = __fadd_rn(g.r2, P.eps_hh);
    float p = __fadd_rn(s.pterm1, ptj);
    // GLSL division carries 2.5 ulp; the 2-ulp hardware quotient is used in the viscosity terms
    if (m.bulk != 0.0f)  // zero with a boundary particle
        p = __fsub_rn(p, __fdividef(__fmul_rn(m.bulk, g.vr), __fmul_rn(__fadd_rn(s.d1, d2), denom)));
    const float c = __fmul_rn(__fmul_rn(mm, p), g.gws);
    float4 t;
    t.x = __fmul_rn(boundary ? 0.0f : m.mass, __fmul_rn(g.gws, g.vr));
    t.y = __fmul_rn(c, g.r.x);
    t.z = __fmul_rn(c, g.r.y);
    t.w = DIM == 3 ? __fmul_rn(c, g.r.z) : 0.0f;
    if (m.visc != 0.0f) {  // zero for an elastic particle and with a boundary particle
        const float q = __fmul_rn(__fmul_rn(mm, m.visc), __fmul_rn(g.gws, g.r2));
        const float u = __fdividef(q, __fmul_rn(__fmul_rn(s.d1, d2), denom));
        t.y = fmaf(-u, g.v.x, t.y);
        t.z = fmaf(-u, g.v.y, t.z);
        if (DIM == 3) t.w = fmaf(-u, g.v.z, t.w);
    }
    return t;
}

// The contact potential and friction of one pair (fluid.rs:176-199).  Few
// pairs have one, and its registers would cost every pair a quarter of the
// resident warps (94 registers against 64), so contacts are evaluated in a
// second walk, over the hits that the first has marked, and have sums of their
// own.  A second walk over all hits wherever some had one took 65 us for 97,336
// particles with a contact in every pair (58 now, 47 without contacts) and 62 of
// 81 us a stage in a scene where a bar touches fluid (53 of 72 now); two marked
// hits' loads in flight spill.
template <int DIM>
__device__ __forceinline__ float3 contact_terms(const Self& s, const PairGeom& g, float d2, float mass2, uint32_t mat2,
                                                bool rubs, const DevInter& it) {
    float3 f = make_float3(0.0f, 0.0f, 0.0f);
    const float cp = contact_potential(it.potential, sqrtf(g.r2), it.radius, it.strength);
    if (cp == 0.0f) return f;
    const float cs = __fmul_rn(__fdiv_rn(__fmul_rn(mass2, cp), d2), g.gws);
    f = make_float3(__fmul_rn(cs, g.r.x), __fmul_rn(cs, g.r.y), __fmul_rn(cs, g.r.z));
    if (it.friction != 0.0f && rubs && s.mat != mat2) {
        // fluid.rs:192-199: friction along the normalised tangential velocity
        const float ix = g.r.x / g.r2, iy = g.r.y / g.r2, iz = g.r.z / g.r2;
        const float cr = __fmul_rn(cs, g.r2);  // contact force . r
        const float nx = ix * cr, ny = iy * cr, nz = iz * cr;
        float tx = g.v.x - ix * g.vr, ty = g.v.y - iy * g.vr, tz = g.v.z - iz * g.vr;
        const float tl = sqrtf(DIM == 3 ? (tx * tx + ty * ty) + tz * tz : tx * tx + ty * ty);
        tx /= tl; ty /= tl; tz /= tl;
        if (isfinite(tx) && isfinite(ty) && isfinite(tz)) {
            // normalize() applied a second time, as the shader does
            const float tl2 = sqrtf(DIM == 3 ? (tx * tx + ty * ty) + tz * tz : tx * tx + ty * ty);
            const float nl = sqrtf(DIM == 3 ? (nx * nx + ny * ny) + nz * nz : nx * nx + ny * ny);
            const float fr = it.friction * nl;
            f = make_float3(__fadd_rn(f.x, __fmul_rn(fr, tx / tl2)), __fadd_rn(f.y, __fmul_rn(fr, ty / tl2)),
                            DIM == 3 ? __fadd_rn(f.z, __fmul_rn(fr, tz / tl2)) : 0.0f);
        }
    }
    return f;
}

__device__ __forceinline__ void add_terms(Acc& acc, float4 t) {
    acc.den = __fadd_rn(acc.den, t.x);
    acc.f.x = __fadd_rn(acc.f.x, t.y);
    acc.f.y = __fadd_rn(acc.f.y, t.z);
    acc.f.z = __fadd_rn(acc.f.z, t.w);
}
__device__ __forceinline__ void add_contact(Acc& acc, float3 t) {
    acc.c.x = __fadd_rn(acc.c.x, t.x);
    acc.c.y = __fadd_rn(acc.c.y, t.y);
    acc.c.z = __fadd_rn(acc.c.z, t.z);
}

__device__ __forceinline__ float4 comb(float4 y0, float4 t, bool keep_w) {
    float4 r;
    r.x = __fadd_rn(y0.x, t.x);
    r.y = __fadd_rn(y0.y, t.y);
    r.z = __fadd_rn(y0.z, t.z);
    r.w = keep_w ? y0.w : __fadd_rn(y0.w, t.w);
    return r;
}
__device__ __forceinline__ float4 axpy(float c, float4 k, float4 t) {
    return make_float4(__fadd_rn(t.x, __fmul_rn(c, k.x)), __fadd_rn(t.y, __fmul_rn(c, k.y)),
                       __fadd_rn(t.z, __fmul_rn(c, k.z)), __fadd_rn(t.w, __fmul_rn(c, k.w)));
}

// The scan and the evaluation see one array of particles: the n mobile ones in
// cell order, then the boundary ones in theirs, so a neighbor is an index and
// a boundary particle one of at least n.

// Pair terms of neighbor j added to `acc` if j lies within the kernel radius
// (the scan's test lets a few others through); returns the pair's material bits
// then, kPairContact the highest, and 0 otherwise.  r^2 < h^2 is h^2 - r^2 > 0,
// grad_w's max(.., 0) test: without flush-to-zero a difference of finite floats is
// zero only when they are equal.
template <int DIM>
__device__ __forceinline__ uint32_t add_hit(Acc& acc, uint32_t j, const PairRec& rj, uint32_t mat2, const Self& s,
                                            const FluidArgs& a, const PairK& K) {
    const PairMat m = s.pm[mat2];
    const PairGeom g = pair_geom<DIM>(s, rj, K);
    const float4 t = pair_terms<DIM>(s, g, rj.x.w, rj.v.w, j >= a.n, m, K);
    const bool in = g.r2 < K.h2;
    if (in) add_terms(acc, t);
    return in ? m.bits : 0u;
}
// The contact terms of neighbor j, for which add_hit returned kPairContact.  `it`:
// the interactions of the particle's material.
template <int DIM>
__device__ __forceinline__ void add_hit_contact(Acc& acc, uint32_t j, const PairRec& rj, uint32_t mat2, const Self& s,
                                                const FluidArgs& a, const DevInter* it, const PairK& K) {
    const PairMat m = s.pm[mat2];
    const PairGeom g = pair_geom<DIM>(s, rj, K);
    const bool rubs = j >= a.n || (m.bits & (kPairElastic1 | kPairElastic2));
    add_contact(acc, contact_terms<DIM>(s, g, rj.x.w, m.mass, mat2, rubs, it[mat2]));
}

// Velocity Verlet, first half of a step (kick, then drift): v' = v + (dt/2) a,
// rho' = rho + (dt/2) drho/dt, x' = x + dt v', with (a, drho/dt) the derivative
// record of the state (its position part is not used).  Each sum is formed as
// y + (0 + c k), the order of the stage epilogue.
__device__ __forceinline__ float4 kick_drift(float4 p, float4 v, float4 fp, float4 fv, float half, float full,
                                             float4& vh) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    vh = comb(v, axpy(half, fv, z), true);  // w holds the material bits
    const float rho = __fadd_rn(p.w, __fadd_rn(0.0f, __fmul_rn(half, fp.w)));
    const float4 dx = axpy(full, make_float4(vh.x, vh.y, vh.z, 0.0f), z);
    return make_float4(__fadd_rn(p.x, dx.x), __fadd_rn(p.y, dx.y), __fadd_rn(p.z, dx.z), rho);
}

// The derivative record of one particle (fluid.rs:243-247, plus the solid
// term when active) and the Runge-Kutta stage epilogue: the store of k, the
// b-weighted accumulator and the next stage state of sorted particle k, in its
// storage slot.  With b.drift_pd the next velocity-Verlet step's kick and drift
// follow.  With b.bin.count the new state is counted into its search cell on the way (the first pass of the grid build that follows, which then
// need not read the positions again).
__device__ __forceinline__ void stage_epilogue(const FluidArgs& a, const Tables& T, const StageCoefs& c,
                                               const StageBuffers& b, uint32_t k, const Acc& acc) {
    const uint32_t slot = a.perm ? a.perm[k] : k;
    const uint32_t sid = a.sid[slot];
    const SceneP& P = T.scenes[T.mats[a.mat[k]].scene];
    const PairRec self = load_rec(a.rec, k);
    const float4 vi = self.v;
    const float d1 = self.x.w;
    const float g_acc = P.g;
    const bool solid_scene = P.solid_branch != 0u;
    float4 kpd = make_float4(vi.x, vi.y, vi.z, acc.den);
    float4 kvm = make_float4(__fdiv_rn(acc.f.x, d1), __fadd_rn(__fdiv_rn(acc.f.y, d1), -g_acc),
                             __fdiv_rn(acc.f.z, d1), 0.0f);
    if (a.solid_branch && sid != kInvalid && solid_scene) {
        const float4 ks = a.ksol[sid];
        kpd.x = __fadd_rn(kpd.x, vi.x);
        kpd.y = __fadd_rn(kpd.y, vi.y);
        kpd.z = __fadd_rn(kpd.z, vi.z);
        kvm.x = __fadd_rn(kvm.x, ks.x);
        kvm.y = __fadd_rn(kvm.y, ks.y);
        kvm.z = __fadd_rn(kvm.z, ks.z);
    }

    // Runge-Kutta stage epilogue
    if (b.store_pd) {
        b.store_pd[slot] = kpd;
        b.store_vm[slot] = kvm;
    }
    const float4 y0p = b.y0_pd[slot];
    const float4 y0v = b.y0_vm[slot];
    float4 accp = make_float4(0.f, 0.f, 0.f, 0.f), accv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c.c_acc != 0.0f) {
        if (!c.acc_first) {
            accp = b.acc_pd[slot];
            accv = b.acc_vm[slot];
        }
        accp = axpy(c.c_acc, kpd, accp);
        accv = axpy(c.c_acc, kvm, accv);
        if (!c.last) {
            b.acc_pd[slot] = accp;
            b.acc_vm[slot] = accv;
        }
    } else if (c.last) {
        accp = b.acc_pd[slot];
        accv = b.acc_vm[slot];
    }
    float4 np, nv;
    if (c.last) {
        np = comb(y0p, accp, false);
        if (c.kick) {  // a velocity-Verlet kick moves no particle: positions come from the drift
            np.x = y0p.x;
            np.y = y0p.y;
            np.z = y0p.z;
        }
        nv = comb(y0v, accv, true);
    } else {
        float4 tp = make_float4(0.f, 0.f, 0.f, 0.f), tv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c.c_prev0 != 0.0f) {
            tp = axpy(c.c_prev0, b.prev0_pd[slot], tp);
            tv = axpy(c.c_prev0, b.prev0_vm[slot], tv);
        }
        if (c.c_prev1 != 0.0f) {
            tp = axpy(c.c_prev1, b.prev1_pd[slot], tp);
            tv = axpy(c.c_prev1, b.prev1_vm[slot], tv);
        }
        if (c.c_prev2 != 0.0f) {
            tp = axpy(c.c_prev2, b.prev2_pd[slot], tp);
            tv = axpy(c.c_prev2, b.prev2_vm[slot], tv);
        }
        if (c.c_self != 0.0f) {
            tp = axpy(c.c_self, kpd, tp);
            tv = axpy(c.c_self, kvm, tv);
        }
        np = comb(y0p, tp, false);
        nv = comb(y0v, tv, true);
    }
    b.next_pd[slot] = np;
    b.next_vm[slot] = nv;
    if (b.drift_pd) {  // a force evaluation of its own leaves the state as it is
        const float4 vh = c.last ? nv : y0v;
        np = kick_drift(c.last ? np : y0p, vh, kpd, kvm, c.half, c.full, nv);
        b.drift_pd[slot] = np;
        b.drift_vm[slot] = nv;
    }
    if (b.bin.count) bin_particle(np, P, T.ncells, slot, b.bin);
}

// The particle's own fields for the pair terms; returns its scene.  `sm`: the
// pair constants of scene `scene0` (kInvalid: none).
__device__ __forceinline__ const SceneP& init_self(uint32_t k, const FluidArgs& a, const Tables& T, const PairMat* sm,
                                                   uint32_t scene0, Self& s) {
    const PairRec r = load_rec(a.rec, k);
    const uint32_t mat = a.mat[k];
    s.x = make_float3(r.x.x, r.x.y, r.x.z);
    s.v = make_float3(r.v.x, r.v.y, r.v.z);
    s.d1 = r.x.w;
    s.pterm1 = r.v.w;
    const DevMat& m = T.mats[mat];
    const SceneP& P = T.scenes[m.scene];
    s.mat = mat - P.mat_base;
    s.m1 = m.mass;
    s.pm = (m.scene == scene0 ? sm : T.pmats + P.inter_base) + s.mat * P.nmat;
    return P;
}

// How the terms of a particle's hits are added up, in every form: hit e of the
// candidate order goes to partial sum e mod 4, each partial sum adds its hits
// in order, and the total is (p0 + p1) + (p2 + p3); contact terms likewise in
// sums of their own, whose total is added last.  Results therefore depend
// neither on the launch shape nor on how lists are cut.
constexpr int kPartials = 4;
__device__ __forceinline__ float sum_partials(float v) {  // over the lanes that differ in their two lowest bits
    v = __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, 1));
    return __fadd_rn(v, __shfl_xor_sync(0xFFFFFFFFu, v, 2));
}

// ---- block form -----------------------------------------------------------------
// BLOCK consecutive cell-sorted particles per block, in two phases per warp.
//   * Scan, one thread per particle: the quantised candidates of its search
//     rows, four to a load, tested into a bit mask of 32; the set bits are
//     appended to its list of CAP entries in shared memory (an odd stride between
//     lists, so lanes at equal counts hit different banks).
//   * Evaluation, four threads per particle, eight particles of the warp at a
//     time: thread q takes hits q, q + 4, ...  Consecutive hits of a particle are
//     mostly consecutive slots of a search row, so the eight lanes that share
//     one L1 pass read two particles' runs instead of eight unrelated places.
// A lane whose list is full stops scanning; the warp then evaluates all lists
// (whole rounds of four, the rest moves to the list's front), keeps the partial
// sums in the tail of the lists of unfinished particles and scans on, so a
// particle may have any number of hits.
//
// Bound: L1 data wavefronts (71 % of peak) and issue slots (65 %), with L1 and
// L2 latency behind them (4.4 warps per issue on the long scoreboard); DRAM is
// idle.  What it replaced, one thread per particle over 16-byte candidates
// read from the positions, took 352 us per stage of the 1,048,576-particle
// fluid and bar scene (RK2, 222 M warp instructions, 69 M wavefronts) and two
// more launches for the particles whose lists overflowed; this takes 281 us
// (208 M, 58 M), the next state's cell keys included.  On the way: 4 threads per
// particle alone 372 us; + quantised candidates 345 us; + 32-byte records 330 us;
// + the next row's bounds and a second hit's record in flight 292 us; + contacts
// walked where they are 281.
// Only the epilogue reads what the solid kernels write, so behind those
// (a.published) a block waits there instead of at its start, and the pair
// sums fill the SMs that the solid kernels' last blocks leave: ten RK2 steps of
// the 1,048,576-particle scene 10,067 -> 9,992 us, 48 batched scenes 10,012 ->
// 9,873, 16,899 particles under velocity Verlet 560 -> 538.
// kBlocksPerSM 128-thread blocks per SM (72 registers): 8 (64 registers, spills)
// take 6 % more, 6 (80 registers) 2 % more.
constexpr int kBlocksPerSM = 7;
template <int DIM, int BLOCK, int CAP>
__global__ void __launch_bounds__(BLOCK, kBlocksPerSM * 128 / BLOCK) k_fluid(FluidArgs a, Tables T, StageCoefs c, StageBuffers b) {
    constexpr int STRIDE = CAP + 1;
    constexpr int TAIL = 7 * kPartials;  // words of saved partial sums
    static_assert(CAP % 2 == 0 && CAP >= TAIL + 8, "odd stride; room to go on beside the saved sums");
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* const lists = reinterpret_cast<uint32_t*>(smem_raw);
    PairMat* const sm = reinterpret_cast<PairMat*>(smem_raw + sizeof(uint32_t) * STRIDE * BLOCK);
    step_begin_unless(a.published, kBlocksPerSM * 128 / BLOCK);
    const uint32_t k0 = blockIdx.x * BLOCK;
    const uint32_t scene0 = T.mats[a.mat[k0]].scene;  // k0 < n: one block per started tile
    {
        const SceneP& S0 = T.scenes[scene0];
        for (uint32_t i = threadIdx.x; i < S0.nmat * S0.nmat; i += BLOCK) sm[i] = T.pmats[S0.inter_base + i];
    }
    __syncthreads();
    const uint32_t k = k0 + threadIdx.x;
    const bool valid = k < a.n;
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u;
    const uint32_t my = threadIdx.x * STRIDE;            // first entry of the list
    const uint32_t wlist = (threadIdx.x & ~31u) * STRIDE;  // of the warp's first list
    uint32_t w = my;                // next free entry
    uint32_t wend = my + CAP;       // where the list is full
    uint32_t row = 0;               // next row to open
    uint32_t jn = 0, hi = 0;        // what is left of the current range
    uint32_t j2 = 0, hi2 = 0;       // the range after it in the same row (boundary, then mobile candidates)
    uint32_t pend = 0, pbase = 0;   // hits not yet listed: bit 31 - i for candidate pbase + i
    bool done = !valid;             // no candidates left
    bool open = valid;              // the sums are not complete
    bool saved = false;             // partial sums lie in the list's tail
    Acc acc;
    acc.den = 0.0f;
    acc.f = make_float3(0.f, 0.f, 0.f);

    for (;;) {
        // scan until the candidates end or the list is full (what the scan
        // needs of the particle is read again after an interruption, so that it
        // need not stay in registers during the evaluation)
        if (!done) {
            const float4 xi = a.rec[2 * (size_t)k];
            const SceneP& P = T.scenes[T.mats[a.mat[k]].scene];
            const SearchRows rows = search_rows<DIM>(xi, finite3(xi), P);
            const uint32_t own = own_code<DIM>(xi, P);
            const uint4* const code4 = reinterpret_cast<const uint4*>(a.code);
            // the bounds of the next row are read while the current one is tested
            uint32_t nb0 = 0, nb1 = 0, nm0 = 0, nm1 = 0;
            auto fetch = [&]() {
                const uint32_t c0 = row < (uint32_t)rows.nrows ? search_row(rows, (int)row, P) : kInvalid;
                nb0 = nb1 = nm0 = nm1 = 0;
                if (c0 != kInvalid) {
                    nb0 = a.bstart[c0];
                    nb1 = a.bstart[c0 + rows.width];
                    nm0 = a.start[c0];
                    nm1 = a.start[c0 + rows.width];
                }
            };
            fetch();
#pragma unroll 1
            for (;;) {
                while (pend && w < wend) {
                    const uint32_t i = (uint32_t)__clz((int)pend);
                    pend ^= 0x80000000u >> i;
                    lists[w++] = pbase + i;
                }
                if (pend) break;
                if (jn >= hi) {
                    if (j2 < hi2) {
                        jn = j2;
                        hi = j2 = hi2;
                    } else {
                        if (row >= (uint32_t)rows.nrows) {
                            done = true;
                            break;
                        }
                        if (nb0 < nb1) {
                            jn = a.n + nb0;
                            hi = a.n + nb1;
                            j2 = nm0;
                            hi2 = nm1;
                        } else {
                            jn = nm0;
                            hi = nm1;
                        }
                        ++row;
                        fetch();
                        if (jn >= hi) continue;
                    }
                }
                // up to 32 candidates from the group of four that holds jn on
                pbase = jn & ~3u;
                const uint32_t g1 = (hi - pbase + 3u) >> 2;
                const uint4* const p = code4 + (pbase >> 2);
                uint32_t m = 0;
                auto test4 = [&](uint4 v) {
                    m = __funnelshift_l((uint32_t)code_test(v.x, own), m, 1);
                    m = __funnelshift_l((uint32_t)code_test(v.y, own), m, 1);
                    m = __funnelshift_l((uint32_t)code_test(v.z, own), m, 1);
                    m = __funnelshift_l((uint32_t)code_test(v.w, own), m, 1);
                };
                {
                    const uint4 v0 = p[0], v1 = p[1], v2 = p[2], v3 = p[3];  // the array is padded
                    test4(v0);
                    test4(v1);
                    test4(v2);
                    test4(v3);
                }
                if (g1 > 4u) {
                    const uint4 v0 = p[4], v1 = p[5];
                    uint4 v2 = make_uint4(0u, 0u, 0u, 0u), v3 = v2;
                    if (g1 > 6u) {
                        v2 = p[6];
                        v3 = p[7];
                    }
                    test4(v0);
                    test4(v1);
                    if (g1 > 6u) {
                        test4(v2);
                        test4(v3);
                    } else {
                        m <<= 8;
                    }
                } else {
                    m <<= 16;
                }
                const uint32_t end = min(hi - pbase, 32u);
                pend = m & (FULL >> (jn - pbase)) & (FULL << (32u - end));
                jn = pbase + 32u;
            }
        }
        __syncwarp();
        // evaluate: all of a finished list, whole rounds of four of another
        const uint32_t cnt = w - my;
        const uint32_t ev = !open ? 0u : done ? cnt : cnt & ~(uint32_t)(kPartials - 1);
        const bool fin = open && done;
        const uint32_t word = cnt << 16 | ev << 2 | (fin ? 2u : 0u) | (saved ? 1u : 0u);
#pragma unroll 1
        for (uint32_t pass = 0; pass < 4u; ++pass) {
            const uint32_t owner = pass * 8u + (lane >> 2);
            const uint32_t ow = __shfl_sync(FULL, word, owner);
            const uint32_t n_ev = ow >> 2 & 0x3FFFu;
            const uint32_t list = wlist + owner * STRIDE;
            Acc part;
            part.den = 0.0f;
            part.f = part.c = make_float3(0.f, 0.f, 0.f);
            if (ow & 1u) {
                const uint32_t t = list + CAP - TAIL + 7u * q;
                part.den = __uint_as_float(lists[t]);
                part.f = make_float3(__uint_as_float(lists[t + 1]), __uint_as_float(lists[t + 2]),
                                     __uint_as_float(lists[t + 3]));
                part.c = make_float3(__uint_as_float(lists[t + 4]), __uint_as_float(lists[t + 5]),
                                     __uint_as_float(lists[t + 6]));
            }
            if (n_ev > q) {
                const uint32_t ko = k - lane + owner;
                Self s;
                const SceneP& P = init_self(ko, a, T, sm, scene0, s);
                const PairK K{P.h2, -6.0f * P.kconst, P.eps_hh};
                uint32_t rubbing = 0;  // a bit for each of the thread's hits: the pair has a contact potential
                static_assert(CAP / kPartials <= 32, "32 bits");
#pragma unroll 1
                for (uint32_t e = q; e < n_ev; e += 2 * kPartials) {  // two hits' loads in flight
                    const bool two = e + kPartials < n_ev;
                    const uint32_t j0 = lists[list + e], j1 = two ? lists[list + e + kPartials] : ko;
                    const PairRec r0 = load_hit(a.rec, j0), r1 = load_hit(a.rec, j1);
                    const uint32_t m0 = a.mat8[j0], m1 = a.mat8[j1];
                    const uint32_t c0 = j0 != ko ? add_hit<DIM>(part, j0, r0, m0, s, a, K) : 0u;
                    rubbing = __funnelshift_l(c0, rubbing, 1);
                    const uint32_t c1 = j1 != ko ? add_hit<DIM>(part, j1, r1, m1, s, a, K) : 0u;
                    rubbing = __funnelshift_l(c1, rubbing, 1);
                }
                if (rubbing) {
                    const DevInter* const it = T.inter + P.inter_base + s.mat * P.nmat;
                    rubbing <<= 32u - 2u * ((n_ev - q + 2 * kPartials - 1) / (2 * kPartials));  // bit 31 - i: hit q + 4 i
#pragma unroll 1
                    do {
                        const uint32_t i = (uint32_t)__clz((int)rubbing);
                        rubbing ^= 0x80000000u >> i;
                        const uint32_t j = lists[list + q + kPartials * i];
                        add_hit_contact<DIM>(part, j, load_hit(a.rec, j), a.mat8[j], s, a, it, K);
                    } while (rubbing);
                }
            }
            __syncwarp();
            const bool unfinished = !(ow & 2u) && n_ev;
            if (__any_sync(FULL, unfinished)) {
                // the rest of the list (fewer than four entries) to its front, the sums to its tail
                const uint32_t rest = (ow >> 16) - n_ev;
                const uint32_t keep = unfinished && q < rest ? lists[list + n_ev + q] : 0u;
                __syncwarp();
                if (unfinished) {
                    if (q < rest) lists[list + q] = keep;
                    const uint32_t t = list + CAP - TAIL + 7u * q;
                    lists[t] = __float_as_uint(part.den);
                    lists[t + 1] = __float_as_uint(part.f.x);
                    lists[t + 2] = __float_as_uint(part.f.y);
                    lists[t + 3] = __float_as_uint(part.f.z);
                    lists[t + 4] = __float_as_uint(part.c.x);
                    lists[t + 5] = __float_as_uint(part.c.y);
                    lists[t + 6] = __float_as_uint(part.c.z);
                }
            }
            const float s0 = sum_partials(part.den);
            float s1 = sum_partials(part.f.x), s2 = sum_partials(part.f.y), s3 = sum_partials(part.f.z);
            if (__any_sync(FULL, part.c.x != 0.0f || part.c.y != 0.0f || part.c.z != 0.0f)) {
                s1 = __fadd_rn(s1, sum_partials(part.c.x));
                s2 = __fadd_rn(s2, sum_partials(part.c.y));
                s3 = __fadd_rn(s3, sum_partials(part.c.z));
            }
            const uint32_t src = (lane & 7u) * 4u;
            const float r0 = __shfl_sync(FULL, s0, src), r1 = __shfl_sync(FULL, s1, src),
                        r2 = __shfl_sync(FULL, s2, src), r3 = __shfl_sync(FULL, s3, src);
            if (fin && lane >> 3 == pass) {
                acc.den = r0;
                acc.f = make_float3(r1, r2, r3);
            }
        }
        if (fin) open = false;
        if (!__any_sync(FULL, open)) break;
        __syncwarp();
        saved = saved || ev > 0u;
        w = my + (open ? cnt - ev : 0u);
        wend = my + CAP - TAIL;
    }
    step_begin();
    if (valid) stage_epilogue(a, T, c, b, k, acc);
}

// ---- group form --------------------------------------------------------------
// LANES threads of a warp share one particle throughout.  In the block form a
// launch takes at least as long as one thread's walk over ~170 candidates,
// however few particles there are; here the walk is LANES times shorter and
// there are LANES times as many warps, which pays until the SMs are full: the
// 16,899-particle 3D scene 22 us per launch with 8 lanes against 58 in the block
// form, the 126,464-particle one 62 us in the block form against 86 with 4 lanes.
// Bound: the latency of the chain of dependent loads of one particle, and whether
// all blocks are resident at once: 8 blocks per SM with 16 lanes (16.5 us for 9,072
// particles, 18.9 with 7), 7 with 4 and 8 (35.5 us for 32,256, 37 with 8, 42 with 6).
//   * Candidates are scanned and hits listed by the lanes together (GroupScan).
//   * Each lane evaluates one hit at a time; with more than four lanes the terms
//     go through shared memory to the lanes that hold the partial sums (partial
//     sum lane mod 4, 16 / LANES components each).
constexpr int kGroupBlock = 128;

template <int DIM, int LANES>
__global__ void __launch_bounds__(kGroupBlock, LANES == 16 ? 8 : 7) k_fluid_group(FluidArgs a, Tables T, StageCoefs c, StageBuffers b) {
    constexpr int NG = kGroupBlock / LANES;       // particles per block
    constexpr int CPL = 16 / LANES;               // components of the partial sum a lane holds
    static_assert(LANES == 4 || LANES == 8 || LANES == 16, "four partial sums of four components over the lanes");
    __shared__ uint32_t s_list[NG][kGroupList];
    __shared__ uint2 s_seg[NG][2 * GroupScan<DIM, LANES>::MAXROWS];
    __shared__ float4 s_term[LANES > 4 ? NG : 1][LANES];
    constexpr unsigned FULL = 0xFFFFFFFFu;
    step_begin_unless(a.published, LANES == 16 ? 8 : 7);
    const uint32_t lane = threadIdx.x % LANES, gi = threadIdx.x / LANES;
    const uint32_t kk = blockIdx.x * NG + gi;
    const bool valid = kk < a.n;
    const uint32_t k = valid ? kk : a.n - 1u;  // idle groups of the last block follow the last particle, without candidates
    Self s;
    const SceneP& P = init_self(k, a, T, nullptr, kInvalid, s);
    const float4 xi = make_float4(s.x.x, s.x.y, s.x.z, 0.0f);
    const PairK K{P.h2, -6.0f * P.kconst, P.eps_hh};
    uint32_t* const list = s_list[gi];

    // components (lane / 4) * CPL + i of partial sum lane mod 4: (density rate,
    // force) and (unused, contact force)
    float acc[CPL], con[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) acc[i] = con[i] = 0.0f;
    // adds one hit's terms per lane (zero where a lane has none: +0 leaves a
    // sum that began at +0 as it is)
    auto add = [&](float* to, float4 t) {
        if (LANES == 4) {
            to[0] = __fadd_rn(to[0], t.x);
            to[1 % CPL] = __fadd_rn(to[1 % CPL], t.y);
            to[2 % CPL] = __fadd_rn(to[2 % CPL], t.z);
            to[3 % CPL] = __fadd_rn(to[3 % CPL], t.w);
        } else {
            float4* const term = s_term[LANES > 4 ? gi : 0];
            term[lane] = t;
            __syncwarp();
            const float* f = reinterpret_cast<const float*>(term) + (lane >> 2) * CPL;
#pragma unroll
            for (int e = 0; e < LANES; e += kPartials)
#pragma unroll
                for (int i = 0; i < CPL; ++i) to[i] = __fadd_rn(to[i], f[4 * (e + (lane & 3u)) + i]);
            __syncwarp();
        }
    };
    bool any_con = false;
    GroupScan<DIM, LANES>::run(xi, valid && finite3(xi), P, ScanArrays{a.code, a.start, a.bstart, a.n}, list, s_seg[gi],
                               [&](uint32_t ev) {
        uint32_t rubbing = 0, e0 = 0;  // a bit for each of the lane's hits: the pair has a contact potential
        static_assert(kGroupList / LANES <= 32, "32 bits");
#pragma unroll 1
        for (; __any_sync(FULL, e0 < ev); e0 += LANES) {
            Acc t;
            uint32_t c = 0u;
            t.den = 0.0f;
            t.f = make_float3(0.f, 0.f, 0.f);
            if (e0 + lane < ev) {
                const uint32_t j = list[e0 + lane];
                if (j != k) c = add_hit<DIM>(t, j, load_hit(a.rec, j), a.mat8[j], s, a, K);
            }
            rubbing = __funnelshift_l(c, rubbing, 1);
            add(acc, make_float4(t.den, t.f.x, t.f.y, t.f.z));
        }
        if (__any_sync(FULL, rubbing != 0u)) {
            any_con = true;
            const DevInter* const it = T.inter + P.inter_base + s.mat * P.nmat;
            rubbing <<= 32u - e0 / LANES;
#pragma unroll 1
            for (uint32_t e = lane; __any_sync(FULL, rubbing != 0u); e += LANES, rubbing <<= 1) {
                const bool mine = (rubbing & kPairContact) != 0u;  // the highest
                if (!__any_sync(FULL, mine)) continue;
                Acc t;
                t.c = make_float3(0.f, 0.f, 0.f);
                if (mine) {
                    const uint32_t j = list[e];
                    add_hit_contact<DIM>(t, j, load_hit(a.rec, j), a.mat8[j], s, a, it, K);
                }
                add(con, make_float4(0.f, t.c.x, t.c.y, t.c.z));
            }
        }
    });
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        acc[i] = sum_partials(acc[i]);
        if (any_con) acc[i] = __fadd_rn(acc[i], sum_partials(con[i]));
    }
    Acc sum;
    sum.den = __shfl_sync(FULL, acc[0], 0, LANES);
    sum.f.x = __shfl_sync(FULL, acc[1 % CPL], 4 * (1 / CPL), LANES);
    sum.f.y = __shfl_sync(FULL, acc[2 % CPL], 4 * (2 / CPL), LANES);
    sum.f.z = __shfl_sync(FULL, acc[3 % CPL], 4 * (3 / CPL), LANES);
    step_begin();
    if (valid && lane == 0) stage_epilogue(a, T, c, b, k, sum);
}

// The kick and drift of a state that no step has written, in storage order; the
// drifted state is counted into its search cells on the way.  A step that ends
// with a force evaluation forms the next one's in its epilogue: as a launch of
// its own it cost 4 of 47 us per step of 16,899 particles.
__global__ void k_verlet_kick_drift(const float4* pd, const float4* vm,
                                    const float4* fpd, const float4* fvm, uint32_t n,
                                    float half, float full, float4* out_pd, float4* out_vm,
                                    Tables T, CellBins bin) {
    step_begin();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 v = vm[k];
    float4 vh;
    const float4 np = kick_drift(pd[k], v, fpd[k], fvm[k], half, full, vh);
    out_pd[k] = np;
    out_vm[k] = vh;
    bin_particle(np, T.scenes[T.mats[__float_as_uint(v.w)].scene], T.ncells, k, bin);
}

// The kick of the plastic strain (4 float4 per solid): e' = e + (0 + c k).
__global__ void k_verlet_kick4(const float4* e, const float4* k4, uint32_t count, float half,
                               float4* out) {
    step_begin();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    out[i] = comb(e[i], axpy(half, k4[i], make_float4(0.f, 0.f, 0.f, 0.f)), false);
}

}  // namespace

int verlet_kick_drift(const float4* pd, const float4* vm, const float4* fpd, const float4* fvm, uint32_t n, float half,
                      float full, float4* out_pd, float4* out_vm, const Tables& T, const CellBins& bin,
                      cudaStream_t st) {
    if (n == 0) return 0;
    launch_step(k_verlet_kick_drift, (n + 255) / 256, 256, 0, st, pd, vm, fpd, fvm, n, half, full, out_pd, out_vm, T, bin);
    return 1;
}

int verlet_kick4(const float4* e, const float4* k4, uint32_t count, float half, float4* out, cudaStream_t st) {
    if (count == 0) return 0;
    launch_step(k_verlet_kick4, (count + 255) / 256, 256, 0, st, e, k4, count, half, out);
    return 1;
}

const FluidVariant kFluidVariants[kNumFluidVariants] = {
    {128, 40, 0}, {128, 44, 0}, {128, 48, 0}, {128, 56, 0}, {128, 64, 0}, {128, 96, 0},
    {256, 40, 0}, {256, 44, 0}, {256, 48, 0}, {256, 56, 0}, {256, 64, 0}, {256, 96, 0},
    {128, 96, 4}, {128, 96, 8}, {128, 96, 16},
};

int launch_fluid(const FluidArgs& a, const Tables& T, int kdim, const StageCoefs& c, const StageBuffers& b,
                 int variant, cudaStream_t st) {
    if (a.n == 0) return 0;
    const FluidVariant v = kFluidVariants[variant < 0 || variant >= kNumFluidVariants ? 0 : variant];
    if (v.lanes) {
        const uint32_t nb = (a.n + (uint32_t)(kGroupBlock / v.lanes) - 1u) / (uint32_t)(kGroupBlock / v.lanes);
#define ARP_GROUP(D, L) \
    if (kdim == D && v.lanes == L) launch_step(k_fluid_group<D, L>, nb, kGroupBlock, 0, st, a, T, c, b);
        ARP_GROUP(3, 4) ARP_GROUP(3, 8) ARP_GROUP(3, 16)
        ARP_GROUP(2, 4) ARP_GROUP(2, 8) ARP_GROUP(2, 16)
#undef ARP_GROUP
        return 1;
    }
    const size_t smem = sizeof(uint32_t) * (v.cap + 1) * v.block + sizeof(PairMat) * T.max_nmat * T.max_nmat;
    const uint32_t nb = (a.n + (uint32_t)v.block - 1u) / (uint32_t)v.block;
#define ARP_FLUID(D, B, C)                                                                                         \
    if (kdim == D && v.block == B && v.cap == C) {                                                                 \
        if (smem > 48 * 1024)                                                                                      \
            cudaFuncSetAttribute(k_fluid<D, B, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);        \
        launch_step(k_fluid<D, B, C>, nb, B, smem, st, a, T, c, b);                                                \
    }
#define ARP_FLUID_CAPS(D, B) \
    ARP_FLUID(D, B, 40) ARP_FLUID(D, B, 44) ARP_FLUID(D, B, 48) ARP_FLUID(D, B, 56) \
    ARP_FLUID(D, B, 64) ARP_FLUID(D, B, 96)
    ARP_FLUID_CAPS(3, 128) ARP_FLUID_CAPS(3, 256) ARP_FLUID_CAPS(2, 128) ARP_FLUID_CAPS(2, 256)
#undef ARP_FLUID_CAPS
#undef ARP_FLUID
    return 1;
}

}  // namespace arp
