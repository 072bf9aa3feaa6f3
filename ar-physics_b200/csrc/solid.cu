// solid.cu -- Total-Lagrangian solid kernels.
//
// Replaces compute_strain (src/soft_body/shaders/strain.rs:71-183),
// solid_forces (src/soft_body/shaders/solid.rs:276-524) and clear_solids
// (solid.rs:5-37).
//
// The reference rebuilds the reference-configuration buckets, the correction
// matrix L = (sum V_j gradW(dX) (x) dX)^-1 and each neighbor's stress for
// every pair of every stage.  Reference positions never change (their time
// derivative is zero), so here:
//   * once per particle set: a CSR list of reference neighbors within h
//     (solid ids, same-material flag, gradW(X_j - X_i), V_j = m_j / rho0_j)
//     and L (k_ref_count / k_ref_fill / k_ref_L);
//   * per stage, 2 or 4 threads per solid: F, Fdot from the list, Seth-Hill
//     strain + Hooke stress (all strain orders, GLSL mat4 semantics),
//     A = sigma L, the Johnson-Cook plastic rate and its stage update
//     (k_solid_stress);
//   * per stage, 2 or 4 threads per solid: elastic force -V_i V_j (A_i + A_j)
//     gradW over the list, then hourglass control and self-contact over the
//     current 3x3x3 cells (k_solid_forces).  A_j is read, not recomputed.
#include "grid.cuh"
#include "launch.cuh"
#include "mat4.cuh"
#include "solid_rec.cuh"

namespace arp {

namespace {

constexpr int kThreads = 128;
// Both stage kernels add up entry e of a solid's reference list in partial sum
// e mod 4 and combine them as (p0 + p2) + (p1 + p3), whatever the number of
// threads per solid: 4 hold one partial sum each, 2 hold two.  Four threads
// halve the chain of dependent loads of one solid, which is what a scene with
// few solids waits for; two repeat less of the work per solid.  Stress and force
// kernels per stage (events on both sides), 4 / 2 threads: 1,274 solids 17.4 / 19.7
// us, 9,072 19.4 / 21.5, 15,872 21.6 / 23.5, 32,256 31.8 / 29.6, 129,024 93.5 / 77.5.
constexpr uint32_t kFewSolids = 24576;
constexpr uint32_t kSameMat = 0x80000000u;
// The stage kernels recompute gradW(dX) and W(dX) of each reference pair from
// the reference positions (a gather that neighboring solids share in L1/L2)
// instead of streaming per-entry values from HBM: a list entry costs its
// 4-byte index.  The stored gradW and volume (rl.gw) serve L and the reverse
// pass.

inline uint32_t blocks_for(uint32_t n, int t) { return (n + (uint32_t)t - 1u) / (uint32_t)t; }

__device__ __forceinline__ float3 sub3(float4 a, float4 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }

// unit diagonal on the axes at or above dim (solid.rs:149, :175, :227)
__device__ __forceinline__ void pad_unit(M4& C, uint32_t dim) {
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
        if (i >= dim) C.m[i][i] = 1.0f;
}

// Walk the 27 reference cells around solid i (search-cell rows ascending,
// ascending solid id inside a search cell) and call f(j, dX, diff) for each
// other solid with h^2 - |dX|^2 > 0.
template <class F>
__device__ __forceinline__ void for_ref_neighbors(uint32_t i, const float4* __restrict__ ref,
                                                  const uint32_t* __restrict__ start, const uint32_t* __restrict__ perm,
                                                  const SceneP& P, F&& f) {
    const float4 xi = ref[i];
    if (!finite3(xi)) return;
    for_reference_block_rows(xi, P, [&](uint32_t c0, uint32_t c1) {
        for (uint32_t k = start[c0]; k < start[c1]; ++k) {
            const uint32_t j = perm[k];
            if (j == i) continue;
            const float3 dX = sub3(ref[j], xi);
            const float diff = P.h2 - dot3(dX, dX);
            if (diff > 0.0f) f(j, dX, diff);
        }
    });
}

__global__ void k_ref_count(const float4* __restrict__ ref, const uint32_t* __restrict__ mat_of, uint32_t ns,
                            const uint32_t* __restrict__ start, const uint32_t* __restrict__ perm, Tables T,
                            uint32_t* __restrict__ count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    uint32_t n = 0;
    const SceneP& P = T.scenes[T.mats[mat_of[i]].scene];
    for_ref_neighbors(i, ref, start, perm, P, [&](uint32_t, float3, float) { ++n; });
    count[i] = n;
}

__global__ void k_ref_fill(const float4* __restrict__ ref, const uint32_t* __restrict__ mat_of, uint32_t ns,
                           const uint32_t* __restrict__ start, const uint32_t* __restrict__ perm, Tables T,
                           const uint32_t* __restrict__ off, uint32_t* __restrict__ nbr, float4* __restrict__ gw) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    uint32_t w = off[i];
    const uint32_t mi = mat_of[i];
    const DevMat* mats = T.mats;
    const SceneP& P = T.scenes[mats[mi].scene];
    for_ref_neighbors(i, ref, start, perm, P, [&](uint32_t j, float3 dX, float diff) {
        const float s = -6.0f * P.kconst * diff * diff;
        const uint32_t mj = mat_of[j];
        nbr[w] = j | (mj == mi ? kSameMat : 0u);
        gw[w] = make_float4(s * dX.x, s * dX.y, s * dX.z, mats[mj].vol0);
        ++w;
    });
}

// L = inverse(sum_j V_j gradW (x) dX), unit diagonal on the unused axes
// (strain.rs:107-136).  Stored as three float4 columns.
__global__ void k_ref_L(const float4* __restrict__ ref, const uint32_t* __restrict__ mat_of, uint32_t ns,
                        const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr,
                        const float4* __restrict__ gw, Tables T, float4* __restrict__ L) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    const SceneP& P = T.scenes[T.mats[mat_of[i]].scene];
    M4 C = m4_zero();
    const float4 xi = ref[i];
    for (uint32_t k = off[i]; k < off[i + 1]; ++k) {
        const uint32_t j = nbr[k] & ~kSameMat;
        const float4 g = gw[k];
        const float3 dX = sub3(ref[j], xi);
        const float d[3] = {dX.x, dX.y, dX.z};
        const float gg[3] = {g.x, g.y, g.z};
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) C.m[c][r] += g.w * (gg[r] * d[c]);
    }
    pad_unit(C, P.dim);
    const M4 Li = m4_inverse(C);
#pragma unroll
    for (int c = 0; c < 3; ++c) L[3 * i + c] = make_float4(Li.m[c][0], Li.m[c][1], Li.m[c][2], Li.m[c][3]);
}

// ---- per-stage strain / stress ----------------------------------------------

__device__ __forceinline__ float trace_dim(const M4& A, uint32_t dim) {
    float t = A.m[0][0];
#pragma unroll
    for (uint32_t i = 1; i < 4; ++i)
        if (i < dim) t += A.m[i][i];
    return t;
}
__device__ inline M4 mat_log5(const M4& A) {  // solid.rs:105-116
    M4 sum = m4_zero();
    M4 term = m4_scale(-1.0f, m4_ident());
    const M4 X = m4_scale(-1.0f, m4_sub(A, m4_ident()));
    for (int i = 1; i <= 5; ++i) {
        term = m4_mul(term, X);
        sum = m4_add(sum, m4_div(term, (float)i));
    }
    return sum;
}
__device__ inline M4 mat_sqrt_db(const M4& Xm) {  // Denman-Beavers, solid.rs:119-133
    M4 Y = Xm, Z = m4_ident();
    for (int i = 0; i < 15; ++i) {
        const M4 Yn = m4_scale(0.5f, m4_add(Y, m4_inverse(Z)));
        const M4 Zn = m4_scale(0.5f, m4_add(Z, m4_inverse(Y)));
        Y = Yn;
        Z = Zn;
    }
    return Y;
}
template <bool ORDER2>
__device__ inline M4 seth_hill(const M4& F, int two_m, uint32_t dim) {  // solid.rs:147-168
    M4 C = m4_mul(m4_transpose(F), F);
    pad_unit(C, dim);
    if (ORDER2) return m4_scale(1.0f / 2.0f, m4_sub(m4_mul(m4_ident(), C), m4_ident()));
    if (two_m == 0) return m4_scale(0.5f, mat_log5(C));
    const int a = two_m < 0 ? -two_m : two_m;
    const int m = a >> 1;
    M4 Cm = m4_ident();
    for (int i = 0; i < m; ++i) Cm = m4_mul(Cm, C);
    if (a & 1) Cm = m4_mul(Cm, mat_sqrt_db(C));
    if (two_m < 0) Cm = m4_inverse(Cm);
    return m4_scale(1.0f / (float)two_m, m4_sub(Cm, m4_ident()));
}
template <bool ORDER2>
__device__ inline M4 seth_hill_rate(const M4& F, const M4& Fd, int two_m, uint32_t dim) {  // solid.rs:170-204
    M4 dC = m4_mul(m4_transpose(Fd), F);
    dC = m4_add(dC, m4_transpose(dC));
    if (ORDER2) return m4_scale(1.0f / 2.0f, m4_mul(m4_ident(), dC));
    M4 C = m4_mul(m4_transpose(F), F);
    pad_unit(C, dim);
    if (two_m == 0) return m4_mul(m4_scale(0.5f, dC), m4_inverse(C));
    const int a = two_m < 0 ? -two_m : two_m;
    const int m = a >> 1;
    M4 rate = m4_zero();
    for (int i = 0; i < m; ++i) {
        M4 term = m4_ident();
        for (int j = 0; j < m; ++j) term = m4_mul(term, j == i ? dC : C);
        rate = m4_add(rate, term);
    }
    rate = m4_scale(1.0f / (float)two_m, rate);
    if (two_m < 0) {
        const M4 iC = m4_inverse(C);
        return m4_mul(m4_mul(m4_scale(-1.0f, iC), rate), iC);
    }
    return rate;
}
__device__ __forceinline__ M4 hooke(const M4& E, float normal, float shear, uint32_t dim) {
    const M4 a = m4_scale(normal * trace_dim(E, dim), m4_ident());
    return m4_add(a, m4_scale(2.0f * shear, E));
}

__device__ __forceinline__ float4 lin4(float c, float4 k, float4 t) {
    return make_float4(__fadd_rn(t.x, __fmul_rn(c, k.x)), __fadd_rn(t.y, __fmul_rn(c, k.y)),
                       __fadd_rn(t.z, __fmul_rn(c, k.z)), __fadd_rn(t.w, __fmul_rn(c, k.w)));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}

// The four partial sums of a solid, LANES threads holding 4 / LANES each:
// (p0 + p2) + (p1 + p3) on every lane.
template <int LANES>
__device__ __forceinline__ float sum4(const float* p) {
    static_assert(LANES == 4 || LANES == 2, "four partial sums");
    if (LANES == 4) return group_sum<4>(p[0]);  // lanes 0..3 hold p0..p3
    return group_sum<2>(__fadd_rn(p[0], p[4 / LANES - 1]));  // lanes 0, 1 hold p0, p2 and p1, p3
}

// 3 x 3 stress chain of strain order 2 without plastic flow: the 4 x 4 forms
// below with their zeros and the padded fourth axis left out.  [column][row].
struct T3 {
    float m[3][3];
};
__device__ __forceinline__ T3 t3_mul(const T3& a, const T3& b) {  // a b
    T3 r;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) r.m[c][k] = (a.m[0][k] * b.m[c][0] + a.m[1][k] * b.m[c][1]) + a.m[2][k] * b.m[c][2];
    return r;
}
__device__ __forceinline__ T3 t3_transpose(const T3& a) {
    T3 r;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) r.m[c][k] = a.m[k][c];
    return r;
}
__device__ __forceinline__ T3 stress_order2(const T3& F, const T3& Fd, float lam, float mu, float lam_d, float mu_d,
                                            uint32_t dim) {
    T3 E = t3_mul(t3_transpose(F), F);
    T3 R = t3_mul(t3_transpose(Fd), F);
    float tr = 0.0f, trd = 0.0f;
    T3 S;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const bool unused = (uint32_t)c >= dim;
            E.m[c][k] = c == k ? (unused ? 0.0f : 0.5f * (E.m[c][k] - 1.0f)) : 0.5f * E.m[c][k];
            S.m[c][k] = 0.5f * (R.m[c][k] + R.m[k][c]);
        }
#pragma unroll
    for (int c = 0; c < 3; ++c)
        if ((uint32_t)c < dim) {
            tr += E.m[c][c];
            trd += S.m[c][c];
        }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float d = c == k ? 1.0f : 0.0f;
            S.m[c][k] = (d * (lam * tr) + 2.0f * mu * E.m[c][k]) + (d * (lam_d * trd) + 2.0f * mu_d * S.m[c][k]);
        }
    return t3_mul(F, t3_transpose(S));
}

// ORDER2: every solid material uses strain order 2 (Green-Lagrange), so the
// log-series, square-root and inverse paths are compiled out.
// PLASTIC: some solid material is plastic; otherwise the plastic strain is
// zero throughout and its buffers are neither read nor written.
// LANES (4 or 2) threads share one solid, each with two entries' records in
// flight; lane 0 finishes the particle.
// Bound: L1 and L2 latency of the neighbors' records (32 + 16 bytes each), and
// for few solids the one thread that runs the stress chain.
template <bool ORDER2, bool PLASTIC, int LANES>
__global__ void __launch_bounds__(kThreads) k_solid_stress(SolidArgs a, Tables T, StageCoefs c) {
    step_begin();
    // a block of its own hands the wait's order on, so that no solid waits for the release
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0) step_publish(a.contact_bound + 2);
    step_let_next();  // after the wait: the kernels let in rely on the grid being there
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i = t / LANES, lane = t % LANES;
    if (i >= a.ns) return;  // whole groups leave together
    const SolidPos pi = load_pos(a.sx, i);
    const float4 xi = pi.x, Xs = pi.X;
    const float4 vi = a.sv[i];
    const uint32_t k1 = a.rl.off[i + 1];
    uint32_t k = a.rl.off[i] + lane;
    const DevMat& mm = T.mats[__float_as_uint(vi.w)];
    const SceneP& P = T.scenes[mm.scene];
    if (!P.solid_branch) return;  // a scene with a single solid skips the solid term
    const float4 L0 = a.L[3 * i], L1 = a.L[3 * i + 1], L2 = a.L[3 * i + 2];
    const float h2 = P.h2, kg = -6.0f * P.kconst;
    // strain.rs:139-160: F = sum V dx (x) (L gradW), Fdot likewise with dv
    constexpr int SETS = 4 / LANES;  // partial sums this thread holds
    float F[3][3], Fs[SETS][3][3] = {}, Fd[3][3], Fds[SETS][3][3] = {};
    auto add = [&](int set, const SolidPos& pj, float4 vj) {
        // gradW(X_j - X_i) as k_ref_fill computes it; V_j rides in X.w
        const float3 dX = sub3(pj.X, Xs);
        const float diff = h2 - dot3(dX, dX);
        const float sg = kg * diff * diff;
        const float3 g = make_float3(sg * dX.x, sg * dX.y, sg * dX.z);
        const float3 dx = sub3(pj.x, xi);
        const float3 dv = sub3(vj, vi);
        const float gr[3] = {pj.X.w * ((L0.x * g.x + L1.x * g.y) + L2.x * g.z),
                             pj.X.w * ((L0.y * g.x + L1.y * g.y) + L2.y * g.z),
                             pj.X.w * ((L0.z * g.x + L1.z * g.y) + L2.z * g.z)};
        const float x[3] = {dx.x, dx.y, dx.z}, v[3] = {dv.x, dv.y, dv.z};
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                Fs[set][cc][r] += x[r] * gr[cc];
                Fds[set][cc][r] += v[r] * gr[cc];
            }
    };
    for (; k + LANES < k1; k += 2 * LANES) {
        const uint32_t j0 = a.rl.nbr[k] & ~kSameMat, j1 = a.rl.nbr[k + LANES] & ~kSameMat;
        const SolidPos p0 = load_pos_at(a.sx, j0), p1 = load_pos_at(a.sx, j1);
        const float4 v0 = a.sv[j0], v1 = a.sv[j1];
        add(0, p0, v0);
        add(SETS - 1, p1, v1);
    }
    if (k < k1) {
        const uint32_t j = a.rl.nbr[k] & ~kSameMat;
        add(0, load_pos_at(a.sx, j), a.sv[j]);
    }
#pragma unroll
    for (int cc = 0; cc < 3; ++cc)
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            float f[SETS], fd[SETS];
#pragma unroll
            for (int q = 0; q < SETS; ++q) {
                f[q] = Fs[q][cc][r];
                fd[q] = Fds[q][cc][r];
            }
            F[cc][r] = sum4<LANES>(f);
            Fd[cc][r] = sum4<LANES>(fd);
        }
    if (lane != 0) return;
    // Bound used to skip the self-contact scan: max |u_i - u_0| over solids
    // (u = x - X) and whether any solid left the box.
    {
        const SolidPos p0 = load_pos(a.sx, 0);
        const float ux = (xi.x - Xs.x) - (p0.x.x - p0.X.x), uy = (xi.y - Xs.y) - (p0.x.y - p0.X.y),
                    uz = (xi.z - Xs.z) - (p0.x.z - p0.X.z);
        const float du = sqrtf((ux * ux + uy * uy) + uz * uz);
        bool outside = !finite3(xi) || !(du == du);
        const float pc[3] = {xi.x, xi.y, xi.z};
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float d = P.grid.dim[ax];
            if (d != 0.0f) {
                const float t = (pc[ax] - P.grid.min[ax]) / d;
                outside = outside || !(t >= 0.0f && t < 1.0f);
            }
        }
        const uint32_t mx = __reduce_max_sync(__activemask(), outside ? 0x7F800000u : __float_as_uint(du));
        const uint32_t any_out = __reduce_or_sync(__activemask(), outside ? 1u : 0u);
        if ((threadIdx.x & 31) == __ffs(__activemask()) - 1) {
            atomicMax(&a.contact_bound[0], mx);
            if (any_out) atomicOr(&a.contact_bound[1], 1u);
        }
    }
    const float2 lm = a.stiff ? a.stiff[i] : make_float2(mm.lam, mm.mu);
    StressRec out;
    out.cell = a.sc[i];
    if (ORDER2 && !PLASTIC) {
        T3 Fm, Fdm, Lm;
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                Fm.m[cc][r] = F[cc][r];
                Fdm.m[cc][r] = Fd[cc][r];
            }
        const float4 Lc[3] = {L0, L1, L2};
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
            Lm.m[cc][0] = Lc[cc].x;
            Lm.m[cc][1] = Lc[cc].y;
            Lm.m[cc][2] = Lc[cc].z;
        }
        const T3 A = t3_mul(stress_order2(Fm, Fdm, lm.x, lm.y, mm.lam_d, mm.mu_d, P.dim), Lm);
#pragma unroll
        for (int cc = 0; cc < 3; ++cc)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                out.A[cc][r] = A.m[cc][r];
                out.F[cc][r] = F[cc][r];
            }
        store_stress(a.AF, i, out);
        return;
    }
    M4 Fm = m4_zero(), Fdm = m4_zero(), Lm = m4_zero(), EP;
#pragma unroll
    for (int cc = 0; cc < 3; ++cc)
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            Fm.m[cc][r] = F[cc][r];
            Fdm.m[cc][r] = Fd[cc][r];
        }
    const float4 Lc[3] = {L0, L1, L2};
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
        Lm.m[cc][0] = Lc[cc].x;
        Lm.m[cc][1] = Lc[cc].y;
        Lm.m[cc][2] = Lc[cc].z;
        Lm.m[cc][3] = Lc[cc].w;
    }
    Lm.m[3][3] = 1.0f;
    if (PLASTIC) {
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const float4 e = a.ep[4 * i + cc];
            EP.m[cc][0] = e.x;
            EP.m[cc][1] = e.y;
            EP.m[cc][2] = e.z;
            EP.m[cc][3] = e.w;
        }
    } else {
        EP = m4_zero();
    }
    // solid.rs:334-341
    const M4 strain = PLASTIC ? m4_add(seth_hill<ORDER2>(Fm, mm.strain_order, P.dim), EP)
                              : seth_hill<ORDER2>(Fm, mm.strain_order, P.dim);
    const M4 rate = seth_hill_rate<ORDER2>(Fm, Fdm, mm.strain_order, P.dim);
    const M4 pk2 = m4_add(hooke(strain, lm.x, lm.y, P.dim), hooke(rate, mm.lam_d, mm.mu_d, P.dim));
    const M4 sigma = m4_mul(Fm, m4_transpose(pk2));
    const M4 A = m4_mul(sigma, Lm);
#pragma unroll
    for (int cc = 0; cc < 3; ++cc)
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            out.A[cc][r] = A.m[cc][r];
            out.F[cc][r] = F[cc][r];
        }
    store_stress(a.AF, i, out);
    // solid.rs:499-517: plastic strain rate (relaxation towards the
    // Johnson-Cook yield surface); the equivalent-strain factor is the
    // shader's integer (dim-1)/dim
    if (!PLASTIC) return;
    M4 kep = m4_zero();
    if (mm.plastic) {
        const float tr = trace_dim(EP, P.dim);
        const M4 dev = m4_sub(EP, m4_div(m4_scale(tr, m4_ident()), (float)P.dim));
        const float eq = (float)((int)(P.dim - 1) / (int)P.dim) * m4_dot(dev, dev);
        float sn = m4_dot(pk2, pk2);
        const float y = (mm.yield_strength + mm.work_hardening * powf(eq, mm.work_hardening_exp / 2.0f)) *
                        (1.0f + mm.kinematic_hardening * logf(1.0f));
        if (y * y <= sn) {
            sn = sqrtf(sn);
            kep = m4_scale((sn - y) / mm.relaxation_time, m4_div(pk2, sn));
        }
    }
    // stage update of the plastic strain (same scheme as the fluid epilogue)
    float4 kv[4];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) kv[cc] = make_float4(kep.m[cc][0], kep.m[cc][1], kep.m[cc][2], kep.m[cc][3]);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const uint32_t o = 4 * i + cc;
        if (a.ep_store) a.ep_store[o] = kv[cc];
        const float4 y0 = a.ep0[o];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c.c_acc != 0.0f) {
            if (!c.acc_first) acc = a.ep_acc[o];
            acc = lin4(c.c_acc, kv[cc], acc);
            if (!c.last) a.ep_acc[o] = acc;
        } else if (c.last) {
            acc = a.ep_acc[o];
        }
        float4 e = y0;
        if (c.last) {
            e = add4(y0, acc);
            a.ep_next[o] = e;
        } else {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c.c_prev0 != 0.0f) t = lin4(c.c_prev0, a.ep_prev0[o], t);
            if (c.c_prev1 != 0.0f) t = lin4(c.c_prev1, a.ep_prev1[o], t);
            if (c.c_prev2 != 0.0f) t = lin4(c.c_prev2, a.ep_prev2[o], t);
            if (c.c_self != 0.0f) t = lin4(c.c_self, kv[cc], t);
            a.ep_next[o] = add4(y0, t);
        }
        if (a.ep_kick)  // the next velocity-Verlet step's kick
            a.ep_kick[o] = add4(e, lin4(c.half, kv[cc], make_float4(0.f, 0.f, 0.f, 0.f)));
    }
}

// Bound: L1 and L2 latency of the neighbors' records (32 + 80 bytes each, two in
// flight per thread).  With separate arrays of float4 columns (position, reference
// position, cell, A, F: ten loads a neighbor) and two threads per solid the two
// kernels took 92 us per stage of 129,024 solids and 36 us for 1,274.
template <int LANES>
__global__ void __launch_bounds__(kThreads) k_solid_forces(SolidArgs a, Tables T) {
    step_let_next();  // the fluid kernel's pair sums need only the grid, which the stress kernel has waited for
    step_begin();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i = t / LANES, lane = t % LANES;
    if (i >= a.ns) return;  // whole groups leave together
    const SolidPos pi = load_pos(a.sx, i);
    const float4 xi = pi.x, Xi = pi.X;
    const uint32_t mat = __float_as_uint(a.sv[i].w);
    const uint32_t k1 = a.rl.off[i + 1];
    uint32_t k = a.rl.off[i] + lane;
    const StressRec si = load_stress(a.AF, i);
    const DevMat& mm = T.mats[mat];
    const SceneP& P = T.scenes[mm.scene];
    if (!P.solid_branch) return;
    const float m1 = mm.mass, d1 = xi.w;
    const float V1 = m1 / d1;
    const float h2 = P.h2, kc = P.kconst, hg_h = P.hg_h, eps_hh = P.eps_hh, eps_h = P.eps_h;
    const uint32_t dim = P.dim;
    constexpr int SETS = 4 / LANES;
    float fs[3][SETS] = {};
    // Reference neighbors of the same material: the elastic force
    // (solid.rs:343-374) and, when the neighbor also sits in the current
    // 3x3x3 cells, hourglass control (solid.rs:430-443; kernel(dX) is
    // non-zero exactly for these pairs).
    auto add = [&](int set, const SolidPos& pj, const StressRec& sj) {
        float &fx = fs[0][set], &fy = fs[1][set], &fz = fs[2][set];
        // dX = X_j - X_i, gradW(dX) = sg dX as k_ref_fill computes it
        const float3 dX = sub3(pj.X, Xi);
        const float diff = h2 - dot3(dX, dX);
        const float sg = -6.0f * kc * diff * diff;
        const float d2 = pj.x.w;
        const float V2 = __fdividef(m1, d2);  // GLSL division carries 2.5 ulp; the 2-ulp hardware quotient is used
        const float s = (-V1 * V2) * sg;
        // components at or above dim are dropped (solid.rs:370)
        fx += s * (((si.A[0][0] + sj.A[0][0]) * dX.x + (si.A[1][0] + sj.A[1][0]) * dX.y) +
                   (si.A[2][0] + sj.A[2][0]) * dX.z);
        if (dim >= 2)
            fy += s * (((si.A[0][1] + sj.A[0][1]) * dX.x + (si.A[1][1] + sj.A[1][1]) * dX.y) +
                          (si.A[2][1] + sj.A[2][1]) * dX.z);
        if (dim >= 3)
            fz += s * (((si.A[0][2] + sj.A[0][2]) * dX.x + (si.A[1][2] + sj.A[1][2]) * dX.y) +
                          (si.A[2][2] + sj.A[2][2]) * dX.z);
        if (in_stencil(sj.cell, si.cell)) {
            const float3 dx = sub3(pj.x, xi);
            const float l = sqrtf(dot3(dx, dx));
            float e[3];
#pragma unroll
            for (int r = 0; r < 3; ++r)
                e[r] = 0.5f * (((si.F[0][r] + sj.F[0][r]) * dX.x + (si.F[1][r] + sj.F[1][r]) * dX.y) +
                               (si.F[2][r] + sj.F[2][r]) * dX.z);
            const float ex = e[0] - dx.x, ey = e[1] - dx.y, ez = e[2] - dx.z;
            const float kern = kc * diff * diff * diff;  // W(dX)
            const float sh = ((__fdividef(100000000.0f * m1 * m1, d1 * d2) *
                               __fdividef(0.5f * ((ex * dx.x + ey * dx.y) + ez * dx.z), l + hg_h)) *
                              __fdividef(1.0f, l * l + eps_hh)) *
                             kern;
            const float u = __fdividef(sh, l + eps_h);
            fx -= u * dx.x;
            fy -= u * dx.y;
            fz -= u * dx.z;
        }
    };
    for (; k + LANES < k1; k += 2 * LANES) {
        const uint32_t e0 = a.rl.nbr[k], e1 = a.rl.nbr[k + LANES];
        const SolidPos p0 = load_pos_at(a.sx, e0 & ~kSameMat), p1 = load_pos_at(a.sx, e1 & ~kSameMat);
        const StressRec s0 = load_stress<true>(a.AF, e0 & ~kSameMat), s1 = load_stress<true>(a.AF, e1 & ~kSameMat);
        if (e0 & kSameMat) add(0, p0, s0);
        if (e1 & kSameMat) add(SETS - 1, p1, s1);
    }
    if (k < k1) {
        const uint32_t e = a.rl.nbr[k], j = e & ~kSameMat;
        if (e & kSameMat) add(0, load_pos_at(a.sx, j), load_stress<true>(a.AF, j));
    }
    float fx = sum4<LANES>(fs[0]), fy = sum4<LANES>(fs[1]), fz = sum4<LANES>(fs[2]);
    if (lane != 0) return;
    // Self-contact (solid.rs:428,445-450): same-material neighbors in the
    // current cells whose reference distance exceeds r_cut.  Skipped when
    // every solid is inside the box and r_cut - max|dx in stencil| exceeds
    // 2 max|u_k - u_0|, which bounds |dX| below r_cut for all such pairs.
    const float U = __uint_as_float(a.contact_bound[0]);
    const bool maybe = !mm.plastic && (P.contact_slack <= 0.0f || a.contact_bound[1] != 0u || !(2.0f * U < P.contact_slack));
    if (maybe && finite3(xi)) {
        for_reference_block_rows(xi, P, [&](uint32_t c0, uint32_t c1) {
            for (uint32_t k = a.start[c0]; k < a.start[c1]; ++k) {
                if (a.mat[k] != mat) continue;
                const uint32_t sj = a.sid_sorted[k];
                if (sj == kInvalid) continue;
                const float4 xj = a.rec[2 * (size_t)k];
                const float3 dx = sub3(xj, xi);
                const float3 dX = sub3(a.ref[sj], Xi);
                const float dXX = dot3(dX, dX), dxx = dot3(dx, dx);
                if (!(dXX > P.rcut2 && dxx < P.rcut2)) continue;
                const float l = sqrtf(dxx);
                const float dr = fmaxf(P.rcut - l, 0.0f);
                const float cs = -5000.0f * sqrtf(dr * P.r_geom);
                fx += (cs * dx.x) / l;
                fy += (cs * dx.y) / l;
                fz += (cs * dx.z) / l;
            }
        });
    }
    // solid.rs:492-494 (den term is zero)
    a.ksol[i] = make_float4(__fdiv_rn(fx, d1), __fadd_rn(__fdiv_rn(fy, d1), -P.g), __fdiv_rn(fz, d1), 0.0f);
}

}  // namespace

int ref_lists_count(const float4* ref, const uint32_t* mat_of, uint32_t ns, const GridBuffers& gb, const Tables& T,
                    uint32_t* count, cudaStream_t st) {
    k_ref_count<<<blocks_for(ns, kThreads), kThreads, 0, st>>>(ref, mat_of, ns, gb.start, gb.perm, T, count);
    return 1;
}

int ref_lists_fill(const float4* ref, const uint32_t* mat_of, uint32_t ns, const GridBuffers& gb, const Tables& T,
                   SolidRefList& rl, float4* L, cudaStream_t st) {
    k_ref_fill<<<blocks_for(ns, kThreads), kThreads, 0, st>>>(ref, mat_of, ns, gb.start, gb.perm, T, rl.off, rl.nbr,
                                                              rl.gw);
    k_ref_L<<<blocks_for(ns, kThreads), kThreads, 0, st>>>(ref, mat_of, ns, rl.off, rl.nbr, rl.gw, T, L);
    return 2;
}

namespace {
template <int L>
void launch_solid_lanes(const SolidArgs& a, const Tables& T, const StageCoefs& c, cudaStream_t st) {
    const uint32_t blocks = blocks_for(a.ns * L, kThreads);
    const uint32_t more = blocks + 1u;  // and the block that publishes
    if (a.all_order2 && !a.any_plastic) launch_step(k_solid_stress<true, false, L>, more, kThreads, 0, st, a, T, c);
    else if (a.all_order2) launch_step(k_solid_stress<true, true, L>, more, kThreads, 0, st, a, T, c);
    else if (!a.any_plastic) launch_step(k_solid_stress<false, false, L>, more, kThreads, 0, st, a, T, c);
    else launch_step(k_solid_stress<false, true, L>, more, kThreads, 0, st, a, T, c);
    launch_step(k_solid_forces<L>, blocks, kThreads, 0, st, a, T);
}
}  // namespace

int launch_solid(const SolidArgs& a, const Tables& T, const StageCoefs& c, cudaStream_t st) {
    if (a.ns == 0) return 0;
    if (!a.counters_cleared) cudaMemsetAsync(a.contact_bound, 0, kStageWords * sizeof(uint32_t), st);
    // a.sx (its stage half), a.sv and a.sc were written by the stage's gather (gather_state)
    if (a.ns <= kFewSolids) launch_solid_lanes<4>(a, T, c, st);
    else launch_solid_lanes<2>(a, T, c, st);
    return 2;
}

}  // namespace arp
