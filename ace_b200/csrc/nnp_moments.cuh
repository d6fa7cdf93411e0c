// nnp_moments.cuh -- symmetry functions and forces of GAUSS angular blocks
// with integer zeta through moments of the neighbours' directions.
//
// A GAUSS angular function is (0.5 + lambda/2 cos)^zeta w_d(r_a) w_d(r_b)
// summed over the pairs (a, b) of two neighbour elements, w_d(r) = fc(r)
// exp(-a_d r^2) (BasisA::symmf, src/nnp/basis_angular.cpp:212-260).  For
// integer zeta <= L the power is a polynomial in cos = u_a . u_b; expanded in
// Legendre polynomials, sum_l c_l P_l(u_a . u_b), each P_l splits by the
// addition theorem into products of one neighbour's functions, so the sum
// over pairs becomes one over neighbours:
//   A^J_{lm,d} = sum_{a in J} w_d(r_a) Y_lm(u_a)            (moments)
//   S^{JK}_{l,d} = sum_m A^J_{lm,d} A^K_{lm,d}
//   G_f = sum_l c_{f,l} S^{JK}_{l,d}                          (J != K)
//   G_f = (sum_l c_{f,l} S^{JJ}_{l,d} - f_f(1) sum_a w_d^2) / 2   (J == K:
//         the sum over ordered pairs without the pairs of a slot with itself)
// and with e_f = dE/dG_f the derivative of the energy with respect to a
// neighbour's displacement is that of sum_d w_d(r) sum_lm B^J_{lm,d} Y_lm(u),
//   B^J_{lm,d} = sum_K (sum_f e_f c_{f,l} [1 + (J == K)]) A^K_{lm,d},
// so neither pass visits pairs.  A pair term costs ~80 instructions in the
// force pass and an atom of the batched workload has 1000 pairs; a neighbour
// (45 per atom) costs ~500 there and ~400 in the symmetry functions.
//
// The moment form's rounding error is ~1e-7 of sum_l |c_l S_l| + f(1) sum w^2, a
// pair sum's ~1e-7 of the sum itself.  The two differ where neighbours lie to one
// side of the centre (an adatom, a tip) or are few: ((1 - cos)/2)^8 of neighbours
// in a cone, ((1 + cos)/2)^8 of two on opposite sides are 1e-4 to 1e-8 of it.  So a
// block is summed pair by pair when one of its functions comes out below
// NNP_MOM_CANCEL of that sum, at any number of pairs.  The symmetry functions
// decide, from the sums that they form anyway, and leave a bit per block in
// mom_mask, which the forces and tangents follow; lists of the (row, block)
// entries are worked off by groups of lanes (mom_few_*: at most NNP_MOM_FEW pairs,
// mom_wide_*: more).  In random cells of 0.05 atoms per cubic A of three elements
// 9 % of the blocks are listed as few and 3.5 % as wide, in crystals none.
// With 1/16 the errors of G and of the forces are those of pair sums, function by
// function (rms), over adatoms, tips, surfaces and random cells; with 1/32 functions
// of zeta = 8 at a free surface had 4.5 times the pair sum's.
//
// Y_lm(u) = Q_lm(z) Re/Im (x + i y)^m with Q_lm the monic polynomial
// proportional to d^m P_l / dz^m: Q_{l+1,m} = z Q_lm - beta_lm Q_{l-1,m},
// beta_lm = (l^2 - m^2) / (4 l^2 - 1), and dQ_lm/dz = (l - m) Q_{l,m+1}.
// The factors N_lm that make sum_m N_lm^2 Y_lm Y_lm = P_l multiply the sums.
//
// Plain CUDA C++ for NVRTC, like nnp_device.cuh.  The class M (written by
// nnp_jit.cpp) gives the potential's sizes and its radial functions:
//   T elements, L largest zeta, ND damping factors per centre element,
//   NR radial and NA angular functions of the largest block, NCUT cutoffs,
//   cut(c), rci_lo(c): cutoff c and the low part of its 1/rc,
//   SAME: every centre element has the same damping factors, and then
//   damp_a(d), damp_lo(d), damp_cut(d): exponent (high and low part) and cutoff,
//   norm(c): factor of the monic Y_lm of component c, gnorm(c): times (l - m)!,
//   radial_row(II, t, r, fc, row): values of the radial functions of a
//   neighbour of element t, radial_force(II, t, r, fc, fcd, eb, out): sum of
//   eb_f dG_f/dr, few_symm(II, tt, cs, w, acc): acc_f += x_f^zeta w_d,
//   few_force(II, tt, cs, e, wa, wda, wb, wdb, hc, ha, hb): dE/dcos, dE/dr_a and
//   dE/dr_b of one pair, radial_drow(II, t, r, fc, fd, row): slopes of the radial
//   functions, few_tangent(II, tt, cs, w, dw, acc): acc_f += dx_f^zeta/dcos w_d +
//   x_f^zeta dw_d.
#pragma once

#include "nnp_device.cuh"

#define NNP_MOM_MAXL 8        // largest zeta taken (above, a moment set is larger than the pairs it replaces)
#define NNP_MOM_MAXD 4        // damping factors of one centre element
#define NNP_MOM_SYMM_WARPS 2  // warps per block, symmetry functions with a warp per atom (15 KB of shared memory each)
#define NNP_MOM_THREADS 128   // threads per block, symmetry functions with a thread per atom
#define NNP_MOM_THREAD_T 4    // most elements of that form (its sums of pairs of elements are unrolled)
#define NNP_MOM_FORCE_WARPS 4 // warps per block, forces
#define NNP_MOM_CANCEL 0.0625f // blocks with a function below this part of its terms' absolute sum are summed pair by pair
#define NNP_MOM_FEW 15        // 16 lanes take such a block if it has at most this many pairs
#define NNP_MOM_FEW_THREADS 128
#define NNP_MOM_LIST_BLOCKS 8 // blocks per SM of the list kernels (64 registers), all resident

namespace nnp {

// Components of one (element, damping pair): m = 0 first (l = 0..L, padded to
// an even count), then for m = 1..L and l = m..L the cos and sin parts side by
// side, so that one 16-byte load reads both parts for two damping factors.
NNP_HD constexpr int mom_m0(int L) { return (L + 2) & ~1; }
NNP_HD constexpr int mom_base(int L, int m)   // first component of m >= 1
{
    return mom_m0(L) + 2 * ((m - 1) * (L + 1) - (m * (m - 1)) / 2);
}
NNP_HD constexpr int mom_comps(int L) { return mom_base(L, L) + 2; }

// Moments in memory: component k = ((element * pairs of damping factors) + pair)
// * comps + component of row r (the r-th atom of the visiting order) is the
// float2 at mom_at(r, k, vals, sh): 2^sh rows interleaved.  Written with a thread
// per row sh = NNP_MOM_SH_T: a warp's access is two whole lines (with 4 rows it
// touched 8 lines, and the tag lookups bounded both kernels: symmetry functions
// of 1.09 M atoms 2.27 -> 2.13 ms, forces 3.51 -> 3.19 ms); written with a warp
// per row sh = NNP_MOM_SH_W: it writes one row's components next to its
// neighbours'.  mom_cnt holds 8 neighbour counts (by element) per row, mom_mask
// the row's blocks that are summed over pairs.
#define NNP_MOM_SH_T 5
#define NNP_MOM_SH_W 2
NNP_HD constexpr int mom_vals(int T, int ND, int L) { return T * ((ND + 1) / 2) * mom_comps(L); }
NNP_HD inline i64 mom_at(i64 r, int k, int vals, int sh) { return (((r >> sh) * vals + k) << sh) + (r & ((1 << sh) - 1)); }

// Blocks that are summed over pairs (or have none): a bit per block of each row, and
// the (row, block) entries, those of few pairs from the start of one array, the
// others from its end backwards (an entry is in one of the two, so rows x blocks
// hold both).
struct MomLists {
    int2 *few, *wide;             // the first entry of either
    int *n;                       // their numbers (DevErr::few, DevErr::wide)
    unsigned long long *mask;
};

// pairs of block (J, K) of an atom
NNP_HD inline int mom_pairs(const unsigned short *cnt, int J, int K)
{
    return J == K ? cnt[J] * (cnt[J] - 1) / 2 : cnt[J] * cnt[K];
}

// Table of a potential (floats, nnp_api.cu):
//   norm[comps] (factors of the monic Y_lm; 0 at the padding),
//   fnorm[comps] (factors of d^m P_l / dz^m), deg[comps] (l, as int),
//   per element: low parts of the damping exponents [NNP_MOM_MAXD],
//   per element and angular function f, [L + 2][fmax]: coefficients c_0 .. c_L
//   (halved for J == K), then f(1)/2 for J == K and 0 otherwise,
//   per element and function, as int: tt | d << 8 | J << 16 | K << 24,
//   then, 16-byte aligned, per element and function mom_dl(L) float2: its
//   coefficients in dE/dA (those above, twice for J == K) in .x for an even
//   damping factor, in .y for an odd one
struct MomTab {
    const float *norm, *fnorm;
    const int *deg;
    const float *a_lo;
    const float *coef;
    const int *fun;
    const float2 *dcoef;
    int fmax;
};

NNP_HD constexpr int mom_dl(int L) { return (L + 3) & ~1; }
NNP_HD inline int mom_tab_base(int T, int L, int fmax)       // floats before dcoef
{
    return (3 * mom_comps(L) + T * NNP_MOM_MAXD + T * fmax * (L + 3) + 3) & ~3;
}

NNP_HD inline int mom_tab_floats(int T, int L, int fmax)
{
    return mom_tab_base(T, L, fmax) + 2 * T * fmax * mom_dl(L);
}

NNP_HD inline MomTab mom_tab(const float *p, int T, int L, int fmax)
{
    MomTab t;
    t.dcoef = reinterpret_cast<const float2 *>(p + mom_tab_base(T, L, fmax));
    t.norm = p; p += mom_comps(L);
    t.fnorm = p; p += mom_comps(L);
    t.deg = reinterpret_cast<const int *>(p); p += mom_comps(L);
    t.a_lo = p; p += T * NNP_MOM_MAXD;
    t.coef = p; p += T * fmax * (L + 2);
    t.fun = reinterpret_cast<const int *>(p);
    t.fmax = fmax;
    return t;
}

// Shared memory of one warp.  Symmetry functions: 32 neighbour rows of
// mom_stage floats (odd stride: lanes write their rows without bank
// conflicts), damping factors per row, moments, sums of w_d^2, S, G row.
NNP_HD constexpr int mom_stage(int L, int NR, int ND) { return (mom_comps(L) + NR + ND) | 1; }
NNP_HD constexpr int mom_s_vals(int T, int ND, int L) { return T * (T + 1) / 2 * ((ND + 1) / 2) * (L + 1); }
NNP_HD constexpr int mom_symm_floats(int T, int ND, int L, int NR, int gstride)
{
    return ((32 * mom_stage(L, NR, ND) + 3) & ~3) + 64 * ((ND + 1) / 2) + 2 * mom_vals(T, ND, L) + T * NNP_MOM_MAXD +
           ((2 * mom_s_vals(T, ND, L) + 3) & ~3) + gstride + 4;
}
// Forces, one thread per atom: D of one neighbour element, dE/dG.
NNP_HD inline int mom_force_thread_floats(int T, int L, int gstride)
{
    return NNP_MOM_THREADS * (2 * T * (L + 1) + gstride);
}

// One thread per atom: S and the sums of w_d^2 of its NNP_MOM_THREADS threads.
NNP_HD constexpr int mom_thread_floats(int T, int ND, int L)
{
    return NNP_MOM_THREADS * 2 * (mom_s_vals(T, ND, L) + T * ((ND + 1) / 2));
}
// Forces, per atom of a warp's group: B, D, the self terms, the dE/dG row.
NNP_HD constexpr int mom_force_floats(int T, int ND, int L, int gstride)
{
    return 2 * mom_vals(T, ND, L) + ((2 * mom_s_vals(T, ND, L) + 3) & ~3) + T * NNP_MOM_MAXD + gstride;
}

#if defined(__CUDACC__)

// ---------------------------------------------------------------- packed FP32 pairs

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f32x2 dup2(float a) { return pk2(a, a); }
__device__ __forceinline__ void up2(f32x2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// the line of a record that is read some iterations later
__device__ __forceinline__ void mom_prefetch(const float4 *p)
{
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

NNP_HD constexpr float mom_beta(int l, int m) { return (float)((double)(l * l - m * m) / (double)(4 * l * l - 1)); }

// ---------------------------------------------------------------- one neighbour

// Second derivative of the cutoff function (f: its value).
__device__ __forceinline__ float cutoff_curve(const DevCut &c, float r, float f)
{
    switch (c.name) {
    case CUT_COS: return c.pirci * c.pirci * (0.5f - f);
    case CUT_TANH: {
        const float t = tanhf(1.f - r * c.rci), t2 = t * t;
        return r < c.rc ? 6.f * t * (1.f - 2.f * t2) * (1.f - t2) * c.rci * c.rci : 0.f;
    }
    case CUT_POLY3: return r < c.rc ? (12.f * (r * c.rci) - 6.f) * c.rci * c.rci : 0.f;
    default: return 0.f;
    }
}

// Distance, unit vector, cutoff values and damping factors of a neighbour.
// The damping factors set the error of the moments, so what FP32 rounding of
// their arguments would lose is put back to first order: r = r_hi + r_lo
// from the residual of the square root, 1/rc and the exponents as hi + lo
// (RMS error of w over a neighbour shell 1.2e-7 -> 0.65e-7).
template <class M, bool DER>
struct MomNbr {
    float ux, uy, uz, r, ir;
    float fc[M::NCUT], fd[M::NCUT];
    float w[M::ND], wd[M::ND];

    // Ty: centre element, a_lo: low parts of its damping exponents
    __device__ __forceinline__ void set(const float4 e, const DevType &Ty, const float *a_lo)
    {
        const float r2 = fmaf(e.x, e.x, fmaf(e.y, e.y, e.z * e.z));
        // r to the nearest float: the reciprocal root's own error is the same for all
        // neighbours of a crystal's shell, so it would not average out (virial)
        const float q = rsqrtf(r2), r0 = r2 * q, d = 0.5f * q * fmaf(-r0, r0, r2);
        r = r0 + d;
        const float rlo = d - (r - r0);
        ir = fmaf(q * q, d, q);
        ux = e.x * ir;
        uy = e.y * ir;
        uz = e.z * ir;
#pragma unroll
        for (int c = 0; c < M::NCUT; ++c) {
            const DevCut C = M::cut(c);
            cutoff_fg(C, r, fc[c], fd[c]);
            const float x = r * C.rci;
            // fc(r + rlo), its argument's rounding and the low part of 1/rc: f += f' rc dx, and
            // the slope likewise: 1/rc is off alike for all neighbours, and the virial, a sum
            // over the slopes, was off by 3e-7 of its norm in crystals with rc = 6.5 (now 1e-7)
            const float dx = fmaf(rlo, C.rci, fmaf(r, M::rci_lo(c), fmaf(r, C.rci, -x)));
            const float h = cutoff_curve(C, r, fc[c]);
            fc[c] = fmaf(fd[c] * C.rc, dx, fc[c]);
            fd[c] = fmaf(h * C.rc, dx, fd[c]);
        }
#pragma unroll
        for (int d = 0; d < M::ND; ++d) {
            w[d] = 0.f;
            wd[d] = 0.f;
            if (M::SAME || d < Ty.ndamp) {
                const float a = M::SAME ? M::damp_a(d) : Ty.damp_a[d], t = -a * r2;
                float ex = expf(t);
                ex = fmaf(ex, fmaf(-a, r2, -t) - (M::SAME ? M::damp_lo(d) : a_lo[d]) * r2, ex);
                const int dc = M::SAME ? M::damp_cut(d) : Ty.damp_cut[d];
                float f = fc[0], g = fd[0];
#pragma unroll
                for (int c = 1; c < M::NCUT; ++c)
                    if (dc == c) {
                        f = fc[c];
                        g = fd[c];
                    }
                w[d] = f * ex;
                if (DER) wd[d] = (g - 2.f * a * r * f) * ex;
            }
        }
    }
};

// Writes the L-moment functions Y_lm(u) of one neighbour to row (components
// as mom_base; the padding is not written).
template <int L>
__device__ __forceinline__ void mom_harmonics(float x, float y, float z, float *row)
{
    float cm = 1.f, sm = 0.f;
#pragma unroll
    for (int m = 0; m <= L; ++m) {
        float q0 = 1.f, q1 = 0.f;
#pragma unroll
        for (int l = m; l <= L; ++l) {
            if (m == 0) {
                row[l] = q0;
            } else {
                row[mom_base(L, m > 0 ? m : 1) + 2 * (l - m)] = q0 * cm;
                row[mom_base(L, m > 0 ? m : 1) + 2 * (l - m) + 1] = q0 * sm;
            }
            const float t = (l == m) ? z * q0 : fmaf(z, q0, -mom_beta(l, m) * q1);
            q1 = q0;
            q0 = t;
        }
        const float c = cm * x - sm * y, s = sm * x + cm * y;
        cm = c;
        sm = s;
    }
}

// d^m P_l / dz^m for l = m .. L (both halves equal):
// (l + 1 - m) Q_{l+1} = (2l + 1) z Q_l - (l + m) Q_{l-1}, Q_mm = (2m - 1)!!.
template <int L, int m>
__device__ __forceinline__ void mom_polys(float z, f32x2 *q)
{
    float q0 = 1.f, q1 = 0.f;
#pragma unroll
    for (int k = 1; k < 2 * m; k += 2) q0 *= (float)k;
#pragma unroll
    for (int l = m; l <= L; ++l) {
        q[l] = dup2(q0);
        const float a = (float)(2 * l + 1) / (float)(l + 1 - m), b = (float)(l + m) / (float)(l + 1 - m);
        const float t = (l == m) ? a * z * q0 : fmaf(a, z * q0, -b * q1);
        q1 = q0;
        q0 = t;
    }
}

// Value V and gradient (X, Y, Z) of sum_lm B_lm Q_lm(z) Re/Im (x + i y)^m for
// each damping factor: the terms of m and above, qa = Q_{l,m}, (cm, sm) = (x +
// i y)^m, (cp, sp) = (x + i y)^(m - 1).
template <int L, int NDP, int m>
__device__ __forceinline__ void mom_gradient(const ulonglong2 *B, float x, float y, float z, const f32x2 *qa, float cm,
                                             float sm, float cp, float sp, f32x2 *V, f32x2 *X, f32x2 *Y, f32x2 *Z)
{
    constexpr int NC = mom_comps(L);
    f32x2 qb[L + 2];
    if constexpr (m < L) mom_polys<L, m + 1>(z, qb);
#pragma unroll
    for (int p = 0; p < NDP; ++p) {
        f32x2 C = 0ull, S = 0ull, Cz = 0ull, Sz = 0ull;
        if constexpr (m == 0) {
#pragma unroll
            for (int l = 0; l <= L; l += 2) {
                const ulonglong2 b = B[(p * NC + l) / 2];
                C = fma2(b.x, qa[l], C);
                if (l > 0) Cz = fma2(b.x, qb[l], Cz);
                if (l + 1 <= L) {
                    C = fma2(b.y, qa[l + 1], C);
                    Cz = fma2(b.y, qb[l + 1], Cz);
                }
            }
            V[p] = C;
            X[p] = Y[p] = 0ull;
            Z[p] = Cz;
        } else {
#pragma unroll
            for (int l = m; l <= L; ++l) {
                const ulonglong2 b = B[(p * NC + mom_base(L, m)) / 2 + (l - m)];
                C = fma2(b.x, qa[l], C);
                S = fma2(b.y, qa[l], S);
                if (l > m) {
                    Cz = fma2(b.x, qb[l], Cz);
                    Sz = fma2(b.y, qb[l], Sz);
                }
            }
            const f32x2 c2 = dup2(cm), s2 = dup2(sm), mc = dup2((float)m * cp), ms = dup2((float)m * sp),
                        nms = dup2(-(float)m * sp);
            V[p] = fma2(C, c2, fma2(S, s2, V[p]));
            X[p] = fma2(C, mc, fma2(S, ms, X[p]));
            Y[p] = fma2(C, nms, fma2(S, mc, Y[p]));
            if (m < L) Z[p] = fma2(Cz, c2, fma2(Sz, s2, Z[p]));
        }
    }
    if constexpr (m < L)
        mom_gradient<L, NDP, m + 1>(B, x, y, z, qb, cm * x - sm * y, sm * x + cm * y, cm, sm, V, X, Y, Z);
}

// ---------------------------------------------------------------- blocks of few pairs

// Block (J, K) of few pairs as 16 lanes see it: neighbour h < nn is slot so + h
// of the larger element (h < no; J == K: of the element) or sp + h - no of the
// other, and lane p < pairs has the pair of neighbours a and b.  With a lane per
// pair instead of a lane per neighbour of the larger element that walks the other
// ones, 1.09 M atoms: symmetry functions 1.97 -> 1.91 ms, forces 2.41 -> 2.32 ms.
struct MomFew {
    int J, K, so, no, sp, np, nn, pairs, a, b;
};

// Elements of block tt, the first slots and numbers of their neighbours (cnt: an
// atom's eight counts, 16-byte aligned).
template <int T>
__device__ __forceinline__ void mom_block(const unsigned short *cnt, int tt, int &J, int &K, int &sJ, int &nJ, int &sK, int &nK)
{
    const uint4 v = *reinterpret_cast<const uint4 *>(cnt);
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
    K = 0;
#pragma unroll
    for (int k = 1; k < T; ++k) K += tt >= k * (k + 1) / 2;
    J = tt - K * (K + 1) / 2;
    sJ = nJ = sK = nK = 0;
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const int c = (int)((w[k / 2] >> (k & 1 ? 16 : 0)) & 0xffffu);
        sJ += k < J ? c : 0;
        nJ = k == J ? c : nJ;
        sK += k < K ? c : 0;
        nK = k == K ? c : nK;
    }
}

template <int T>
__device__ __forceinline__ MomFew mom_few(const unsigned short *cnt, int tt, int p)
{
    MomFew f;
    int sJ, nJ, sK, nK;
    mom_block<T>(cnt, tt, f.J, f.K, sJ, nJ, sK, nK);
    const bool j = nJ >= nK;
    f.so = j ? sJ : sK;
    f.sp = j ? sK : sJ;
    f.no = j ? nJ : nK;
    f.np = j ? nK : nJ;
    if (f.J == f.K) {                                            // at most 6 neighbours: a < b, p = b (b - 1) / 2 + a
        f.nn = f.no;
        f.pairs = f.no * (f.no - 1) / 2;
        f.b = 1 + (p >= 1) + (p >= 3) + (p >= 6) + (p >= 10);
        f.a = p - f.b * (f.b - 1) / 2;
    } else {                                                     // at most 16: p = (b - no) no + a
        f.nn = f.no + f.np;
        f.pairs = f.no * f.np;
        const int q = (int)__fdividef((float)p + 0.5f, (float)f.no);
        f.b = f.no + q;
        f.a = p - q * f.no;
    }
    return f;
}

__device__ __forceinline__ int mom_few_slot(const MomFew &f, int h)
{
    const int k = min(h, f.nn - 1);
    return k < f.no ? f.so + k : f.sp + k - f.no;
}

// Symmetry functions of block tt by the 16 lanes `mask` (h: lane among them),
// to Gb (the block's functions).  src: the atom's records.
template <class M>
__device__ __forceinline__ void mom_few_symm(unsigned mask, int h, const float4 *__restrict__ src,
                                             const unsigned short *cnt, const DevType &Ty, int II, int tt,
                                             const float *a_lo, float *Gb)
{
    const MomFew b = mom_few<M::T>(cnt, tt, h);
    MomNbr<M, false> v;
    v.set(src[mom_few_slot(b, h)], Ty, a_lo);
    float cs = 0.f, w[M::ND], acc[M::NA];
    cs = fmaf(__shfl_sync(mask, v.ux, b.a, 16), __shfl_sync(mask, v.ux, b.b, 16), cs);
    cs = fmaf(__shfl_sync(mask, v.uy, b.a, 16), __shfl_sync(mask, v.uy, b.b, 16), cs);
    cs = fmaf(__shfl_sync(mask, v.uz, b.a, 16), __shfl_sync(mask, v.uz, b.b, 16), cs);
#pragma unroll
    for (int d = 0; d < M::ND; ++d) w[d] = __shfl_sync(mask, v.w[d], b.a, 16) * __shfl_sync(mask, v.w[d], b.b, 16);
#pragma unroll
    for (int f = 0; f < M::NA; ++f) acc[f] = 0.f;
    if (h < b.pairs) M::few_symm(II, tt, cs, w, acc);
    const int n = Ty.ba[tt].n;
#pragma unroll
    for (int f = 0; f < M::NA; ++f) {
        float s = acc[f];
#pragma unroll
        for (int q = 8; q; q >>= 1) s += __shfl_xor_sync(mask, s, q, 16);
        if (h == 0 && f < n) Gb[f] = s;
    }
}

// ---------------------------------------------------------------- blocks of many pairs
//
// A warp per block.  The block's neighbours (of J, then of K; J == K: of the
// element) are loaded a lane each, 32 at a time (such blocks have mostly 7 to 16).
// For sums over pairs a lane then takes a pair, with the values of both ends by
// shuffles (mom_wide_pairs); for the forces it takes a neighbour a (as many lanes each
// as fit, a's partners divided among them) and walks the partners, so that it gets
// the gradient at a without a second exchange, at two evaluations a pair
// (mom_wide_walk).
// Bound: latency of the chain from the list entry to the neighbours (entry and atom
// are fetched one turn ahead), then issue.

struct MomWide {
    int sJ, nJ, sK, nn;           // first slots, neighbours of J and of the block
    bool one;                     // J == K
    __device__ __forceinline__ int slot(int k) const { return k < nJ ? sJ + k : sK + k - nJ; }
};

template <int T>
__device__ __forceinline__ MomWide mom_wide(const unsigned short *cnt, int tt)
{
    MomWide w;
    int J, K, nK;
    mom_block<T>(cnt, tt, J, K, w.sJ, w.nJ, w.sK, nK);
    w.one = J == K;
    w.nn = w.nJ + (w.one ? 0 : nK);
    return w;
}

// Entries q, q + step, .. of the list, the next entry and its atom on the way.
struct MomQueue {
    const int2 *p;
    const int *order;
    int q, n, step, i, ni;
    int2 it, nx;
    __device__ __forceinline__ MomQueue(const int2 *list, int count, const int *ord, int first, int stride)
        : p(list), order(ord), q(first), n(count), step(stride), i(0), ni(0)
    {
        if (q < n) {
            it = at(q);
            nx = at(q + step);
            i = order[it.x];
        }
    }
    __device__ __forceinline__ int2 at(int k) const { return p[-(i64)min(k, n - 1)]; }
    __device__ __forceinline__ void ahead() { ni = order[nx.x]; }
    __device__ __forceinline__ void next()
    {
        q += step;
        it = nx;
        i = ni;
        nx = at(q + step);
    }
};

// First entry of the few-pair list for a group of 16 lanes, of `all` groups: the
// round goes on where that of the other list, a warp each, ended.
__device__ __forceinline__ int mom_few_first(const MomLists &ls, int group, int all)
{
    const int f = group - 2 * (ls.n[1] % (all / 2));
    return f < 0 ? f + all : f;
}

// load(slot) -> a neighbour's values; pair(A, la, B, lb, ok) for every pair of the
// block: its ends are the values of lanes la in A and lb in B (ok: the lane has one)
template <class Load, class Pair>
__device__ __forceinline__ void mom_wide_pairs(const MomWide &w, Load load, Pair pair)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int a0 = 0; a0 < (w.one ? w.nn : w.nJ); a0 += 32) {
        const int ca = min(32, w.nn - a0);
        const auto A = load(w.slot(a0 + min(lane, ca - 1)));
#pragma unroll 1
        for (int b0 = a0; b0 < w.nn; b0 += 32) {
            const int cb = min(32, w.nn - b0);
            auto B = A;
            if (b0 != a0) B = load(w.slot(b0 + min(lane, cb - 1)));
            // a's are lanes [0, na) of A, b's lanes [fb, cb) of B
            const int na = w.one ? ca : min(ca, w.nJ - a0), fb = w.one ? 0 : max(w.nJ - b0, 0);
            const bool tri = w.one && a0 == b0;
            const int np = tri ? na * (na - 1) / 2 : na * max(cb - fb, 0);
#pragma unroll 1
            for (int p0 = 0; p0 < np; p0 += 32) {
                const int p = min(p0 + lane, np - 1);
                // p = b (b - 1) / 2 + a, a < b, or (b - fb) na + a (exact in FP32: p < 1024)
                const int b = tri ? (int)(0.5f + sqrtf(0.25f + 2.f * (float)p)) : fb + (int)__fdividef((float)p + 0.5f, (float)na);
                const int a = tri ? p - b * (b - 1) / 2 : p - (b - fb) * na;
                pair(A, a, B, b, p0 + lane < np);
            }
        }
    }
}

// take(v, lane) -> the values that a lane holds; pair(a, B, q, ok) for each step: b is
// the value of lane q in B (ok: the lane has a pair); end(A, a, lane that loaded a,
// first lane of a, lanes per a)
template <class Load, class Take, class Pair, class End>
__device__ __forceinline__ void mom_wide_walk(const MomWide &w, Load load, Take take, Pair pair, End end)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int a0 = 0; a0 < w.nn; a0 += 32) {
        const int ca = min(32, w.nn - a0);
        const int sh = 31 - __clz(32 / ca);                      // 1 << sh lanes per a
        const int la = min(lane >> sh, ca - 1), ia = a0 + la, part = lane & ((1 << sh) - 1);
        const bool act = (lane >> sh) < ca;
        const auto A = load(w.slot(a0 + min(lane, ca - 1)));
        const auto a = take(A, la);
#pragma unroll 1
        for (int b0 = 0; b0 < w.nn; b0 += 32) {
            const int cb = min(32, w.nn - b0);
            auto B = A;
            if (b0 != a0) B = load(w.slot(b0 + min(lane, cb - 1)));
            // partners of a, and the most that any a has
            const int lo = w.one || ia >= w.nJ ? b0 : max(b0, w.nJ), hi = w.one || ia < w.nJ ? b0 + cb : min(b0 + cb, w.nJ);
            const int most = w.one ? cb : max(b0 + cb - max(b0, w.nJ), min(b0 + cb, w.nJ) - b0);
#pragma unroll 1
            for (int t = 0; t < most; t += 1 << sh) {
                const int q = lo + part + t;
                pair(a, B, min(q - b0, cb - 1), act && q < hi && !(w.one && q == ia));
            }
        }
        end(A, a, la, act && part == 0, 1 << sh);
    }
}

// Symmetry functions of block tt by a warp, to Gb.
template <class M>
__device__ __noinline__ void mom_wide_symm(const float4 *__restrict__ src, const unsigned short *cnt, const DevType &Ty,
                                           int II, int tt, const float *a_lo, float *Gb)
{
    struct Nbr {
        float u[3], w[M::ND];
    };
    float acc[M::NA];
#pragma unroll
    for (int f = 0; f < M::NA; ++f) acc[f] = 0.f;
    mom_wide_pairs(
        mom_wide<M::T>(cnt, tt),
        [&](int k) {
            MomNbr<M, false> v;
            v.set(src[k], Ty, a_lo);
            Nbr o;
            o.u[0] = v.ux;
            o.u[1] = v.uy;
            o.u[2] = v.uz;
#pragma unroll
            for (int d = 0; d < M::ND; ++d) o.w[d] = v.w[d];
            return o;
        },
        [&](const Nbr &A, int a, const Nbr &B, int b, bool ok) {
            float cs = 0.f, w[M::ND];
#pragma unroll
            for (int x = 0; x < 3; ++x)
                cs = fmaf(__shfl_sync(NNP_FULL, A.u[x], a), __shfl_sync(NNP_FULL, B.u[x], b), cs);
#pragma unroll
            for (int d = 0; d < M::ND; ++d) w[d] = __shfl_sync(NNP_FULL, A.w[d], a) * __shfl_sync(NNP_FULL, B.w[d], b);
            if (ok) M::few_symm(II, tt, cs, w, acc);
        });
    const int n = Ty.ba[tt].n;
#pragma unroll
    for (int f = 0; f < M::NA; ++f) {
        const float s = warp_sum(acc[f]);
        if ((threadIdx.x & 31) == 0 && f < n) Gb[f] = s;
    }
}

// Symmetry functions of the listed blocks (thread-per-atom form).
template <class M>
__device__ void mom_list_symm_body(const MomLists ls, i64 lo, const DevPot *__restrict__ pot,
                                   const float *__restrict__ tab, int fmax, const int *__restrict__ type,
                                   const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
                                   const unsigned short *__restrict__ mom_cnt, float *__restrict__ G)
{
    const MomTab tb = mom_tab(tab, M::T, M::L, fmax);
    const int id = blockIdx.x * NNP_MOM_FEW_THREADS + threadIdx.x, all = gridDim.x * (NNP_MOM_FEW_THREADS / 16);
    for (MomQueue u(ls.wide, ls.n[1], order + lo, id >> 5, all / 2); u.q < u.n; u.next()) {
        const i64 i = u.i;
        const int II = type[i], tt = u.it.y;
        const DevType &Ty = pot->t[II];
        u.ahead();
        mom_wide_symm<M>(nbr + i * cap, mom_cnt + 8 * (i64)u.it.x, Ty, II, tt, tb.a_lo + II * NNP_MOM_MAXD,
                         G + i * gstride + Ty.ba[tt].off_g);
    }
    __syncwarp();
    const int n = ls.n[0], h = threadIdx.x & 15;
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    for (int q = mom_few_first(ls, id >> 4, all); q < n; q += all) {
        const int2 it = ls.few[q];
        const i64 i = order[lo + it.x];
        const int II = type[i];
        const DevType &Ty = pot->t[II];
        mom_few_symm<M>(mask, h, nbr + i * cap, mom_cnt + 8 * (i64)it.x, Ty, II, it.y, tb.a_lo + II * NNP_MOM_MAXD,
                        G + i * gstride + Ty.ba[it.y].off_g);
    }
}

// Forces of the listed blocks of many pairs: per pair the gradient at a.
template <class M>
__device__ __noinline__ void mom_wide_force_body(int block, int nblock, int threads, const MomLists ls, i64 lo,
                                                 const DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
                                                 const int *__restrict__ type, const int *__restrict__ order,
                                                 const float4 *__restrict__ nbr, int cap, int gstride,
                                                 const unsigned short *__restrict__ mom_cnt,
                                                 const float *__restrict__ dEdG, double *__restrict__ F, DevErr *err,
                                                 const int *__restrict__ atom_struct, double *__restrict__ vir)
{
    struct Nbr {
        float u[3], ir, w[M::ND], wd[M::ND];
        float4 rec;
    };
    const MomTab tb = mom_tab(tab, M::T, M::L, fmax);
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (MomQueue u(ls.wide, ls.n[1], order + lo, (block * threads + (int)threadIdx.x) >> 5, nblock * (threads / 32)); u.q < u.n;
         u.next()) {
        const i64 i = u.i;
        const int II = type[i], tt = u.it.y;
        const DevType &Ty = pot->t[II];
        u.ahead();
        const float *a_lo = tb.a_lo + II * NNP_MOM_MAXD, *e = dEdG + i * gstride + Ty.ba[tt].off_g;
        const float4 *src = nbr + i * cap;
        double f[3] = {0, 0, 0}, wv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        float g[3] = {0.f, 0.f, 0.f};
        bool bad = false;
        mom_wide_walk(
            mom_wide<M::T>(mom_cnt + 8 * (i64)u.it.x, tt),
            [&](int k) {
                Nbr o;
                o.rec = src[k];
                MomNbr<M, true> v;
                v.set(o.rec, Ty, a_lo);
                o.u[0] = v.ux;
                o.u[1] = v.uy;
                o.u[2] = v.uz;
                o.ir = v.ir;
#pragma unroll
                for (int d = 0; d < M::ND; ++d) {
                    o.w[d] = v.w[d];
                    o.wd[d] = v.wd[d];
                }
                return o;
            },
            [](const Nbr &v, int q) {
                Nbr o;
#pragma unroll
                for (int x = 0; x < 3; ++x) o.u[x] = __shfl_sync(NNP_FULL, v.u[x], q);
                o.ir = __shfl_sync(NNP_FULL, v.ir, q);
#pragma unroll
                for (int d = 0; d < M::ND; ++d) {
                    o.w[d] = __shfl_sync(NNP_FULL, v.w[d], q);
                    o.wd[d] = __shfl_sync(NNP_FULL, v.wd[d], q);
                }
                o.rec = make_float4(0.f, 0.f, 0.f, __shfl_sync(NNP_FULL, v.rec.w, q));
                return o;
            },
            [&](const Nbr &a, const Nbr &B, int q, bool ok) {
                float b[3], wb[M::ND], none[M::ND];
#pragma unroll
                for (int x = 0; x < 3; ++x) b[x] = __shfl_sync(NNP_FULL, B.u[x], q);
#pragma unroll
                for (int d = 0; d < M::ND; ++d) {
                    wb[d] = __shfl_sync(NNP_FULL, B.w[d], q);
                    none[d] = 0.f;
                }
                const float cs = fmaf(a.u[2], b[2], fmaf(a.u[1], b[1], a.u[0] * b[0]));
                float hc = 0.f, ha = 0.f, hb = 0.f;              // dE/dcos, dE/dr_a
                if (ok) M::few_force(II, tt, cs, e, a.w, a.wd, wb, none, hc, ha, hb);
                const float ta = hc * a.ir, sa = ha - ta * cs;
#pragma unroll
                for (int x = 0; x < 3; ++x) g[x] += fmaf(sa, a.u[x], ta * b[x]);
            },
            [&](const Nbr &A, const Nbr &a, int la, bool first, int lanes) {
                const i64 j = __float_as_int(a.rec.w) & 0x0fffffff;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    for (int o = lanes >> 1; o; o >>= 1) g[x] += __shfl_xor_sync(NNP_FULL, g[x], o);
                    if (first) {
                        bad |= !(fabsf(g[x]) <= 3.402823466e38f);
                        atomicAdd(&F[3 * j + x], (double)g[x]);
                        f[x] += (double)g[x];
                    }
                }
                if (vir) {
                    const double d3[3] = {__shfl_sync(NNP_FULL, A.rec.x, la), __shfl_sync(NNP_FULL, A.rec.y, la),
                                          __shfl_sync(NNP_FULL, A.rec.z, la)};
#pragma unroll
                    for (int x = 0; x < 3; ++x)
#pragma unroll
                        for (int y = 0; y < 3; ++y) wv[3 * x + y] -= first ? (double)g[x] * d3[y] : 0.0;
                }
#pragma unroll
                for (int x = 0; x < 3; ++x) g[x] = 0.f;
            });
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const double s = warp_sum(f[x]);
            if (lane == x) atomicAdd(&F[3 * i + x], -s);
        }
        if (vir) {
            double *ws = vir + 9 * (i64)atom_struct[i];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const double s = warp_sum(wv[q]);
                if (lane == 0) atomicAdd(ws + q, s);
            }
        }
        if (bad) atomicMax(&err->nonfinite, 1);
    }
}

// Forces of the listed blocks of few pairs, 16 lanes each: lane p evaluates pair p,
// then lane h gathers the gradient at neighbour h from the pairs that it is in.
template <class M>
__device__ void mom_few_force_body(int block, int nblock, int threads, const MomLists ls, i64 lo, const DevPot *__restrict__ pot,
                                   const float *__restrict__ tab, int fmax, const int *__restrict__ type,
                                   const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
                                   const unsigned short *__restrict__ mom_cnt, const float *__restrict__ dEdG,
                                   double *__restrict__ F, DevErr *err, const int *__restrict__ atom_struct,
                                   double *__restrict__ vir)
{
    const MomTab tb = mom_tab(tab, M::T, M::L, fmax);
    const int n = ls.n[0], h = threadIdx.x & 15, all = nblock * (threads / 16);
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    for (int q = mom_few_first(ls, (block * threads + (int)threadIdx.x) >> 4, all); q < n; q += all) {
        const int2 it = ls.few[q];
        const i64 i = order[lo + it.x];
        const int II = type[i], tt = it.y;
        const DevType &Ty = pot->t[II];
        const MomFew b = mom_few<M::T>(mom_cnt + 8 * (i64)it.x, tt, h);
        const float *a_lo = tb.a_lo + II * NNP_MOM_MAXD, *e = dEdG + i * gstride + Ty.ba[tt].off_g;
        MomNbr<M, true> v;
        const float4 rv = nbr[i * cap + mom_few_slot(b, h)];
        v.set(rv, Ty, a_lo);
        float ua[3] = {v.ux, v.uy, v.uz}, ub[3], wa[M::ND], wb[M::ND], da[M::ND], db[M::ND];
        float cs = 0.f;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            ub[x] = __shfl_sync(mask, ua[x], b.b, 16);
            ua[x] = __shfl_sync(mask, ua[x], b.a, 16);
            cs = fmaf(ua[x], ub[x], cs);
        }
        const float ia = __shfl_sync(mask, v.ir, b.a, 16), ib = __shfl_sync(mask, v.ir, b.b, 16);
#pragma unroll
        for (int d = 0; d < M::ND; ++d) {
            wa[d] = __shfl_sync(mask, v.w[d], b.a, 16);
            wb[d] = __shfl_sync(mask, v.w[d], b.b, 16);
            da[d] = __shfl_sync(mask, v.wd[d], b.a, 16);
            db[d] = __shfl_sync(mask, v.wd[d], b.b, 16);
        }
        float hc = 0.f, ha = 0.f, hb = 0.f;                      // dE/dcos, dE/dr of a and b
        if (h < b.pairs) M::few_force(II, tt, cs, e, wa, da, wb, db, hc, ha, hb);
        const float ta = hc * ia, sa = ha - ta * cs, tb2 = hc * ib, sb = hb - tb2 * cs;   // dcos/dd_a = (u_b - cos u_a) / r_a
        float ga[3], gb[3], g[3] = {0.f, 0.f, 0.f};              // gradient at a, at b, at neighbour h
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            ga[x] = fmaf(sa, ua[x], ta * ub[x]);
            gb[x] = fmaf(sb, ub[x], tb2 * ua[x]);
        }
        if (b.J == b.K) {
#pragma unroll 1
            for (int t = 0; t < b.no; ++t) {
                const int k = max(h, t), pr = k * (k - 1) / 2 + min(h, t);
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const float qa = __shfl_sync(mask, ga[x], pr, 16), qb = __shfl_sync(mask, gb[x], pr, 16);
                    g[x] += t == h ? 0.f : h < t ? qa : qb;
                }
            }
        } else {
#pragma unroll 1
            for (int t = 0; t < b.np; ++t)
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const float qa = __shfl_sync(mask, ga[x], h + t * b.no, 16);
                    g[x] += h < b.no ? qa : 0.f;
                }
#pragma unroll 1
            for (int t = 0; t < b.no; ++t)
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const float qb = __shfl_sync(mask, gb[x], (h - b.no) * b.no + t, 16);
                    g[x] += h < b.no ? 0.f : qb;
                }
        }
        const bool own = h < b.nn;
        const i64 j = __float_as_int(rv.w) & 0x0fffffff;
        bool bad = false;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            bad |= own && !(fabsf(g[x]) <= 3.402823466e38f);
            if (own) atomicAdd(&F[3 * j + x], (double)g[x]);
            double f = own ? (double)g[x] : 0.0;
#pragma unroll
            for (int r = 8; r; r >>= 1) f += __shfl_xor_sync(mask, f, r, 16);
            if (h == x) atomicAdd(&F[3 * i + x], -f);
        }
        if (vir) {
            double *ws = vir + 9 * (i64)atom_struct[i];
            const double d3[3] = {rv.x, rv.y, rv.z};
#pragma unroll
            for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y) {
                    double w = own ? -(double)g[x] * d3[y] : 0.0;
#pragma unroll
                    for (int r = 8; r; r >>= 1) w += __shfl_xor_sync(mask, w, r, 16);
                    if (h == 0) atomicAdd(ws + 3 * x + y, w);
                }
        }
        if (bad) atomicMax(&err->nonfinite, 1);
    }
}

// ---------------------------------------------------------------- symmetry functions

// G_f of one angular function from S (float2 [tt][pair][l]) and the sum of
// w_d^2, and whether its terms cancel.
template <int L, int NDP>
__device__ __forceinline__ float mom_function(const MomTab &tb, int fu, const float *cf, const float2 *S, const float *w2,
                                             bool &cancels)
{
    const int tt = fu & 0xff, d = (fu >> 8) & 0xff;
    const float2 *s = S + (tt * NDP + (d >> 1)) * (L + 1);
    float g = 0.f, most = 0.f;
#pragma unroll
    for (int l = L; l >= 0; --l) {
        const float c = cf[l * tb.fmax], v = (d & 1) ? s[l].y : s[l].x;
        g = fmaf(c, v, g);
        most = fmaf(fabsf(c), fabsf(v), most);
    }
    const float self = cf[(L + 1) * tb.fmax];
    g = fmaf(-self, *w2, g);
    cancels = g < NNP_MOM_CANCEL * fmaf(self, *w2, most);
    return g;
}

// block tt of row r goes to one of the lists
template <int T>
__device__ __forceinline__ void mom_push(const MomLists &ls, i64 r, int tt, const unsigned short *cnt)
{
    int K = 0;
#pragma unroll
    for (int k = 1; k < T; ++k) K += tt >= k * (k + 1) / 2;
    const int np = mom_pairs(cnt, tt - K * (K + 1) / 2, K);
    if (np <= NNP_MOM_FEW) {
        if (np > 0) ls.few[atomicAdd(ls.n, 1)] = make_int2((int)r, tt);
    } else {
        ls.wide[-(i64)atomicAdd(ls.n + 1, 1)] = make_int2((int)r, tt);
    }
}

// Symmetry functions of atoms order[lo .. hi) and their moments (row idx - lo),
// one warp per atom (NNP::compute_symm, src/nnp/nnp.cpp:350-392): for batches
// too small to fill the GPU with a thread per atom.
// Lane = neighbour for the geometry, the radial functions, the damping factors
// and the Y_lm, which it leaves as a row in shared memory; then lane =
// component for the sums over the rows of each neighbour element (the rows are
// grouped by element), radial functions and w_d as further components.  Sums
// run in two chains per 32-row chunk; that of Y_00, whose terms all have one
// sign and whose rounding sets the error of G, is a shuffle tree.  G may be
// NULL (moments only).
// Bound: shared-memory wavefronts of the rows and instruction issue.
template <class M>
__device__ void mom_symm_body(i64 lo, i64 hi, const DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
                              const int *__restrict__ type, const int *__restrict__ order,
                              const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap, int gstride,
                              float *__restrict__ G, float2 *__restrict__ mom, unsigned short *__restrict__ mom_cnt,
                              const MomLists ls, float *smem)
{
    constexpr int T = M::T, TT = T * (T + 1) / 2, L = M::L, ND = M::ND, NDP = (ND + 1) / 2, NC = mom_comps(L),
                  NR = M::NR, ROW = mom_stage(L, NR, ND), NQ = (NC + NR + ND + 31) / 32,
                  NV = mom_vals(T, ND, L), NS = mom_s_vals(T, ND, L);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *rows = smem + (size_t)warp * mom_symm_floats(T, ND, L, NR, gstride);
    float *W = rows + ((32 * ROW + 3) & ~3);                     // [32][2 NDP]
    float *A = W + 64 * NDP;                                     // [T][NDP][NC] float2
    float *W2 = A + 2 * NV;                                      // [T][NNP_MOM_MAXD]
    float *S = W2 + T * NNP_MOM_MAXD;
    float *Gs = S + ((NS * 2 + 3) & ~3);
    unsigned short *cnt = reinterpret_cast<unsigned short *>(Gs + gstride);   // [8]
    const DevPot &P = *pot;
    const MomTab tb = mom_tab(tab, T, L, fmax);
    float nl[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) nl[q] = (lane + 32 * q < NC) ? tb.norm[lane + 32 * q] : 0.f;
    // the padding component and unused radial slots of the rows stay 0
    for (int k = lane; k < 32 * ROW; k += 32) rows[k] = 0.f;
    __syncwarp();
    for (i64 idx = lo + blockIdx.x * (i64)NNP_MOM_SYMM_WARPS + warp; idx < hi; idx += (i64)gridDim.x * NNP_MOM_SYMM_WARPS) {
        const i64 i = order[idx];
        const int II = type[i], n = nbr_cnt[i];
        if ((unsigned)II >= (unsigned)T) continue;               // type out of range (reported by the call)
        const DevType &Ty = P.t[II];
        const float4 *src = nbr + i * cap;
        for (int k = lane; 4 * k < 2 * NV + T * NNP_MOM_MAXD; k += 32)
            reinterpret_cast<float4 *>(A)[k] = make_float4(0.f, 0.f, 0.f, 0.f);   // A, W2
        for (int k = lane; 4 * k < gstride + 4; k += 32)          // G row, counts
            reinterpret_cast<float4 *>(Gs)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        for (int kb = 0; kb < n; kb += 32) {
            int t = T;
            float w[2 * NDP];
#pragma unroll
            for (int d = 0; d < 2 * NDP; ++d) w[d] = 0.f;
            if (kb + lane < n) {
                const float4 e = src[kb + lane];
                t = (int)((unsigned)__float_as_int(e.w) >> 28);
                MomNbr<M, false> v;
                v.set(e, Ty, tb.a_lo + II * NNP_MOM_MAXD);
                float *row = rows + lane * ROW;
                mom_harmonics<L>(v.ux, v.uy, v.uz, row);
                M::radial_row(II, t, v.r, v.fc, row + NC);
#pragma unroll
                for (int d = 0; d < 2 * NDP; ++d) {
                    if (d < ND) row[NC + NR + d] = w[d] = v.w[d < ND ? d : 0];
                    W[lane * 2 * NDP + d] = w[d];
                }
            }
            __syncwarp();
            int k0 = 0;
#pragma unroll 1
            for (int J = 0; J < T; ++J) {
                const int nj = __popc(__ballot_sync(NNP_FULL, t == J));
                if (nj == 0) continue;
                if (lane == 0) cnt[J] += nj;
                f32x2 acc[2][NQ][NDP];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
#pragma unroll
                        for (int p = 0; p < NDP; ++p) acc[h][q][p] = 0ull;
                auto add = [&](int h, int k) {
                    const float *row = rows + k * ROW + lane;
                    f32x2 f[NDP];
#pragma unroll
                    for (int p = 0; p < NDP; ++p) f[p] = reinterpret_cast<const f32x2 *>(W)[k * NDP + p];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        // (the last group's lanes past the row read the next row or W; their sums are not used)
                        const f32x2 y = dup2(row[32 * q]);
                        const bool any_rad = 32 * q + 31 >= NC && 32 * q < NC + NR;
                        const bool rad = any_rad && lane + 32 * q >= NC && lane + 32 * q < NC + NR;
#pragma unroll
                        for (int p = 0; p < NDP; ++p) {
                            const f32x2 g = rad ? 0x3f8000003f800000ull : f[p];
                            acc[h][q][p] = fma2(y, g, acc[h][q][p]);
                        }
                    }
                };
                int k = k0;
#pragma unroll 2
                for (; k + 1 < k0 + nj; k += 2) {
                    add(0, k);
                    add(1, k + 1);
                }
                if (k < k0 + nj) add(0, k);
                k0 += nj;
                const DevBlockR B = Ty.br[J];
#pragma unroll
                for (int p = 0; p < NDP; ++p) {
                    const float t0 = warp_sum(t == J ? w[2 * p] : 0.f), t1 = warp_sum(t == J ? w[2 * p + 1] : 0.f);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const int c = lane + 32 * q;
                        float a0, a1, b0, b1;
                        up2(acc[0][q][p], a0, a1);
                        up2(acc[1][q][p], b0, b1);
                        a0 += b0;
                        a1 += b1;
                        if (c == 0) {                            // Y_00 = 1
                            a0 = t0;
                            a1 = t1;
                        }
                        if (c < NC) {
                            float2 *dst = reinterpret_cast<float2 *>(A) + (J * NDP + p) * NC + c;
                            *dst = make_float2(fmaf(a0, nl[q], dst->x), fmaf(a1, nl[q], dst->y));
                        } else if (c < NC + NR) {
                            if (p == 0 && c - NC < B.n) Gs[B.off_g + c - NC] += a0;
                        } else if (c < NC + NR + ND) {
                            const int d = c - NC - NR;
                            if ((d >> 1) == p) W2[J * NNP_MOM_MAXD + d] += (d & 1) ? a1 : a0;
                        }
                    }
                }
            }
            __syncwarp();
        }
        __syncwarp();
        unsigned long long mask;                                 // blocks that are summed over pairs
        {
            // S^{JK}_{l,d}: lane = (l, pair of damping factors, element pair), largest l first
            for (int s = lane; s < NS; s += 32) {
                const int l = L - s / (TT * NDP), rem = s % (TT * NDP), p = rem / TT, tt = rem % TT;
                int K = 0;
#pragma unroll
                for (int k = 1; k < T; ++k) K += tt >= k * (k + 1) / 2;
                const int J = tt - K * (K + 1) / 2;
                const f32x2 *a = reinterpret_cast<const f32x2 *>(A) + (J * NDP + p) * NC;
                const f32x2 *b = reinterpret_cast<const f32x2 *>(A) + (K * NDP + p) * NC;
                f32x2 s0 = mul2(a[l], b[l]), s1 = 0ull;
#pragma unroll
                for (int m = 1; m <= L; ++m) {
                    if (m <= l) {
                        const int c = mom_base(L, m) + 2 * (l - m);
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(a + c);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(b + c);
                        s0 = fma2(x.x, y.x, s0);
                        s1 = fma2(x.y, y.y, s1);
                    }
                }
                reinterpret_cast<f32x2 *>(S)[(tt * NDP + p) * (L + 1) + l] = add2(s0, s1);
            }
            __syncwarp();
            // G: lane = angular function
            const int na = Ty.n_input - Ty.n_input_r;
            unsigned long long list = 0, few = 0, none = 0;
            for (int f = lane; f < na; f += 32) {
                const int fu = tb.fun[II * fmax + f];
                bool cancels;
                Gs[Ty.n_input_r + f] = mom_function<L, NDP>(tb, fu, tb.coef + (i64)II * (L + 2) * fmax + f,
                                                             reinterpret_cast<const float2 *>(S),
                                                             W2 + ((fu >> 16) & 0xff) * NNP_MOM_MAXD + ((fu >> 8) & 0xff),
                                                             cancels);
                if (cancels) list |= 1ull << (fu & 0xff);
            }
            list = (unsigned long long)__reduce_or_sync(NNP_FULL, (unsigned)(list >> 32)) << 32 |
                   __reduce_or_sync(NNP_FULL, (unsigned)list);
            __syncwarp();
            for (int K = 0, tt = 0; K < T; ++K)
                for (int J = 0; J <= K; ++J, ++tt) {
                    const int np = mom_pairs(cnt, J, K);
                    if (np == 0) none |= 1ull << tt;
                    else if (np <= NNP_MOM_FEW) few |= 1ull << tt;
                }
            mask = none | list;
            for (unsigned long long m = G ? list & ~none & ~few : 0; m; m &= m - 1) {
                const int tt = __ffsll(m) - 1;
                mom_wide_symm<M>(src, cnt, Ty, II, tt, tb.a_lo + II * NNP_MOM_MAXD, Gs + Ty.ba[tt].off_g);
            }
            if (none)
                for (int f = lane; f < na; f += 32)
                    if (none >> (tb.fun[II * fmax + f] & 0xff) & 1) Gs[Ty.n_input_r + f] = 0.f;
            // blocks of few pairs, one per half warp
            few = G ? few & list : 0;
            while (few) {
                const int t0 = __ffsll(few) - 1;
                few &= few - 1;
                const int t1 = few ? __ffsll(few) - 1 : -1, tt = lane < 16 ? t0 : t1;
                few &= few - 1;
                if (tt >= 0)
                    mom_few_symm<M>(0xffffu << (lane & 16), lane & 15, src, cnt, Ty, II, tt, tb.a_lo + II * NNP_MOM_MAXD,
                                    Gs + Ty.ba[tt].off_g);
            }
            __syncwarp();
            for (int k = lane; G && 4 * k < gstride; k += 32)
                reinterpret_cast<float4 *>(G + i * gstride)[k] = reinterpret_cast<const float4 *>(Gs)[k];
        }
        {
            const i64 r = idx - lo;
            for (int k = lane; k < NV; k += 32) mom[mom_at(r, k, NV, NNP_MOM_SH_W)] = reinterpret_cast<const float2 *>(A)[k];
            if (lane < 8) mom_cnt[8 * r + lane] = cnt[lane];
            if (lane == 0) ls.mask[r] = mask;
            for (int tt = lane; tt < TT; tt += 32) if (mask >> tt & 1) mom_push<T>(ls, r, tt, cnt);
        }
        __syncwarp();
    }
}

// Angular functions of a thread's atom from S and the sums of w_d^2 (entries
// BT apart): G_f = sum_l c_l S_l - self (c and self as in dE/dA: half of them
// for J == K), self = -wscale sum w_d^2.  Blocks that are summed over pairs are
// written too and replaced.  `mask` has those without pairs (0 here); with MARK it
// gets those whose terms cancel.  The absolute sum of the terms is taken as that of
// the sums over even and over odd l (with J == K, S_l >= 0 and the coefficients'
// signs are those of lambda^l, so it is the absolute sum; J and K to one side or
// opposite sides likewise), and at least the term of l = 0 (J and K at right angles):
// no further sums (with sums of |c_l S_l| the stage of 1.09 M atoms took 2.01 ms
// instead of 1.99).
template <class M, bool MARK>
__device__ __forceinline__ unsigned long long mom_functions_thread(const MomTab &tb, int fmax, int II, const DevType &Ty,
                                                                   unsigned long long mask, const f32x2 *S, const f32x2 *W2,
                                                                   float wscale, float *Gi)
{
    constexpr int T = M::T, L = M::L, NDP = (M::ND + 1) / 2, DL = mom_dl(L), BT = NNP_MOM_THREADS;
#pragma unroll 1
    for (int K = 0, tt = 0; K < T; ++K)
#pragma unroll 1
        for (int J = 0; J <= K; ++J, ++tt) {
            const bool none = mask >> tt & 1;
            const int off = Ty.ba[tt].off_g, bn = Ty.ba[tt].n, f0 = II * fmax + off - Ty.n_input_r;
            const ulonglong2 *cf = reinterpret_cast<const ulonglong2 *>(tb.dcoef + (i64)f0 * DL);
            const float h = J == K ? 0.5f : 1.f;
            bool cancels = false;
            f32x2 st[DL];                                    // S, -sum of w_d^2
#pragma unroll
            for (int l = 0; l < DL; ++l) st[l] = 0ull;
#pragma unroll 2
            for (int f = 0; f < bn; ++f) {
                const int p = NDP > 1 ? (tb.fun[f0 + f] >> 9) & 0x7f : 0;
                if (NDP > 1 || f == 0) {
#pragma unroll
                    for (int l = 0; l <= L; ++l) st[l] = S[((tt * NDP + p) * (L + 1) + l) * BT];
                    st[L + 1] = mul2(W2[(J * NDP + p) * BT], dup2(wscale));
                }
                f32x2 c[DL], ge = 0ull, go = 0ull;               // even and odd l
#pragma unroll
                for (int l = 0; l < DL; l += 2) {
                    const ulonglong2 v = __ldg(cf + f * (DL / 2) + l / 2);
                    c[l] = v.x;
                    c[l + 1] = v.y;
                }
#pragma unroll
                for (int l = L; l >= 0; --l) {
                    if (l & 1) go = fma2(c[l], st[l], go);
                    else ge = fma2(c[l], st[l], ge);
                }
                const f32x2 self = mul2(c[L + 1], st[L + 1]);    // at most 0
                float e0, e1, g0, g1;
                up2(ge, e0, e1);
                up2(add2(fma2(c[L + 1], st[L + 1], ge), go), g0, g1);
                if (MARK) {
                    float o0, o1, s0, s1, z0, z1;
                    up2(go, o0, o1);
                    up2(self, s0, s1);
                    up2(mul2(c[0], st[0]), z0, z1);
                    cancels |= g0 + g1 < NNP_MOM_CANCEL * (fmaxf(fabsf(e0 + e1) + fabsf(o0 + o1), z0 + z1) - (s0 + s1));
                }
                if (Gi) Gi[off + f] = none ? 0.f : h * (g0 + g1);
            }
            if (MARK && cancels) mask |= 1ull << tt;
        }
    return mask;
}

// The same with one thread per atom: the moments of one neighbour element and
// damping pair are the thread's registers (81 packed pairs for L = 8) while it
// walks that element's segment of its list, so nothing is staged, exchanged or
// reduced; the finished moments go to mom, from which the thread forms S
// (through shared memory, entry-major) and G.  Lanes differ in the length of a
// segment (on average 21 of 32 worked on the batched workload), so the atoms are
// visited in the order of their neighbour counts (run_len_order: 29 of 32).
// Y_00's sum keeps its rounding errors in a second register (see above).
// Bound: latency of the phases between the segments and FP32 issue at 8 warps
// per SM (registers).  1.09 M atoms: 2.66 ms; lines of the list prefetched 2.43;
// sorted visits 2.28; moments 32 rows interleaved 2.13; G from contiguous
// coefficients, norms as literals 1.97 (the sort and the blocks of few pairs
// included).
template <class M>
__device__ void mom_symm_thread_body(i64 lo, i64 hi, const DevPot *__restrict__ pot, const float *__restrict__ tab,
                                     int fmax, const int *__restrict__ type, const int *__restrict__ order,
                                     const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap,
                                     int gstride, float *__restrict__ G, float2 *mom,
                                     unsigned short *__restrict__ mom_cnt, const MomLists ls, float *smem)
{
    constexpr int T = M::T, TT = T * (T + 1) / 2, L = M::L, ND = M::ND, NDP = (ND + 1) / 2, NC = mom_comps(L),
                  NR = M::NR, NV = mom_vals(T, ND, L), NS = mom_s_vals(T, ND, L), BT = NNP_MOM_THREADS;
    f32x2 *S = reinterpret_cast<f32x2 *>(smem) + threadIdx.x;    // [NS][BT]
    f32x2 *W2 = S + NS * BT;                                     // [T][NDP][BT]
    const DevPot &P = *pot;
    const MomTab tb = mom_tab(tab, T, L, fmax);
    for (i64 idx = lo + blockIdx.x * (i64)BT + threadIdx.x; idx < hi; idx += (i64)gridDim.x * BT) {
        const i64 i = order[idx], r = idx - lo;
        const int II = type[i];
        if ((unsigned)II >= (unsigned)T) continue;               // type out of range (reported by the call)
        const int n = nbr_cnt[i];
        const DevType &Ty = P.t[II];
        const float4 *src = nbr + i * cap;
        float *Gi = G ? G + i * gstride : nullptr;
        unsigned short *cnt = mom_cnt + 8 * r;
#pragma unroll 1
        for (int p = 0; p < NDP; ++p) {
            int k = 0;
            float4 e = n > 0 ? src[0] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
#pragma unroll 1
            for (int J = 0; J < T; ++J) {
                const int k0 = k;
                f32x2 acc[NC], c00 = 0ull, ww = 0ull;
                float rad[NR];
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[c] = 0ull;
#pragma unroll
                for (int f = 0; f < NR; ++f) rad[f] = 0.f;
#pragma unroll 1
                while ((int)((unsigned)__float_as_int(e.w) >> 28) == J) {
                    MomNbr<M, false> v;
                    v.set(e, Ty, tb.a_lo + II * NNP_MOM_MAXD);
                    ++k;
                    mom_prefetch(src + min(k + 6, n - 1));
                    e = k < n ? src[k] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
                    f32x2 cw = pk2(v.w[0], ND > 1 ? v.w[ND > 1 ? 1 : 0] : 0.f);
                    if (NDP > 1 && p > 0) cw = pk2(v.w[ND > 2 ? 2 : 0], ND > 3 ? v.w[ND > 3 ? 3 : 0] : 0.f);
                    ww = fma2(cw, cw, ww);
                    {                                            // two-sum of acc[0] and w
                        const f32x2 neg = dup2(-1.f);
                        const f32x2 s = add2(acc[0], cw), bb = fma2(neg, acc[0], s);
                        c00 = add2(c00, add2(fma2(neg, fma2(neg, bb, s), acc[0]), fma2(neg, bb, cw)));
                        acc[0] = s;
                    }
                    const f32x2 x2 = dup2(v.ux), y2 = dup2(v.uy), ny2 = dup2(-v.uy);
                    f32x2 sw = 0ull;
#pragma unroll
                    for (int m = 0; m <= L; ++m) {               // (cw, sw) = w Re/Im (x + i y)^m
                        float q0 = 1.f, q1 = 0.f;
#pragma unroll
                        for (int l = m; l <= L; ++l) {
                            const f32x2 q2 = dup2(q0);
                            if (m == 0) {
                                if (l > 0) acc[l] = fma2(q2, cw, acc[l]);
                            } else {
                                const int c = mom_base(L, m > 0 ? m : 1) + 2 * (l - m);
                                acc[c] = fma2(q2, cw, acc[c]);
                                acc[c + 1] = fma2(q2, sw, acc[c + 1]);
                            }
                            const float t = (l == m) ? v.uz * q0 : fmaf(v.uz, q0, -mom_beta(l, m) * q1);
                            q1 = q0;
                            q0 = t;
                        }
                        const f32x2 c = cw;
                        cw = m == 0 ? mul2(c, x2) : fma2(sw, ny2, mul2(c, x2));
                        sw = m == 0 ? mul2(c, y2) : fma2(sw, x2, mul2(c, y2));
                    }
                    if (NDP == 1 || p == 0) {
                        float rv[NR];
#pragma unroll
                        for (int f = 0; f < NR; ++f) rv[f] = 0.f;
                        M::radial_row(II, J, v.r, v.fc, rv);
#pragma unroll
                        for (int f = 0; f < NR; ++f) rad[f] += rv[f];
                    }
                }
                cnt[J] = (unsigned short)(k - k0);
                acc[0] = add2(acc[0], c00);
                f32x2 *dst = reinterpret_cast<f32x2 *>(mom) + mom_at(r, (J * NDP + p) * NC, NV, NNP_MOM_SH_T);
#pragma unroll
                for (int c = 0; c < NC; ++c) dst[c << NNP_MOM_SH_T] = mul2(acc[c], dup2(M::norm(c)));
                W2[(J * NDP + p) * BT] = ww;
                if (G && p == 0) {
                    const DevBlockR B = Ty.br[J];
#pragma unroll
                    for (int f = 0; f < NR; ++f)
                        if (f < B.n) Gi[B.off_g + f] = rad[f];
                }
            }
        }
        const f32x2 *a = reinterpret_cast<const f32x2 *>(mom) + mom_at(r, 0, NV, NNP_MOM_SH_T);
#pragma unroll 1
        for (int p = 0; p < NDP; ++p)
#pragma unroll
            for (int l = 0; l <= L; ++l) {
                f32x2 s[TT];
#pragma unroll
                for (int m = 0; m <= l; ++m)
#pragma unroll
                    for (int h = 0; h < (m ? 2 : 1); ++h) {
                        const int c = m == 0 ? l : mom_base(L, m > 0 ? m : 1) + 2 * (l - m) + h;
                        f32x2 v[T];
#pragma unroll
                        for (int J = 0; J < T; ++J) v[J] = a[((J * NDP + p) * NC + c) << NNP_MOM_SH_T];
#pragma unroll
                        for (int K = 0; K < T; ++K)
#pragma unroll
                            for (int J = 0; J <= K; ++J) {
                                const int tt = K * (K + 1) / 2 + J;
                                s[tt] = m == 0 ? mul2(v[J], v[K]) : fma2(v[J], v[K], s[tt]);
                            }
                    }
#pragma unroll
                for (int tt = 0; tt < TT; ++tt) S[((tt * NDP + p) * (L + 1) + l) * BT] = s[tt];
            }
        unsigned long long mask = 0;
        for (int K = 0, tt = 0; K < T; ++K)
            for (int J = 0; J <= K; ++J, ++tt)
                if (mom_pairs(cnt, J, K) == 0) mask |= 1ull << tt;
        mask = mom_functions_thread<M, true>(tb, fmax, II, Ty, mask, S, W2, -1.f, Gi);
        ls.mask[r] = mask;
#pragma unroll
        for (int tt = 0; tt < TT; ++tt)
            if (mask >> tt & 1) mom_push<T>(ls, r, tt, cnt);
        for (int f = Ty.n_input; G && f < gstride; ++f) Gi[f] = 0.f;
    }
}

// ---------------------------------------------------------------- forces

// Forces from the moments (NNP::compute_force, src/nnp/nnp.cpp:412-476): a
// warp takes NA atoms (2 when there are enough atoms: 45 neighbours leave the
// second of two 32-lane passes half empty, the 90 of two atoms fill three;
// the virial takes NA = 1).
// It forms B of each atom from its moments and dE/dG, then lane = neighbour
// evaluates sum_d w_d sum_lm B Y_lm and its gradient with the broadcast B (two
// damping factors per 8-byte half, cos and sin parts per 16-byte load, packed
// FP32 arithmetic), adds the radial terms and scatters dE_i/dd_j in FP64 as
// force_body does.  Here Q_lm = d^m P_l / dz^m, so that dQ_lm/dz = Q_{l,m+1}
// needs no factor.  With NA = 1 the launch's first thread blocks take the listed blocks
// of pairs (a small call is a chain of launches; behind the others they were a tail).
// Bound: instruction issue (FP32 pipe).
template <class M, int NA>
__device__ void mom_force_body(int block, int nblock, i64 lo, i64 hi, const DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
                               const float2 *__restrict__ rpar, const int *__restrict__ type,
                               const int *__restrict__ order, const float4 *__restrict__ nbr,
                               const int *__restrict__ nbr_cnt, int cap, int gstride, const float *__restrict__ dEdG,
                               const float2 *__restrict__ mom, int msh, const unsigned long long *__restrict__ mom_mask,
                               double *__restrict__ F, DevErr *err, const int *__restrict__ atom_struct,
                               double *__restrict__ vir, float *smem)
{
    constexpr int T = M::T, TT = T * (T + 1) / 2, L = M::L, ND = M::ND, NDP = (ND + 1) / 2, NC = mom_comps(L),
                  NV = mom_vals(T, ND, L), NS = mom_s_vals(T, ND, L), LA = NA == 1 ? 0 : 1;
    static_assert(NA == 1 || NA == 2, "atoms per warp");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = mom_force_floats(T, ND, L, gstride);         // floats per atom
    float *base = smem + (size_t)warp * NA * per;
    const int oD = 2 * NV, oD1 = oD + ((2 * NS + 3) & ~3), oE = oD1 + T * NNP_MOM_MAXD;
    const DevPot &P = *pot;
    const MomTab tb = mom_tab(tab, T, L, fmax);
    const i64 step = (i64)nblock * NNP_MOM_FORCE_WARPS * NA;
    for (i64 idx = lo + (block * (i64)NNP_MOM_FORCE_WARPS + warp) * NA; idx < hi; idx += step) {
        // atom lane & (NA - 1) of the group (II = T: none)
        const int al = lane & (NA - 1);
        i64 i_l = 0;
        int II_l = T, n_l = 0;
        if (idx + al < hi) {
            i_l = order[idx + al];
            const int t = type[i_l];
            if ((unsigned)t < (unsigned)T) {                     // else out of range (reported by the call)
                II_l = t;
                n_l = nbr_cnt[i_l];
            }
        }
        const int n0 = __shfl_sync(NNP_FULL, n_l, 0), n1 = NA == 2 ? __shfl_sync(NNP_FULL, n_l, NA - 1) : 0;
        const i64 i0 = __shfl_sync(NNP_FULL, i_l, 0), i1 = __shfl_sync(NNP_FULL, i_l, NA - 1);
        const int II0 = __shfl_sync(NNP_FULL, II_l, 0), II1 = __shfl_sync(NNP_FULL, II_l, NA - 1);
        const i64 row = idx - lo;
        for (int k = lane; k < gstride; k += 32) {
            base[oE + k] = dEdG[i0 * gstride + k];
            if (NA == 2) base[per + oE + k] = dEdG[i1 * gstride + k];   // (no second atom: atom 0's row, not used)
        }
        __syncwarp();
        // D^{JK}_{l,d} = sum_f e_f c_{f,l} [1 + (J == K)], and the self terms
        if (II_l < T) {
            float *mine = base + al * per;
            const float *e = mine + oE;
            const DevType &Ty = P.t[II_l];
            const unsigned long long mask = mom_mask[row + al];
            for (int s = lane >> LA; s < TT * NDP * (L + 2); s += 32 / NA) {
                const int l = s % (L + 2), rem = s / (L + 2), p = rem % NDP, tt = rem / NDP;
                int K = 0;
#pragma unroll
                for (int k = 1; k < T; ++k) K += tt >= k * (k + 1) / 2;
                const int J = tt - K * (K + 1) / 2;
                const int bn = Ty.ba[tt].n, off = Ty.ba[tt].off_g, f0 = off - Ty.n_input_r;
                float s0 = 0.f, s1 = 0.f;
                if (!(mask >> tt & 1)) {
                    const float *cf = tb.coef + ((i64)II_l * (L + 2) + l) * fmax + f0;
                    const int *fu = tb.fun + II_l * fmax + f0;
#pragma unroll 2
                    for (int f = 0; f < bn; ++f) {
                        const int d = (fu[f] >> 8) & 0xff;
                        const float v = (NDP == 1 || (d >> 1) == p) ? cf[f] * e[off + f] : 0.f;
                        s0 += (d & 1) ? 0.f : v;
                        s1 += (d & 1) ? v : 0.f;
                    }
                }
                if (J == K) {
                    s0 *= 2.f;
                    s1 *= 2.f;
                }
                if (l <= L) {
                    reinterpret_cast<float2 *>(mine + oD)[(tt * NDP + p) * (L + 1) + l] = make_float2(s0, s1);
                } else if (J == K) {
                    mine[oD1 + J * NNP_MOM_MAXD + 2 * p] = s0;
                    mine[oD1 + J * NNP_MOM_MAXD + 2 * p + 1] = s1;
                }
            }
        }
        __syncwarp();
        if (II_l < T) {
            float *mine = base + al * per;
            const f32x2 *src = reinterpret_cast<const f32x2 *>(mom) + mom_at(row + al, 0, NV, msh);
#pragma unroll 2
            for (int c = lane >> LA; c < NC; c += 32 / NA) {
                const int l = tb.deg[c];
                const f32x2 nn = dup2(tb.fnorm[c]);
#pragma unroll
                for (int p = 0; p < NDP; ++p) {
                    f32x2 a[T];
#pragma unroll
                    for (int K = 0; K < T; ++K) a[K] = __ldg(src + ((i64)((K * NDP + p) * NC + c) << msh));
#pragma unroll
                    for (int J = 0; J < T; ++J) {
                        f32x2 b = 0ull;
#pragma unroll
                        for (int K = 0; K < T; ++K) {
                            const int tt = J > K ? J * (J + 1) / 2 + K : K * (K + 1) / 2 + J;
                            b = fma2(reinterpret_cast<const f32x2 *>(mine + oD)[(tt * NDP + p) * (L + 1) + l], a[K], b);
                        }
                        reinterpret_cast<f32x2 *>(mine)[(J * NDP + p) * NC + c] = mul2(b, nn);
                    }
                }
            }
        }
        __syncwarp();
        double f0[3] = {0, 0, 0}, f1[3] = {0, 0, 0};
        double wv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        bool bad = false;
        for (int q = lane; q < n0 + n1; q += 32) {
            const bool sec = NA == 2 && q >= n0;                 // neighbour of the second atom
            const i64 i = sec ? i1 : i0;
            const int II = sec ? II1 : II0;
            const float *mine = base + (sec ? per : 0);
            const float4 rec = nbr[i * cap + (sec ? q - n0 : q)];
            const int jt = __float_as_int(rec.w);
            const int t = (int)((unsigned)jt >> 28);
            const DevType &Ty = P.t[II];
            MomNbr<M, true> v;
            v.set(rec, Ty, tb.a_lo + II * NNP_MOM_MAXD);
            f32x2 V[NDP], X[NDP], Y[NDP], Z[NDP];
            f32x2 q0[L + 2];
            mom_polys<L, 0>(v.uz, q0);
            mom_gradient<L, NDP, 0>(reinterpret_cast<const ulonglong2 *>(mine + t * (NDP * NC * 2)), v.ux, v.uy, v.uz, q0,
                                    1.f, 0.f, 0.f, 0.f, V, X, Y, Z);
            // radial terms
            const DevBlockR Br = Ty.br[t];
            const float *e = mine + oE;
            float fc = v.fc[0], fd = v.fd[0];
#pragma unroll
            for (int c = 1; c < M::NCUT; ++c)
                if (Br.cut == c) {
                    fc = v.fc[c];
                    fd = v.fd[c];
                }
            float gr = 0.f;
            if (!M::radial_force(II, t, v.r, fc, fd, e + Br.off_g, gr)) {
                for (int f = 0; f < Br.n; ++f) {
                    const float2 q2 = rpar[Br.par + f];
                    float val, der;
                    radial_fd(Br.form, v.r, q2.x, q2.y, fc, fd, val, der);
                    gr = fmaf(e[Br.off_g + f], der, gr);
                }
            }
            float gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
            for (int p = 0; p < NDP; ++p) {
                float v0, v1, x0, x1, y0, y1, z0, z1;
                up2(V[p], v0, v1);
                up2(X[p], x0, x1);
                up2(Y[p], y0, y1);
                up2(Z[p], z0, z1);
                {
                    const float w = v.w[2 * p], dw = v.wd[2 * p];
                    gr = fmaf(fmaf(-mine[oD1 + t * NNP_MOM_MAXD + 2 * p], w, v0), dw, gr);
                    gx = fmaf(w, x0, gx);
                    gy = fmaf(w, y0, gy);
                    gz = fmaf(w, z0, gz);
                }
                if (2 * p + 1 < ND) {
                    const float w = v.w[2 * p + 1 < ND ? 2 * p + 1 : 0], dw = v.wd[2 * p + 1 < ND ? 2 * p + 1 : 0];
                    gr = fmaf(fmaf(-mine[oD1 + t * NNP_MOM_MAXD + 2 * p + 1], w, v1), dw, gr);
                    gx = fmaf(w, x1, gx);
                    gy = fmaf(w, y1, gy);
                    gz = fmaf(w, z1, gz);
                }
            }
            // dE/dd = u dE/dr + (I - u u^T) dE/du / r
            const float pr = gr - v.ir * (gx * v.ux + gy * v.uy + gz * v.uz);
            const float h[3] = {fmaf(gx, v.ir, pr * v.ux), fmaf(gy, v.ir, pr * v.uy), fmaf(gz, v.ir, pr * v.uz)};
            const i64 j = jt & 0x0fffffff;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                bad |= !(fabsf(h[x]) <= 3.402823466e38f);
                atomicAdd(&F[3 * j + x], (double)h[x]);
                f0[x] += (double)(sec ? 0.f : h[x]);
                if (NA == 2) f1[x] += (double)(sec ? h[x] : 0.f);
            }
            if (NA == 1 && vir) {
                // virial W_ab = -sum_k g_a d_b (see force_body)
                const double d3[3] = {rec.x, rec.y, rec.z};
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                    for (int y = 0; y < 3; ++y) wv[3 * x + y] -= (double)h[x] * d3[y];
            }
        }
        __syncwarp();
        if (NA == 1) {
#pragma unroll
            for (int x = 0; x < 3; ++x) f0[x] = warp_sum(f0[x]);
            if (lane < 3 && II0 < T) atomicAdd(&F[3 * i0 + lane], lane == 0 ? -f0[0] : lane == 1 ? -f0[1] : -f0[2]);
        } else {
            // lanes below 16 keep the first atom's sums, the others the second's
            const bool up = lane >= 16;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                double s = (up ? f1[x] : f0[x]) + __shfl_xor_sync(NNP_FULL, up ? f0[x] : f1[x], 16);
#pragma unroll
                for (int o = 8; o; o >>= 1) s += __shfl_xor_sync(NNP_FULL, s, o);
                f0[x] = s;
            }
            const int x = lane & 15;
            if (x < 3 && (up ? II1 : II0) < T)
                atomicAdd(&F[3 * (up ? i1 : i0) + x], x == 0 ? -f0[0] : x == 1 ? -f0[1] : -f0[2]);
        }
        if (vir && NA == 1) {
#pragma unroll
            for (int q = 0; q < 9; ++q) wv[q] = warp_sum(wv[q]);
            if (lane == 0 && II0 < T) {
                double *ws = vir + 9 * (i64)atom_struct[i0];
#pragma unroll
                for (int q = 0; q < 9; ++q) atomicAdd(ws + q, wv[q]);
            }
        }
        if (__any_sync(NNP_FULL, bad) && lane == 0) atomicMax(&err->nonfinite, 1);
        __syncwarp();
    }
}

// dE/dG of a segment's radial functions in the threads' columns of shared memory
struct MomStrided {
    const float *p;
    __device__ __forceinline__ float operator[](int f) const { return p[f * NNP_MOM_THREADS]; }
};

// One neighbour's sum_lm B Y_lm and its gradient with B in registers (b, scaled
// by gnorm), both damping factors side by side.  r_n^m = d^m P_l / dz^m up to a
// factor, n = l - m, scaled so that dr_n^m/dz = r_(n-1)^(m+1):
//   r_(n+1) = z / (n + 1) r_n - beta / (n (n + 1)) r_(n-1),  r_0 = 1.
// Row m serves the values of order m and the z slopes of order m - 1; the sums
// over m are Horner's scheme in x - i y (f, its derivative g, and h for z).
template <int L, int m>
__device__ __forceinline__ void mom_gradient_regs(const f32x2 *b, float z, const float *zn, f32x2 x2, f32x2 y2, f32x2 ny2,
                                                  f32x2 &fr, f32x2 &fi, f32x2 &gr, f32x2 &gi, f32x2 &hr, f32x2 &hi)
{
    f32x2 C = 0ull, S = 0ull, Cz = 0ull, Sz = 0ull;
    float q0 = 1.f, q1 = 0.f;
#pragma unroll
    for (int l = m; l <= L; ++l) {
        const f32x2 q2 = dup2(q0);
        const int n = l - m;
        if constexpr (m == 0) {
            C = n == 0 ? b[0] : fma2(q2, b[l], C);
        } else {
            const f32x2 *bm = b + mom_base(L, m) + 2 * n;
            C = n == 0 ? bm[0] : fma2(q2, bm[0], C);
            S = n == 0 ? bm[1] : fma2(q2, bm[1], S);
            if constexpr (m == 1) {
                Cz = n == 0 ? b[l] : fma2(q2, b[l], Cz);
            } else {
                const f32x2 *bp = b + mom_base(L, m - 1) + 2 * (n + 1);
                Cz = n == 0 ? bp[0] : fma2(q2, bp[0], Cz);
                Sz = n == 0 ? bp[1] : fma2(q2, bp[1], Sz);
            }
        }
        const float t = n == 0 ? z : fmaf(zn[n], q0, (-mom_beta(l, m) / (float)(n * (n + 1) > 0 ? n * (n + 1) : 1)) * q1);
        q1 = q0;
        q0 = t;
    }
    if constexpr (m == L) {
        fr = C;
        fi = S;
        gr = gi = 0ull;
        hr = Cz;
        hi = Sz;
    } else {
        f32x2 t = fma2(gr, x2, fma2(gi, y2, fr));
        gi = fma2(gi, x2, fma2(gr, ny2, fi));
        gr = t;
        t = fma2(fr, x2, fma2(fi, y2, C));
        if constexpr (m > 0) fi = fma2(fi, x2, fma2(fr, ny2, S));
        fr = t;
        if constexpr (m > 0) {
            t = fma2(hr, x2, fma2(hi, y2, Cz));
            if constexpr (m > 1) hi = fma2(hi, x2, fma2(hr, ny2, Sz));
            hr = t;
        }
    }
    if constexpr (m > 0) mom_gradient_regs<L, m - 1>(b, z, zn, x2, y2, ny2, fr, fi, gr, gi, hr, hi);
}

// Forces with one thread per atom (at most two damping factors): B of one
// neighbour element is the thread's registers while it walks that element's
// segment of its list, so nothing of it is read again per neighbour (the warp
// form's loads of B kept the shared-memory pipe 77 % busy).  Before each segment
// the thread forms D^{JK} from its dE/dG, which a few 16-byte loads put into its
// column of shared memory, and B from D and the moments.
// Bound: issue and latency at 8 warps per SM (registers).  Forces of 1.09 M atoms
// 3.29 (two atoms per warp) -> 2.41 ms, 354 k atoms of four elements 1.38 -> 1.16,
// 131 k of a two-element crystal 0.46 -> 0.36.
template <class M>
__device__ void mom_force_thread_body(int block, int nblock, i64 lo, i64 hi, const DevPot *__restrict__ pot,
                                      const float *__restrict__ tab, int fmax, const float2 *__restrict__ rpar,
                                      const int *__restrict__ type, const int *__restrict__ order,
                                      const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap, int gstride,
                                      const float *__restrict__ dEdG, const float2 *__restrict__ mom,
                                      const unsigned long long *__restrict__ mom_mask, double *__restrict__ F,
                                      DevErr *err, float *smem)
{
    constexpr int T = M::T, L = M::L, ND = M::ND, NC = mom_comps(L),
                  NV = mom_vals(T, ND, L), DL = mom_dl(L), BT = NNP_MOM_THREADS;
    f32x2 *D = reinterpret_cast<f32x2 *>(smem) + threadIdx.x;    // [T][L + 1][BT]: of one element
    float *e = reinterpret_cast<float *>(reinterpret_cast<f32x2 *>(smem) + T * (L + 1) * BT) + threadIdx.x;   // [gstride][BT]: dE/dG
    const DevPot &P = *pot;
    const MomTab tb = mom_tab(tab, T, L, fmax);
    for (i64 idx = lo + block * (i64)BT + threadIdx.x; idx < hi; idx += (i64)nblock * BT) {
        const i64 i = order[idx], row = idx - lo;
        const int II = type[i];
        if ((unsigned)II >= (unsigned)T) continue;               // type out of range (reported by the call)
        const int n = nbr_cnt[i];
        const DevType &Ty = P.t[II];
        const float4 *src = nbr + i * cap;
        const unsigned long long mask = mom_mask[row];
        const float *ei = dEdG + i * gstride;
#pragma unroll 8
        for (int k = 0; 4 * k < gstride; ++k) {
            const float4 e4 = __ldg(reinterpret_cast<const float4 *>(ei) + k);
            e[(4 * k) * BT] = e4.x;
            e[(4 * k + 1) * BT] = e4.y;
            e[(4 * k + 2) * BT] = e4.z;
            e[(4 * k + 3) * BT] = e4.w;
        }
        double f0[3] = {0, 0, 0};
        bool bad = false;
        int k = 0;
        float4 rec = n > 0 ? src[0] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
#pragma unroll 1
        for (int J = 0; J < T; ++J) {
            const DevBlockR Br = Ty.br[J];
            // D^{JK}_{l,d} = sum_f e_f c_{f,l} [1 + (J == K)], and the self terms
            float d0 = 0.f, d1 = 0.f;
#pragma unroll 1
            for (int K = 0; K < T; ++K) {
                const int tt = J > K ? J * (J + 1) / 2 + K : K * (K + 1) / 2 + J;
                const bool few = mask >> tt & 1;
                const int off = Ty.ba[tt].off_g, bn = Ty.ba[tt].n;
                const ulonglong2 *cf =
                    reinterpret_cast<const ulonglong2 *>(tb.dcoef + (i64)(II * fmax + off - Ty.n_input_r) * DL);
                f32x2 acc[DL];
#pragma unroll
                for (int l = 0; l < DL; ++l) acc[l] = 0ull;
#pragma unroll 4
                for (int f = 0; f < bn; ++f) {
                    const f32x2 e2 = dup2(few ? 0.f : e[(off + f) * BT]);
#pragma unroll
                    for (int l = 0; l < DL; l += 2) {
                        const ulonglong2 c = __ldg(cf + f * (DL / 2) + l / 2);
                        acc[l] = fma2(e2, c.x, acc[l]);
                        acc[l + 1] = fma2(e2, c.y, acc[l + 1]);
                    }
                }
#pragma unroll
                for (int l = 0; l <= L; ++l) D[(K * (L + 1) + l) * BT] = acc[l];
                if (J == K) up2(acc[L + 1], d0, d1);
            }
            // B^J = norm sum_K D^{JK} A^K
            f32x2 b[NC];
            {
                const f32x2 *a = reinterpret_cast<const f32x2 *>(mom) + mom_at(row, 0, NV, NNP_MOM_SH_T);
#pragma unroll
                for (int l = 0; l <= L; ++l) {
                    f32x2 dk[T];
#pragma unroll
                    for (int K = 0; K < T; ++K) dk[K] = D[(K * (L + 1) + l) * BT];
#pragma unroll
                    for (int m = 0; m <= l; ++m) {
                        const int c0 = m == 0 ? l : mom_base(L, m > 0 ? m : 1) + 2 * (l - m);
#pragma unroll
                        for (int h = 0; h < (m ? 2 : 1); ++h) {
                            f32x2 v = 0ull;
#pragma unroll
                            for (int K = 0; K < T; ++K) v = fma2(dk[K], __ldg(a + ((K * NC + c0 + h) << NNP_MOM_SH_T)), v);
                            b[c0 + h] = mul2(v, dup2(M::gnorm(c0)));
                        }
                    }
                }
            }
#pragma unroll 1
            while ((int)((unsigned)__float_as_int(rec.w) >> 28) == J) {
                MomNbr<M, true> v;
                v.set(rec, Ty, tb.a_lo + II * NNP_MOM_MAXD);
                const i64 j = __float_as_int(rec.w) & 0x0fffffff;
                ++k;
                mom_prefetch(src + min(k + 6, n - 1));
                rec = k < n ? src[k] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
                f32x2 fr, fi, gr2, gi2, hr, hi2;
                {
                    float zn[L + 1];
#pragma unroll
                    for (int q = 1; q <= L; ++q) zn[q] = v.uz * (1.f / (float)(q + 1));
                    mom_gradient_regs<L, L>(b, v.uz, zn, dup2(v.ux), dup2(v.uy), dup2(-v.uy), fr, fi, gr2, gi2, hr, hi2);
                }
                float fc = v.fc[0], fd = v.fd[0];
#pragma unroll
                for (int c = 1; c < M::NCUT; ++c)
                    if (Br.cut == c) {
                        fc = v.fc[c];
                        fd = v.fd[c];
                    }
                float gr = 0.f;
                M::radial_force(II, J, v.r, fc, fd, MomStrided{e + Br.off_g * BT}, gr);
                float a0, a1, gx, gy, gz;
                up2(fr, a0, a1);
                gr = fmaf(fmaf(-d0, v.w[0], a0), v.wd[0], gr);
                if (ND > 1) gr = fmaf(fmaf(-d1, v.w[ND > 1 ? 1 : 0], a1), v.wd[ND > 1 ? 1 : 0], gr);
                const float w0 = v.w[0], w1 = ND > 1 ? v.w[ND > 1 ? 1 : 0] : 0.f;
                up2(gr2, a0, a1);
                gx = fmaf(w1, a1, w0 * a0);
                up2(gi2, a0, a1);
                gy = fmaf(w1, a1, w0 * a0);
                up2(hr, a0, a1);
                gz = fmaf(w1, a1, w0 * a0);
                // dE/dd = u dE/dr + (I - u u^T) dE/du / r
                const float pr = gr - v.ir * (gx * v.ux + gy * v.uy + gz * v.uz);
                const float q[3] = {fmaf(gx, v.ir, pr * v.ux), fmaf(gy, v.ir, pr * v.uy), fmaf(gz, v.ir, pr * v.uz)};
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    bad |= !(fabsf(q[x]) <= 3.402823466e38f);
                    atomicAdd(&F[3 * j + x], (double)q[x]);
                    f0[x] += (double)q[x];
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) atomicAdd(&F[3 * i + x], -f0[x]);
        if (bad) atomicMax(&err->nonfinite, 1);
    }
}

// ---------------------------------------------------------------- tangents

// C_i = sum_k dG_i/dx_k V_k of the training gradient (see tangent_body), one
// thread per atom with at most two damping factors: the moments' derivatives
//   A' = sum_k w'_k rr_k Y(u_k) + w_k (u'_k . grad) Y,
//   rr = u . dv, u' = (dv - rr u) / r, dv = V_i - V_k,
// are the thread's registers as in mom_symm_thread_body, and S' = A'^J A^K +
// A^J A'^K replaces S.  r_n^m and its slope r_(n-1)^(m+1) as in
// mom_gradient_regs; (C, S) = w (x + i y)^m and (Cd, Sd) its derivative.
// Bound: issue and latency at 8 warps per SM (registers).  41 k atoms of two
// elements: training step 909 us (a warp per atom over the pairs) -> 794 us.
template <class M>
__device__ void mom_tangent_thread_body(i64 lo, i64 hi, const DevPot *__restrict__ pot, const float *__restrict__ tab,
                                        int fmax, const int *__restrict__ type, const int *__restrict__ order,
                                        const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap,
                                        int gstride, const float4 *__restrict__ V, const float2 *__restrict__ mom,
                                        float2 *momd, const unsigned long long *__restrict__ mom_mask,
                                        float *__restrict__ Cout, float *smem)
{
    constexpr int T = M::T, TT = T * (T + 1) / 2, L = M::L, ND = M::ND, NC = mom_comps(L), NR = M::NR,
                  NV = mom_vals(T, ND, L), NS = mom_s_vals(T, ND, L), BT = NNP_MOM_THREADS;
    f32x2 *S = reinterpret_cast<f32x2 *>(smem) + threadIdx.x;    // [NS][BT]
    f32x2 *W2 = S + NS * BT;                                     // [T][BT]: sums of w w' rr
    const DevPot &P = *pot;
    const MomTab tb = mom_tab(tab, T, L, fmax);
    for (i64 idx = lo + blockIdx.x * (i64)BT + threadIdx.x; idx < hi; idx += (i64)gridDim.x * BT) {
        const i64 i = order[idx], r = idx - lo;
        const int II = type[i];
        if ((unsigned)II >= (unsigned)T) continue;               // type out of range (reported by the call)
        const int n = nbr_cnt[i];
        const DevType &Ty = P.t[II];
        const float4 *src = nbr + i * cap;
        float *Ci = Cout + i * gstride;
        const float4 vi = V[i];
        int k = 0;
        const float4 none = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
        float4 e = n > 0 ? src[0] : none, ve = vi;
        if (n > 0) ve = V[__float_as_int(e.w) & 0x0fffffff];
#pragma unroll 1
        for (int J = 0; J < T; ++J) {
            f32x2 acc[NC], ww = 0ull;
            float rad[NR];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c] = 0ull;
#pragma unroll
            for (int f = 0; f < NR; ++f) rad[f] = 0.f;
#pragma unroll 1
            while ((int)((unsigned)__float_as_int(e.w) >> 28) == J) {
                MomNbr<M, true> v;
                v.set(e, Ty, tb.a_lo + II * NNP_MOM_MAXD);
                const float dx = vi.x - ve.x, dy = vi.y - ve.y, dz = vi.z - ve.z;
                ++k;
                mom_prefetch(src + min(k + 6, n - 1));
                e = k < n ? src[k] : none;
                if (k < n) ve = V[__float_as_int(e.w) & 0x0fffffff];
                const float rr = v.ux * dx + v.uy * dy + v.uz * dz;
                const float xd = (dx - rr * v.ux) * v.ir, yd = (dy - rr * v.uy) * v.ir, zd = (dz - rr * v.uz) * v.ir;
                const f32x2 w2 = pk2(v.w[0], ND > 1 ? v.w[ND > 1 ? 1 : 0] : 0.f);
                f32x2 C = w2, Sn = 0ull, Sd = 0ull, Cd = pk2(v.wd[0] * rr, ND > 1 ? v.wd[ND > 1 ? 1 : 0] * rr : 0.f);
                ww = fma2(C, Cd, ww);
                const f32x2 x2 = dup2(v.ux), y2 = dup2(v.uy), ny2 = dup2(-v.uy), xd2 = dup2(xd), yd2 = dup2(yd),
                            nyd2 = dup2(-yd), zd2 = dup2(zd);
                float zn[L + 1];
#pragma unroll
                for (int q = 1; q <= L; ++q) zn[q] = v.uz * (1.f / (float)(q + 1));
#pragma unroll
                for (int m = 0; m <= L; ++m) {
                    const f32x2 Cz = mul2(C, zd2), Sz = mul2(Sn, zd2);
                    float q0 = 1.f, q1 = 0.f, p0 = 0.f, p1 = 0.f;   // r_n^m, its slope
#pragma unroll
                    for (int l = m; l <= L; ++l) {
                        const int n1 = l - m;
                        const f32x2 q2 = dup2(q0), p2 = dup2(p0);
                        if (m == 0) {
                            acc[l] = fma2(q2, Cd, acc[l]);
                            if (n1 > 0) acc[l] = fma2(p2, Cz, acc[l]);
                        } else {
                            const int c = mom_base(L, m > 0 ? m : 1) + 2 * n1;
                            acc[c] = fma2(q2, Cd, acc[c]);
                            acc[c + 1] = fma2(q2, Sd, acc[c + 1]);
                            if (n1 > 0) {
                                acc[c] = fma2(p2, Cz, acc[c]);
                                acc[c + 1] = fma2(p2, Sz, acc[c + 1]);
                            }
                        }
                        const float t = n1 == 0 ? v.uz
                                                : fmaf(zn[n1 > 0 ? n1 : 1], q0,
                                                       (-mom_beta(l, m) / (float)(n1 > 0 ? n1 * (n1 + 1) : 1)) * q1);
                        q1 = q0;
                        q0 = t;
                        // r_(n1)^(m+1) from its two before (n1 - 1 of order m + 1 is l of m + 1)
                        const float s = n1 == 0 ? 1.f
                                        : n1 == 1 ? v.uz
                                                  : fmaf(zn[n1 > 1 ? n1 - 1 : 1], p0,
                                                         (-mom_beta(l, m + 1) / (float)(n1 > 1 ? (n1 - 1) * n1 : 1)) * p1);
                        p1 = p0;
                        p0 = s;
                    }
                    const f32x2 c = C, cd = Cd;
                    Cd = fma2(Sd, ny2, fma2(Sn, nyd2, fma2(cd, x2, mul2(c, xd2))));
                    Sd = fma2(Sd, x2, fma2(Sn, xd2, fma2(cd, y2, mul2(c, yd2))));
                    C = fma2(Sn, ny2, mul2(c, x2));
                    Sn = fma2(Sn, x2, mul2(c, y2));
                }
                {
                    float rv[NR];
#pragma unroll
                    for (int f = 0; f < NR; ++f) rv[f] = 0.f;
                    M::radial_drow(II, J, v.r, v.fc, v.fd, rv);
#pragma unroll
                    for (int f = 0; f < NR; ++f) rad[f] = fmaf(rv[f], rr, rad[f]);
                }
            }
            f32x2 *dst = reinterpret_cast<f32x2 *>(momd) + mom_at(r, J * NC, NV, NNP_MOM_SH_T);
#pragma unroll
            for (int c = 0; c < NC; ++c) dst[c << NNP_MOM_SH_T] = mul2(acc[c], dup2(M::gnorm(c)));
            W2[J * BT] = ww;
            const DevBlockR B = Ty.br[J];
#pragma unroll
            for (int f = 0; f < NR; ++f)
                if (f < B.n) Ci[B.off_g + f] = rad[f];
        }
        const f32x2 *a = reinterpret_cast<const f32x2 *>(mom) + mom_at(r, 0, NV, NNP_MOM_SH_T);
        const f32x2 *d = reinterpret_cast<const f32x2 *>(momd) + mom_at(r, 0, NV, NNP_MOM_SH_T);
#pragma unroll
        for (int l = 0; l <= L; ++l) {
            f32x2 s[TT];
#pragma unroll
            for (int tt = 0; tt < TT; ++tt) s[tt] = 0ull;
#pragma unroll
            for (int m = 0; m <= l; ++m)
#pragma unroll
                for (int h = 0; h < (m ? 2 : 1); ++h) {
                    const int c = m == 0 ? l : mom_base(L, m > 0 ? m : 1) + 2 * (l - m) + h;
                    f32x2 va[T], vd[T];
#pragma unroll
                    for (int J = 0; J < T; ++J) {
                        va[J] = a[(J * NC + c) << NNP_MOM_SH_T];
                        vd[J] = d[(J * NC + c) << NNP_MOM_SH_T];
                    }
#pragma unroll
                    for (int K = 0; K < T; ++K)
#pragma unroll
                        for (int J = 0; J <= K; ++J) {
                            const int tt = K * (K + 1) / 2 + J;
                            s[tt] = fma2(va[J], vd[K], fma2(vd[J], va[K], s[tt]));
                        }
                }
#pragma unroll
            for (int tt = 0; tt < TT; ++tt) S[(tt * (L + 1) + l) * BT] = s[tt];
        }
        mom_functions_thread<M, false>(tb, fmax, II, Ty, mom_mask[r], S, W2, -2.f, Ci);
        for (int f = Ty.n_input; f < gstride; ++f) Ci[f] = 0.f;
    }
}

// Tangents of the listed blocks: of many pairs, a warp each, a lane per pair; of few,
// 16 lanes each, a lane per pair.
template <class M>
__device__ void mom_list_tangent_body(const MomLists ls, i64 lo, const DevPot *__restrict__ pot,
                                      const float *__restrict__ tab, int fmax, const int *__restrict__ type,
                                      const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
                                      const unsigned short *__restrict__ mom_cnt, const float4 *__restrict__ V,
                                      float *__restrict__ Cout)
{
    struct Nbr {
        float u[3], ud[3], w[M::ND], wr[M::ND];   // direction and damping factors, and their derivatives
    };
    const MomTab tb = mom_tab(tab, M::T, M::L, fmax);
    const int id = blockIdx.x * NNP_MOM_FEW_THREADS + threadIdx.x, all = gridDim.x * (NNP_MOM_FEW_THREADS / 16);
    for (MomQueue u(ls.wide, ls.n[1], order + lo, id >> 5, all / 2); u.q < u.n; u.next()) {
        const i64 i = u.i;
        const int II = type[i], tt = u.it.y;
        const DevType &Ty = pot->t[II];
        u.ahead();
        const float *a_lo = tb.a_lo + II * NNP_MOM_MAXD;
        const float4 *src = nbr + i * cap;
        const float4 vi = V[i];
        float acc[M::NA];
#pragma unroll
        for (int f = 0; f < M::NA; ++f) acc[f] = 0.f;
        mom_wide_pairs(
            mom_wide<M::T>(mom_cnt + 8 * (i64)u.it.x, tt),
            [&](int k) {
                const float4 rec = src[k], vk = V[__float_as_int(rec.w) & 0x0fffffff];
                MomNbr<M, true> v;
                v.set(rec, Ty, a_lo);
                const float dv[3] = {vi.x - vk.x, vi.y - vk.y, vi.z - vk.z};
                const float rr = v.ux * dv[0] + v.uy * dv[1] + v.uz * dv[2];
                Nbr o;
                o.u[0] = v.ux;
                o.u[1] = v.uy;
                o.u[2] = v.uz;
#pragma unroll
                for (int x = 0; x < 3; ++x) o.ud[x] = (dv[x] - rr * o.u[x]) * v.ir;
#pragma unroll
                for (int d = 0; d < M::ND; ++d) {
                    o.w[d] = v.w[d];
                    o.wr[d] = v.wd[d] * rr;
                }
                return o;
            },
            [&](const Nbr &A, int a, const Nbr &B, int b, bool ok) {
                float cs = 0.f, cd = 0.f, w[M::ND], dw[M::ND];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const float ua = __shfl_sync(NNP_FULL, A.u[x], a), ub = __shfl_sync(NNP_FULL, B.u[x], b);
                    const float da = __shfl_sync(NNP_FULL, A.ud[x], a), db = __shfl_sync(NNP_FULL, B.ud[x], b);
                    cs = fmaf(ua, ub, cs);
                    cd = fmaf(da, ub, fmaf(ua, db, cd));
                }
#pragma unroll
                for (int d = 0; d < M::ND; ++d) {
                    const float wa = __shfl_sync(NNP_FULL, A.w[d], a), wb = __shfl_sync(NNP_FULL, B.w[d], b);
                    const float ra = __shfl_sync(NNP_FULL, A.wr[d], a), rb = __shfl_sync(NNP_FULL, B.wr[d], b);
                    w[d] = wa * wb * cd;
                    dw[d] = fmaf(ra, wb, wa * rb);
                }
                if (ok) M::few_tangent(II, tt, cs, w, dw, acc);
            });
        const int n = Ty.ba[tt].n;
        float *Cb = Cout + i * gstride + Ty.ba[tt].off_g;
#pragma unroll
        for (int f = 0; f < M::NA; ++f) {
            const float v = warp_sum(acc[f]);
            if ((threadIdx.x & 31) == 0 && f < n) Cb[f] = v;
        }
    }
    __syncwarp();
    const int nit = ls.n[0], h = threadIdx.x & 15;
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    for (int q = mom_few_first(ls, id >> 4, all); q < nit; q += all) {
        const int2 it = ls.few[q];
        const i64 i = order[lo + it.x];
        const int II = type[i], tt = it.y;
        const DevType &Ty = pot->t[II];
        const MomFew b = mom_few<M::T>(mom_cnt + 8 * (i64)it.x, tt, h);
        MomNbr<M, true> v;
        const float4 rec = nbr[i * cap + mom_few_slot(b, h)], vi = V[i], vk = V[__float_as_int(rec.w) & 0x0fffffff];
        v.set(rec, Ty, tb.a_lo + II * NNP_MOM_MAXD);
        const float dv[3] = {vi.x - vk.x, vi.y - vk.y, vi.z - vk.z}, u[3] = {v.ux, v.uy, v.uz};
        const float rr = u[0] * dv[0] + u[1] * dv[1] + u[2] * dv[2];
        float cs = 0.f, cd = 0.f, w[M::ND], dw[M::ND], acc[M::NA];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const float ud = (dv[x] - rr * u[x]) * v.ir;
            const float ua = __shfl_sync(mask, u[x], b.a, 16), ub = __shfl_sync(mask, u[x], b.b, 16);
            const float da = __shfl_sync(mask, ud, b.a, 16), db = __shfl_sync(mask, ud, b.b, 16);
            cs = fmaf(ua, ub, cs);
            cd = fmaf(da, ub, fmaf(ua, db, cd));
        }
#pragma unroll
        for (int d = 0; d < M::ND; ++d) {
            const float wr = v.wd[d] * rr;
            const float wa = __shfl_sync(mask, v.w[d], b.a, 16), wb = __shfl_sync(mask, v.w[d], b.b, 16);
            const float ra = __shfl_sync(mask, wr, b.a, 16), rb = __shfl_sync(mask, wr, b.b, 16);
            w[d] = wa * wb * cd;
            dw[d] = fmaf(ra, wb, wa * rb);
        }
#pragma unroll
        for (int f = 0; f < M::NA; ++f) acc[f] = 0.f;
        if (h < b.pairs) M::few_tangent(II, tt, cs, w, dw, acc);
        const int n = Ty.ba[tt].n;
        float *Cb = Cout + i * gstride + Ty.ba[tt].off_g;
#pragma unroll
        for (int f = 0; f < M::NA; ++f) {
            float s = acc[f];
#pragma unroll
            for (int o = 8; o; o >>= 1) s += __shfl_xor_sync(mask, s, o, 16);
            if (h == 0 && f < n) Cb[f] = s;
        }
    }
}

#endif  // __CUDACC__

}  // namespace nnp
