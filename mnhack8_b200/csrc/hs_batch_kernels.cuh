// hs_batch_kernels.cuh -- kernels of the batched mixed-precision solver
// (hs_batch.cu).  Many independent transient-heat solves advance together:
// every launch covers the slab tiles (operator) or flat blocks (vector work)
// of all instances, and a block finds its instance through a map.  Each
// implicit-Euler step solves (M + dt K) T = M T_old by defect correction:
// FP64 residual r = b - A T (the slab operator in FP64, ABFT checked),
// an FP32 Jacobi-PCG solve of A d = r to a loose relative tolerance (FP32
// operator and preconditioner, FP64 dot products of the FP32 values), and
// T += d in FP64, until ||b - A T|| / ||b|| < rtol.
// The sums of the FP64 applies (the outer residual ||b - A T||, ||b||, the
// ABFT checksum sums of the FP64 applies) and the inner solve's starting r.z
// and r.r are accumulated in FP64 with compensation (hs_csum.h); the inner
// FP32 iterations' sums are plain FP64 sums of FP32 values.  A compensated
// partial is a pair (hi, lo), stored as quantity q and q + NQ, and merged pair-wise.
#pragma once
#include "hs_kernels.cuh"
#include "hs_csum.h"

namespace hs {

// canonical block tree (as cta_tree_sum) over compensated pairs; sh holds
// 2*NQ rows of 8; result valid in thread 0
template <int NQ>
__device__ __forceinline__ void cta_tree_csum(CSum (&v)[NQ], double (*sh)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const CSum o{__shfl_xor_sync(0xffffffffu, v[q].hi, off), __shfl_xor_sync(0xffffffffu, v[q].lo, off)};
            csum_merge(v[q], o);
        }
    }
    __syncthreads();
    if (lane == 0 && warp < 8) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) { sh[q][warp] = v[q].hi; sh[NQ + q][warp] = v[q].lo; }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            CSum u{(lane < 8) ? sh[q][lane] : 0.0, (lane < 8) ? sh[NQ + q][lane] : 0.0};
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) {
                const CSum o{__shfl_xor_sync(0xffffffffu, u.hi, off), __shfl_xor_sync(0xffffffffu, u.lo, off)};
                csum_merge(u, o);
            }
            v[q] = u;
        }
    }
}
// store a block's compensated partials: hi as quantity q, lo as q + NQ
template <int NQ>
__device__ __forceinline__ void store_cpartials(const CSum (&v)[NQ], double* base, long long stride, long long idx) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        base[q * stride + idx] = v[q].hi;
        base[(NQ + q) * stride + idx] = v[q].lo;
    }
}

// per-instance scalars, device resident
struct BState {
    // inner FP32 PCG
    double rho, alpha, beta, bn_in, tol_in;
    int iter, done, broken, pad0;
    // outer defect correction
    double bn64, rel64, d1_last, d1_max64, d1_max32;
    double norm_wA, norm_wM;
    int outer, odone, pad1, pad2;
    // counters over the run
    long long inner_total, outer_total, applies32, applies64;
    // armed vector fault of the current step: level 5 p32 (after formation),
    // 6 r32 (after its update), 7 Ap32 (after projection), at correction
    // fi_outer (1-based) and inner iteration fi_iter; 0 = none
    int fi_vec, fi_outer, fi_iter, fi_bit;
    long long fi_idx;
    int fi_fired;           // the armed fault has fired
    int stalls;             // steps that ended at max_outer without reaching rtol
    int inner_bad;          // the current inner solve went non-finite: its correction is discarded
    int inner_faults;       // inner solves discarded so far
    int has_prev;           // the previous step's field is kept (extrapolated start)
    int extrap;             // this step starts from 2 T - T_prev
    unsigned tick_a, tick_u;   // blocks of the running inner apply / update that are done
    int stuck;              // a bounded wait gave up: the inner solve is discarded
    int pend;               // d += alpha p of the last (even) inner iteration is still owed
    double alpha_prev;      // alpha of the inner iteration before
};

__device__ __forceinline__ float flipf(float x, int bit) {
    return __uint_as_float(__float_as_uint(x) ^ (1u << bit));
}
// the armed fault of level `vec` fires in this inner iteration
__device__ __forceinline__ bool fi_now(const BState* st, int vec) {
    return st->fi_vec == vec && st->outer == st->fi_outer && st->iter == st->fi_iter;
}

// instance descriptor (device array, rewritten by the host between rounds)
struct BInst {
    Part part;                 // slab tiles and flat blocks of this instance
    long long tile0, flat0;    // first global tile / flat block
    long long chunk0, nchunk;  // first block of the inner update, and their number
    double dt;
    double cm[4], ck[4];       // wht eigen-constants / 8 of this grid
    float cmf[4], ckf[4];
    int active;
    int uniform;               // rho*c is one value: k32 holds k alone
    float rc32;                // and its value
    int rounds;                // of UR nodes that a block of it takes (upd_rounds)
    double* T;                 // solution (updated in place)
    double* b;                 // right-hand side M T_old
    double* y64;               // FP64 operator output
    double* r64;               // FP64 residual
    double* Tm1;               // field at the start of the previous step (extrapolated start)
    const double2* coef64;     // (rho*c, k) per element
    const float2* coef32;      // varying rho*c
    const float* k32;          // uniform rho*c (the same buffer)
    const double* wA;          // ABFT weights A 1_int, M 1_int (FP64)
    const double* wM;
    const float* dinv32;       // 1 / diag, FP32
    float* r32;
    float* z32;
    float* p32a;
    float* p32b;
    float* Ap32;
    float* d32;                // correction
    BState* st;
};

struct BatchArgs {
    const BInst* inst;
    const int* tile2inst;      // global tile -> instance slot (-1: none)
    const int* flat2inst;      // global flat block -> instance slot
    const int* chunk2inst;     // block of the inner update -> instance slot
    int n_inst, pad;
    long long ntiles, nflat, nchunk;   // capacity of the grids
    double* pa;                // apply partials: [q * ntiles + tile]
    double* pf;                // flat partials:  [q * nflat + block]
    double rtol, inner_tol;
    int max_outer, max_inner;
    int detect, extrapolate;
    unsigned long long neg0;   // (-0.f, -0.f), see f2_mul
};

template <typename V> struct VTraits;
template <> struct VTraits<float> {
    using V2 = float2;
    __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ static float sub(float a, float b) { return __fsub_rn(a, b); }
    __device__ static float mul(float a, float b) { return __fmul_rn(a, b); }
    __device__ static float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
};
template <> struct VTraits<double> {
    using V2 = double2;
    __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static double sub(double a, double b) { return __dsub_rn(a, b); }
    __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
    __device__ static double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
};

// the Walsh-Hadamard element operator in precision V (same structure as elem_wht)
template <typename V>
__device__ __forceinline__ void elem_wht_v(V* v, V rhoc, V dk, const V* cm, const V* ck) {
    using T = VTraits<V>;
#pragma unroll
    for (int bit = 1; bit <= 4; bit <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (!(q & bit)) { const V u = v[q], w = v[q | bit]; v[q] = T::add(u, w); v[q | bit] = T::sub(u, w); }
    const V l0 = T::mul(rhoc, cm[0]);
    const V l1 = T::fma(dk, ck[1], T::mul(rhoc, cm[1]));
    const V l2 = T::fma(dk, ck[2], T::mul(rhoc, cm[2]));
    const V l3 = T::fma(dk, ck[3], T::mul(rhoc, cm[3]));
    v[0] = T::mul(v[0], l0);
    v[1] = T::mul(v[1], l1); v[2] = T::mul(v[2], l1); v[4] = T::mul(v[4], l1);
    v[3] = T::mul(v[3], l2); v[5] = T::mul(v[5], l2); v[6] = T::mul(v[6], l2);
    v[7] = T::mul(v[7], l3);
#pragma unroll
    for (int bit = 1; bit <= 4; bit <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (!(q & bit)) { const V u = v[q], w = v[q | bit]; v[q] = T::add(u, w); v[q | bit] = T::sub(u, w); }
}

struct __align__(16) BSlabSmem {
    double P[2][SPOS];
    double2 Y1[SPOS], Y2[SPOS], Y3[SPOS];
    double sh[2 * MAXQ][8];
};

// Batched slab operator in FP64.  KIND 0: y64 = A T (residual); 1: b = M T
// (right-hand side).  Partials per tile (compensated): D1's 1_int.y, w.x, x.x.
enum BKind { BK_RESID = 0, BK_RHS = 1 };

template <int KIND>
__global__ void __launch_bounds__(ST, 2) kb_apply(BatchArgs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BSlabSmem& S = *reinterpret_cast<BSlabSmem*>(smem_raw);
    const long long t = blockIdx.x;
    if (t >= B.ntiles) return;
    const int slot = B.tile2inst[t];
    if (slot < 0) return;
    const BInst& I = B.inst[slot];
    if (!I.active) return;
    if (KIND == BK_RESID && I.st->odone) return;
    const Part& P = I.part;
    const int N = P.N, Cw = P.Cw;
    // node and element indices fit in 32 bits (N <= 1200)
    const unsigned plane = (unsigned)P.NN * (unsigned)P.NN, eplane = (unsigned)N * (unsigned)N;
    const SlabTile Tt = slab_tile(P, t - I.tile0);
    const SlabPos G = slab_pos(P, Tt, threadIdx.x);
    const unsigned fl = G.fl;
    const int tid = threadIdx.x, xa = Tt.xa, xb = Tt.xb;
    const double dtv = (KIND == BK_RHS) ? 0.0 : I.dt;
    double cm[4], ck[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { cm[j] = I.cm[j]; ck[j] = I.ck[j]; }
    const double* src = I.T;
    double* yout = KIND == BK_RHS ? I.b : I.y64;
    const double* w = (KIND == BK_RHS) ? I.wM : I.wA;
    const bool d1 = B.detect != 0;
    CSum part[MAXQ] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};

    double pA[SK], pB[SK], aA[SK], aB[SK], ra[SK], cr[SK], ckk[SK], wv[SK];
    auto ld_raw = [&](int px) {
        const bool pv = px >= 0 && px <= N;
        const unsigned base = (unsigned)px * plane;
#pragma unroll
        for (int k = 0; k < SK; ++k) ra[k] = (pv && sp_valid(fl, k)) ? __ldg(src + (base + (unsigned)G.noff[k])) : 0.0;
    };
    auto ld_coef = [&](int ex) {
        const bool ev = ex >= 0 && ex < N;
        const unsigned base = (unsigned)ex * eplane;
#pragma unroll
        for (int k = 0; k < SK; ++k) {
            const bool v = ev && sp_elem(fl, k);
            const double2 c = v ? __ldg(I.coef64 + (base + (unsigned)G.eoff[k])) : make_double2(0.0, 0.0);
            cr[k] = c.x; ckk[k] = c.y;
        }
    };
    auto ld_w = [&](int px) {
        const bool pv = px >= xa && px <= xb;
        const unsigned base = (unsigned)px * plane;
#pragma unroll
        for (int k = 0; k < SK; ++k)
            wv[k] = (pv && d1 && sp_out(fl, k)) ? __ldg(w + (base + (unsigned)G.noff[k])) : 0.0;
    };
    auto layer = [&](int ix, int cur, double (&pc)[SK], double (&pn)[SK], double (&ac)[SK], double (&an)[SK]) {
        const int nxt = cur ^ 1;
#pragma unroll
        for (int k = 0; k < SK; ++k) { pn[k] = ra[k]; S.P[nxt][tid + k * ST] = pn[k]; }
        ld_raw(ix + 2 <= xb + 1 ? ix + 2 : -2);
        __syncthreads();
        if (ix >= 0 && ix < N) {
#pragma unroll
            for (int k = 0; k < SK; ++k) {
                if (!sp_elem(fl, k)) continue;
                const int j = tid + k * ST;
                double v[8];
                v[0] = pc[k];
                v[1] = S.P[cur][j + 1];
                v[2] = S.P[cur][j + Cw];
                v[3] = S.P[cur][j + Cw + 1];
                v[4] = pn[k];
                v[5] = S.P[nxt][j + 1];
                v[6] = S.P[nxt][j + Cw];
                v[7] = S.P[nxt][j + Cw + 1];
                elem_wht_v<double>(v, cr[k], dmul(dtv, ckk[k]), cm, ck);
                ac[k] = dadd(ac[k], v[0]);
                an[k] = dadd(0.0, v[4]);
                S.Y1[j + 1] = make_double2(v[1], v[5]);
                S.Y2[j + Cw] = make_double2(v[2], v[6]);
                S.Y3[j + Cw + 1] = make_double2(v[3], v[7]);
            }
        }
        ld_coef(ix + 1 <= xb ? ix + 1 : -1);
        __syncthreads();
        const unsigned base = (unsigned)ix * plane;
        const bool xbnd = ix == 0 || ix == N;
#pragma unroll
        for (int k = 0; k < SK; ++k) {
            if (!sp_out(fl, k)) continue;
            const int j = tid + k * ST;
            const bool yzin = !sp_yzb(fl, k);
            double2 y3 = make_double2(0.0, 0.0), y2 = y3, y1 = y3;
            if (yzin) { y3 = S.Y3[j]; y2 = S.Y2[j]; y1 = S.Y1[j]; }
            if (ix >= xa) {
                const unsigned n = base + (unsigned)G.noff[k];
                const bool bnd = !yzin || xbnd;
                const double y = bnd ? 0.0 : dadd(dadd(dadd(ac[k], y3.x), y2.x), y1.x);
                // p read once: with pc[k] itself in the sums the march took 12 % longer
                // (8 instances at N=32: 31.4 against 28.0 us, N=96 x 4: 76.4 against 70.9)
                const double pv = pc[k];
                if (d1) {
                    if (!bnd) csum_add(part[1], y);
                    csum_fma(part[2], wv[k], pv);
                    part[3].hi = dfma(pv, pv, part[3].hi);  // the norm only scales the threshold
                }
                __stwb(yout + n, y);                      // global stores (the pointers come from global memory)
            }
            an[k] = yzin ? dadd(dadd(dadd(an[k], y3.y), y2.y), y1.y) : 0.0;
        }
        ld_w(ix + 1);
    };
    ld_raw(xa - 1);
#pragma unroll
    for (int k = 0; k < SK; ++k) { pA[k] = ra[k]; S.P[0][tid + k * ST] = pA[k]; aA[k] = 0.0; aB[k] = 0.0; }
    ld_raw(xa);
    ld_coef(xa - 1);
    for (int ix = xa - 1; ix <= xb; ++ix) {
        layer(ix, (ix - xa + 1) & 1, pA, pB, aA, aB);
#pragma unroll
        for (int k = 0; k < SK; ++k) { pA[k] = pB[k]; aA[k] = aB[k]; }
    }
    if (!d1) return;
    cta_tree_csum<MAXQ>(part, S.sh);
    if (threadIdx.x == 0) store_cpartials<MAXQ>(part, B.pa, B.ntiles, t);
}

__device__ __forceinline__ double d1_rel(const double (&p)[MAXQ], double nw) {
    const double nx = __dsqrt_rn(p[3]);
    double rel = __ddiv_rn(fabs(dsub(p[1], p[2])), dfma(nw, nx, 1e-300));
    if (!isfinite(rel)) rel = 1e300;
    return rel;
}

// ---- the FP32 inner loop: operator ------------------------------------------------
// The slab march of the FP64 operator (k_apply_slab: one barrier per layer,
// p stored and checked as it is formed) in FP32: a thread applies its FK
// elements two at a time in packed FP32 registers, and uniform rho*c is read as
// one value.  The FP64 sums of the FP32 products (p.Ap, 1_int.Ap, w.p, p.p) are
// per thread, per tile (a block tree), and then per instance by the last CTA of
// the instance to finish (an atomic ticket), which also sets alpha; a launch
// per iteration did that before.
//
// Bound by issue and latency (N=160: 54 us, IPC 0.55 a scheduler, against 20 us
// of HBM traffic).  Measured (B200, device ms of all steps; two barriers a layer,
// separate final kernels -> this): 24 instances of N 16..96, 20 steps 158.8 ->
// 148; N=160, 10 steps 162.6 -> 148, of which the packed arithmetic 153 -> 148.  Slower: 512 threads of two
// positions (64 registers: spills, 158 and 162), three or four CTAs per SM (169
// and 193, 215 and 298), inputs two layers ahead (164 and 170).
constexpr int FT = 256, FK = SPOS / FT;
struct __align__(16) FSlabSmem {
    float P[3][SPOS];
    float2 Y1[SPOS], Y2[SPOS], Y3[SPOS];
    double sh[MAXQ][16];
    unsigned long long free_bar;
    unsigned last;
};

// sum over a CTA of W warps: xor butterfly per warp, then over the warp sums;
// valid in thread 0
template <int NQ, int W>
__device__ __forceinline__ void cta_tree_w(double (&v)[NQ], double (*sh)[16]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = dadd(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) sh[q][warp] = v[q];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = sh[q][lane % W];
#pragma unroll
        for (int off = W / 2; off >= 1; off >>= 1)
#pragma unroll
            for (int q = 0; q < NQ; ++q) v[q] = dadd(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
    }
}
// The CTA's sums become partial idx of an instance's count partials (quantity q
// at base + q * stride); true in the last CTA to get here, which adds them up
// (inst_total).  The state it needs for its scalar step is read in between: after
// the totals those loads came one after the other (2 instances at N=16 2.71 -> 2.58
// ms of 4 steps, one at N=160 28.2 -> 27.3).
template <int NQ, int NT>
__device__ __forceinline__ bool inst_arrive(double (&v)[NQ], double* base, long long stride, long long idx,
                                            long long count, unsigned* ticket, double (*sh)[16], unsigned* s_last) {
    cta_tree_w<NQ, NT / 32>(v, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) base[q * stride + idx] = v[q];
        __threadfence();
        *s_last = atomicAdd(ticket, 1u) == (unsigned)(count - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (!*s_last) return false;
    __threadfence();
    return true;
}
// strided sums of the instance's partials, then the tree: the totals in thread 0
template <int NQ, int NT, int FB>
__device__ __forceinline__ void inst_total(double (&v)[NQ], const double* base, long long stride, long long count,
                                           unsigned* ticket, double (*sh)[16]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = 0.0;
    for (long long k0 = threadIdx.x; k0 < count; k0 += (long long)NT * FB) {
        double t[NQ][FB];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int u = 0; u < FB; ++u) {
                const long long k = k0 + (long long)u * NT;
                t[q][u] = k < count ? __ldcg(base + q * stride + k) : 0.0;
            }
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int u = 0; u < FB; ++u) v[q] = dadd(v[q], t[q][u]);
    }
    cta_tree_w<NQ, NT / 32>(v, sh);
    if (threadIdx.x == 0) *ticket = 0u;
}

// Two FP32 lanes in one 64-bit register, each rounded like the scalar operation.
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_get(F2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { F2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
// A product as a multiply-add of -0, which the caller passes as a run-time
// value: the assembler contracts mul.rn.f32x2, and a multiply-add of a constant
// -0, with the addition that follows (seen on sm_100a with CUDA 12.9 despite
// --fmad=false; it changes the result's last bit).
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b, F2 neg0) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg0));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
// elem_wht_v on two elements side by side
__device__ __forceinline__ void elem_wht_f2(F2* v, F2 rhoc, F2 dk, const float* cm, const float* ck, F2 neg0) {
#pragma unroll
    for (int bit = 1; bit <= 4; bit <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (!(q & bit)) { const F2 u = v[q], w = v[q | bit]; v[q] = f2_add(u, w); v[q | bit] = f2_sub(u, w); }
    const F2 l0 = f2_mul(rhoc, f2(cm[0], cm[0]), neg0);
    F2 l[4];
#pragma unroll
    for (int j = 1; j < 4; ++j) l[j] = f2_fma(dk, f2(ck[j], ck[j]), f2_mul(rhoc, f2(cm[j], cm[j]), neg0));
    v[0] = f2_mul(v[0], l0, neg0);
    v[1] = f2_mul(v[1], l[1], neg0); v[2] = f2_mul(v[2], l[1], neg0); v[4] = f2_mul(v[4], l[1], neg0);
    v[3] = f2_mul(v[3], l[2], neg0); v[5] = f2_mul(v[5], l[2], neg0); v[6] = f2_mul(v[6], l[2], neg0);
    v[7] = f2_mul(v[7], l[3], neg0);
#pragma unroll
    for (int bit = 1; bit <= 4; bit <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (!(q & bit)) { const F2 u = v[q], w = v[q | bit]; v[q] = f2_add(u, w); v[q | bit] = f2_sub(u, w); }
}

// RC: uniform rho*c.  FI: an armed flip of p or Ap fires in this iteration.
template <bool RC, bool FI>
__device__ __forceinline__ void kb_march32(const BatchArgs& B, FSlabSmem& S, const BInst& I, const SlabTile& T,
                                           double (&part)[MAXQ]) {
    using VT = VTraits<float>;
    BState* st = I.st;
    const Part& P = I.part;
    const int N = P.N, Cw = P.Cw, npos = P.Rw * P.Cw;
    const unsigned plane = (unsigned)P.NN * (unsigned)P.NN, eplane = (unsigned)N * (unsigned)N;
    const int tid = threadIdx.x, lane = tid & 31, xa = T.xa, xb = T.xb;
    // geometry (slab_pos with FT threads): node and element offsets, flags as there
    unsigned noff[FK], eoff[FK], fl = 0u;
    bool on[FK];                                    // some position of this warp's k-th row exists
#pragma unroll
    for (int k = 0; k < FK; ++k) {
        const int j = tid + k * FT;
        const int lr = j / Cw, lc = j - lr * Cw, gy = T.y0 - 1 + lr, gz = T.z0 - 1 + lc;
        const bool in = j < npos;
        const bool valid = in && gy >= 0 && gy <= N && gz >= 0 && gz <= N;
        const bool elem = in && lr <= P.Rw - 2 && lc <= Cw - 2 && gy >= 0 && gy < N && gz >= 0 && gz < N;
        const bool out = valid && lr >= 1 && lr <= P.Rw - 2 && lc >= 1 && lc <= Cw - 2;
        const bool yzb = gy == 0 || gy == N || gz == 0 || gz == N;
        noff[k] = valid ? (unsigned)(gy * P.NN + gz) : 0u;
        eoff[k] = elem ? (unsigned)(gy * N + gz) : 0u;
        fl |= (valid ? 1u : 0u) << k | (elem ? 1u : 0u) << (8 + k) | (out ? 1u : 0u) << (16 + k) |
              (yzb ? 1u : 0u) << (24 + k);
        on[k] = (j & ~31) < npos;
    }
    const float dtv = (float)I.dt, rc = RC ? I.rc32 : 0.f;
    float cm[4], ck[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { cm[j] = I.cmf[j]; ck[j] = I.ckf[j]; }
    const int iter = st->iter;
    const float beta = (float)st->beta;
    const float* src_a = I.z32;
    const bool two = iter > 0;
    const float* src_b = two ? ((iter & 1) ? I.p32a : I.p32b) : src_a;
    float* pout = (iter & 1) ? I.p32b : I.p32a;
    float* yout = I.Ap32;
    const double* w = I.wA;
    const bool d1 = B.detect != 0;
    const bool fi_p = FI && fi_now(st, FI_P), fi_ap = FI && fi_now(st, FI_AP);
    const int fi_bit = FI ? st->fi_bit : 0;
    const long long fi_idx = FI ? st->fi_idx : -1;

    float cr[FK], ckk[FK];
    auto ld_raw = [&](int px, float (&ra)[FK], float (&rb)[FK], double (&wv)[FK]) {
        const bool pv = px >= 0 && px <= N, pt = px >= xa && px <= xb;
        const unsigned base = (unsigned)px * plane;
#pragma unroll
        for (int k = 0; k < FK; ++k) {
            const bool v = pv && sp_valid(fl, k);
            const unsigned n = base + noff[k];
            ra[k] = v ? __ldg(src_a + n) : 0.f;
            rb[k] = (v && two) ? __ldg(src_b + n) : 0.f;
            wv[k] = (pt && d1 && sp_out(fl, k)) ? __ldg(w + n) : 0.0;
        }
    };
    auto form = [&](int px, float* Pl, const float (&ra)[FK], const float (&rb)[FK], const double (&wv)[FK]) {
        const bool pt = px >= xa && px <= xb;
        const unsigned base = (unsigned)px * plane;
#pragma unroll
        for (int k = 0; k < FK; ++k) {
            float v = two ? VT::fma(beta, rb[k], ra[k]) : ra[k];
            if (fi_p && sp_valid(fl, k) && (long long)px * plane + noff[k] == fi_idx) {
                v = flipf(v, fi_bit);
                st->fi_fired = 1;
            }
            Pl[tid + k * FT] = v;
            if (pt && sp_out(fl, k)) {
                if (d1) {
                    const double vd = (double)v;
                    part[2] = dfma(wv[k], vd, part[2]);
                    part[3] = dfma(vd, vd, part[3]);
                }
                __stwb(pout + (base + noff[k]), v);        // global stores (the pointers come from global memory)
            }
        }
    };
    auto ld_coef = [&](int ex) {
        const bool ev = ex >= 0 && ex < N;
        const unsigned base = (unsigned)ex * eplane;
#pragma unroll
        for (int k = 0; k < FK; ++k) {
            const bool v = ev && sp_elem(fl, k);
            if constexpr (RC) {
                ckk[k] = v ? __ldg(I.k32 + (base + eoff[k])) : 0.f;
            } else {
                const float2 c = v ? __ldg(I.coef32 + (base + eoff[k])) : make_float2(0.f, 0.f);
                cr[k] = c.x; ckk[k] = c.y;
            }
        }
    };
    const unsigned free_bar = (unsigned)__cvta_generic_to_shared(&S.free_bar);
    unsigned phase = 0;
    float ac[FK], an[FK], ra[FK], rb[FK];
    double wv[FK];
    auto layer = [&](int ix, float* P0, float* P1, float* P2) {
        const bool el = ix >= 0 && ix < N;
#pragma unroll
        for (int k = 0; k < FK; k += 2) {
            an[k] = an[k + 1] = 0.f;
            F2 v[8];
            const int j = tid + k * FT, i = j + FT;
            if (el && on[k]) {
                v[0] = f2(P0[j], P0[i]);
                v[1] = f2(P0[j + 1], P0[i + 1]);
                v[2] = f2(P0[j + Cw], P0[i + Cw]);
                v[3] = f2(P0[j + Cw + 1], P0[i + Cw + 1]);
                v[4] = f2(P1[j], P1[i]);
                v[5] = f2(P1[j + 1], P1[i + 1]);
                v[6] = f2(P1[j + Cw], P1[i + Cw]);
                v[7] = f2(P1[j + Cw + 1], P1[i + Cw + 1]);
                elem_wht_f2(v, RC ? f2(rc, rc) : f2(cr[k], cr[k + 1]), f2(VT::mul(dtv, ckk[k]), VT::mul(dtv, ckk[k + 1])),
                            cm, ck, B.neg0);
                float a, b;
                f2_get(v[0], a, b);
                ac[k] = VT::add(ac[k], a); ac[k + 1] = VT::add(ac[k + 1], b);
                f2_get(v[4], a, b);
                an[k] = VT::add(0.f, a); an[k + 1] = VT::add(0.f, b);
            }
            // the hand-over buffers are free again
            if (k == 0 && ix >= xa && !mbar_wait(free_bar, phase)) st->stuck = 1;
            if (el) {
                float a[8], b[8];
#pragma unroll
                for (int q = 1; q < 8; ++q) f2_get(v[q], a[q], b[q]);
                if (sp_elem(fl, k)) {
                    S.Y1[j + 1] = make_float2(a[1], a[5]);
                    S.Y2[j + Cw] = make_float2(a[2], a[6]);
                    S.Y3[j + Cw + 1] = make_float2(a[3], a[7]);
                }
                if (sp_elem(fl, k + 1)) {
                    S.Y1[i + 1] = make_float2(b[1], b[5]);
                    S.Y2[i + Cw] = make_float2(b[2], b[6]);
                    S.Y3[i + Cw + 1] = make_float2(b[3], b[7]);
                }
            }
        }
        if (ix >= xa) phase ^= 1u;
        ld_coef(ix + 1 <= xb ? ix + 1 : -1);
        form(ix + 2, P2, ra, rb, wv);
        ld_raw(ix + 3 <= xb + 1 ? ix + 3 : -2, ra, rb, wv);
        __syncthreads();
        const unsigned base = (unsigned)ix * plane;
        const bool xbnd = ix == 0 || ix == N;
#pragma unroll
        for (int k = 0; k < FK; ++k) {
            if (!sp_out(fl, k)) continue;
            const int j = tid + k * FT;
            const bool yzin = !sp_yzb(fl, k);
            float2 y3 = make_float2(0.f, 0.f), y2 = y3, y1 = y3;
            if (yzin) { y3 = S.Y3[j]; y2 = S.Y2[j]; y1 = S.Y1[j]; }
            if (ix >= xa) {
                const unsigned n = base + noff[k];
                const bool bnd = !yzin || xbnd;
                float y = bnd ? 0.f : VT::add(VT::add(VT::add(ac[k], y3.x), y2.x), y1.x);
                if (fi_ap && (long long)n == fi_idx) { y = flipf(y, fi_bit); st->fi_fired = 1; }
                const double yd = (double)y;
                part[0] = dfma((double)P0[j], yd, part[0]);
                if (d1 && !bnd) part[1] = dadd(part[1], yd);
                __stwb(yout + n, y);
            }
            ac[k] = yzin ? VT::add(VT::add(VT::add(an[k], y3.y), y2.y), y1.y) : 0.f;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(free_bar);
    };
    if (tid == 0) mbar_init(free_bar, FT / 32);
    float *P0 = S.P[0], *P1 = S.P[1], *P2 = S.P[2];
    {
        float ra0[FK], rb0[FK];
        double wv0[FK];
        ld_raw(xa - 1, ra0, rb0, wv0);
        ld_raw(xa, ra, rb, wv);
        ld_coef(xa - 1);
#pragma unroll
        for (int k = 0; k < FK; ++k) ac[k] = 0.f;
        form(xa - 1, P0, ra0, rb0, wv0);
        form(xa, P1, ra, rb, wv);
        ld_raw(xa + 1, ra, rb, wv);
    }
    __syncthreads();
    for (int ix = xa - 1; ix <= xb; ++ix) {
        layer(ix, P0, P1, P2);
        float* t = P0; P0 = P1; P1 = P2; P2 = t;
    }
}

// p = z + beta p, Ap = A p on every tile; per instance p.Ap -> alpha and the FP32 checksum
__global__ void __launch_bounds__(FT, 2) kb_apply32(BatchArgs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FSlabSmem& S = *reinterpret_cast<FSlabSmem*>(smem_raw);
    const long long t = blockIdx.x;
    const int slot = B.tile2inst[t];
    if (slot < 0) return;
    const BInst& I = B.inst[slot];
    if (!I.active) return;
    BState* st = I.st;
    if (st->odone || st->done) return;
    const SlabTile T = slab_tile(I.part, t - I.tile0);
    double part[MAXQ] = {0.0, 0.0, 0.0, 0.0};
    const bool fi = fi_now(st, FI_P) || fi_now(st, FI_AP);
    if (I.uniform) {
        if (fi) kb_march32<true, true>(B, S, I, T, part);
        else kb_march32<true, false>(B, S, I, T, part);
    } else {
        if (fi) kb_march32<false, true>(B, S, I, T, part);
        else kb_march32<false, false>(B, S, I, T, part);
    }
    const long long nt = I.part.ntiles;
    double* const base = B.pa + I.tile0;
    if (!inst_arrive<MAXQ, FT>(part, base, B.ntiles, t - I.tile0, nt, &st->tick_a, S.sh, &S.last)) return;
    const double nw = __ldcg(&st->norm_wA), d1_max = __ldcg(&st->d1_max32), rho = __ldcg(&st->rho), alpha = __ldcg(&st->alpha);
    const long long applies = __ldcg(&st->applies32);
    const int stuck = __ldcg(&st->stuck);
    inst_total<MAXQ, FT, 2>(part, base, B.ntiles, nt, &st->tick_a, S.sh);
    if (threadIdx.x != 0) return;
    if (B.detect) {
        const double rel = d1_rel(part, nw);
        st->d1_last = rel;
        st->d1_max32 = fmax(d1_max, rel);
    }
    st->applies32 = applies + 1;
    if (!isfinite(part[0]) || stuck) { st->inner_bad = 1; st->done = 1; st->stuck = 0; }
    else if (fabs(part[0]) < 1e-30) { st->broken = 1; st->done = 1; }
    else { st->alpha_prev = alpha; st->alpha = __ddiv_rn(rho, part[0]); }
}

// compensated sums of one instance's partials: count (hi, lo) pairs per
// quantity, hi of quantity q at base + q*qstride, lo at base + (q+NQ)*qstride;
// RT strided sequential merges, then the block tree; valid in thread 0
template <int NQ>
__device__ __forceinline__ void inst_sums(double (&v)[NQ], const double* base, long long count, long long qstride,
                                          double (*sh)[8]) {
    constexpr int FB = 8;
    CSum acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = CSum{0.0, 0.0};
    for (long long k0 = threadIdx.x; k0 < count; k0 += (long long)RT * FB) {
        double th[NQ][FB], tl[NQ][FB];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int u = 0; u < FB; ++u) {
                const long long k = k0 + (long long)u * RT;
                th[q][u] = (k < count) ? __ldcg(base + q * qstride + k) : 0.0;
                tl[q][u] = (k < count) ? __ldcg(base + (NQ + q) * qstride + k) : 0.0;
            }
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int u = 0; u < FB; ++u)
                if (k0 + (long long)u * RT < count) csum_merge(acc[q], CSum{th[q][u], tl[q][u]});
    }
    cta_tree_csum<NQ>(acc, sh);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = csum_value(acc[q]);
}

// one block per instance: an FP64 apply's partials -> D1
template <int KIND>
__global__ void __launch_bounds__(RT) kb_final_apply(BatchArgs B) {
    __shared__ double sh[2 * MAXQ][8];
    const int slot = blockIdx.x;
    if (slot >= B.n_inst) return;
    const BInst& I = B.inst[slot];
    if (!I.active) return;
    BState* st = I.st;
    if (KIND == BK_RESID && st->odone) return;
    double p[MAXQ];
    inst_sums<MAXQ>(p, B.pa + I.tile0, I.part.ntiles, B.ntiles, sh);
    if (threadIdx.x != 0) return;
    if (B.detect) {
        const double rel = d1_rel(p, KIND == BK_RHS ? st->norm_wM : st->norm_wA);
        st->d1_last = rel;
        st->d1_max64 = fmax(st->d1_max64, rel);
    }
    st->applies64 += 1;
}

// flat block of an instance: slot, local block, first node, node count (0..KF)
struct FlatPos { int slot; long long m0; int cnt; };
__device__ __forceinline__ FlatPos flat_pos(const BatchArgs& B) {
    FlatPos f{-1, 0, 0};
    const long long g = blockIdx.x;
    if (g >= B.nflat) return f;
    const int slot = B.flat2inst[g];
    if (slot < 0) return f;
    const BInst& I = B.inst[slot];
    const long long lb = g - I.flat0;
    f.slot = slot;
    f.m0 = (lb * RT + threadIdx.x) * KF;
    const long long Nn = I.part.Nn;
    f.cnt = (f.m0 + 1 < Nn) ? 2 : (f.m0 < Nn ? 1 : 0);
    return f;
}

// residual r = b - A T in FP64 and the start of an inner solve:
// r32 = r, z32 = r32 / d, d32 = 0; partials r.r, b.b (FP64), r32.z32, r32.r32
__global__ void __launch_bounds__(RT) kb_resid(BatchArgs B) {
    __shared__ double sh[2 * MAXQ][8];
    const FlatPos f = flat_pos(B);
    CSum part[4] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    if (f.slot >= 0) {
        const BInst& I = B.inst[f.slot];
        if (I.active && !I.st->odone) {
            for (int k = 0; k < f.cnt; ++k) {
                const long long m = f.m0 + k;
                const double bv = I.b[m];
                const double rv = dsub(bv, I.y64[m]);
                I.r64[m] = rv;
                const float r32 = (float)rv;
                const float z = __fmul_rn(r32, I.dinv32[m]);
                I.r32[m] = r32; I.z32[m] = z; I.d32[m] = 0.f;
                csum_fma(part[0], rv, rv);
                csum_fma(part[1], bv, bv);
                csum_add(part[2], dmul((double)r32, (double)z));     // products of FP32 values are exact
                csum_add(part[3], dmul((double)r32, (double)r32));
            }
        }
    }
    cta_tree_csum<4>(part, sh);
    if (threadIdx.x == 0 && blockIdx.x < B.nflat) store_cpartials<4>(part, B.pf, B.nflat, blockIdx.x);
}

// one block per instance: outer convergence test and the inner solve's start
__global__ void __launch_bounds__(RT) kb_outer_final(BatchArgs B) {
    __shared__ double sh[2 * MAXQ][8];
    const int slot = blockIdx.x;
    if (slot >= B.n_inst) return;
    const BInst& I = B.inst[slot];
    if (!I.active) return;
    BState* st = I.st;
    if (st->odone) return;
    double p[4];
    inst_sums<4>(p, B.pf + I.flat0, I.part.nflat, B.nflat, sh);
    if (threadIdx.x != 0) return;
    if (st->outer == 0) {
        double bn = __dsqrt_rn(p[1]);
        if (bn < 1e-30) bn = 1.0;
        st->bn64 = bn;
    }
    st->rel64 = __ddiv_rn(__dsqrt_rn(p[0]), st->bn64);
    const bool conv = st->rel64 < B.rtol;
    if (conv || st->outer >= B.max_outer) {
        if (!conv) st->stalls += 1;
        st->odone = 1; st->done = 1;
        return;
    }
    st->outer += 1;
    st->outer_total += 1;
    st->rho = p[2];
    st->bn_in = __dsqrt_rn(p[3]);
    // solve only as far as the outer target needs: max(inner_tol, rtol / (2 rel64))
    st->tol_in = fmax(B.inner_tol, __ddiv_rn(0.5 * B.rtol, st->rel64));
    st->iter = 0; st->broken = 0; st->beta = 0.0; st->inner_bad = 0; st->pend = 0;
    st->done = (st->bn_in < 1e-300 || !isfinite(st->bn_in) || !isfinite(p[2])) ? 1 : 0;
    if (!isfinite(st->bn_in) || !isfinite(p[2])) st->inner_bad = 1;
}

// ---- the FP32 inner loop: vector update ----------------------------------------------
// r -= alpha Ap, z = r / diag; r.r and r.z; and at odd iterations d += alpha p
// for the previous iteration and this one (the same two multiply-adds in the
// same order; the previous p is still in the other buffer), which saves 4 of 32
// bytes per node on average.  The unit is a round of UR consecutive nodes (UV groups
// of four per thread, their loads in flight together) with its own block tree and
// partial sums, so an instance's bits do not depend on how rounds are dealt to
// blocks.  The last block of an instance to finish adds up its rounds' sums and does
// the inner solve's scalar step (beta, convergence).
//
// Rounds per block, by the rounds of all instances: one while they are resident at
// once (148 SMs of 4 blocks), two up to twice as many, else four.  Few are bound by
// latency, and a further round in a block is one more chain of loads on a mostly idle
// GPU; many by the memory, and then by the fence and ticket that each block costs.
// Device ms of 4 steps (B200) with one | two | four rounds: 2 instances at N=16 2.45 |
// 2.50 | 2.77, 2 at N=64 (268 rounds) 6.99 | 7.23 | 7.84, one at N=104 (566) 10.4 | 10.5 |
// 11.2, one at N=112 (705) 14.0 | 13.3 | 13.8, 16 at N=48 (928) 9.08 | 8.74 | 9.28, 12 of
// N=30..65 9.65 | 9.32 | 9.80, one at N=128 (1049) 14.5 | 14.1 | 14.7, one at N=140 (1369)
// 20.0 | 19.8 | 18.9, 16 at N=96 78.4 | 75.1 | 74.7, 256 of N=17..92 315 | 296 | 288.
constexpr int UV = 2, UR = RT * 4 * UV, UMAX = 4, kUpdBlocks = 148 * 4;
inline int upd_rounds(long long all) { return all <= kUpdBlocks ? 1 : all <= 2 * kUpdBlocks ? 2 : UMAX; }
__global__ void __launch_bounds__(RT, 4) kb_update32(BatchArgs B) {
    __shared__ double sh[2][16];
    __shared__ double shr[UMAX][2][RT / 32];
    __shared__ unsigned s_last;
    const int slot = B.chunk2inst[blockIdx.x];
    if (slot < 0) return;
    const BInst& I = B.inst[slot];
    BState* st = I.st;
    if (!I.active || st->odone || st->done) return;
    const long long Nn = I.part.Nn, nround = (Nn + UR - 1) / UR;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rounds = I.rounds;
    const long long round0 = (blockIdx.x - I.chunk0) * rounds;
    const float alpha = (float)st->alpha;
    const bool odd = st->iter & 1;
    const float alpha_prev = odd ? (float)st->alpha_prev : 0.f;
    const bool fr = fi_now(st, FI_RV);
    const long long fi_idx = fr ? st->fi_idx : -1;
    // four nodes from m on (the buffers are 256-byte aligned, m a multiple of 4); the end of the grid one by one
    auto ld4 = [&](const float* v, long long m) {
        if (m + 3 < Nn) return *reinterpret_cast<const float4*>(v + m);
        return make_float4(m < Nn ? v[m] : 0.f, m + 1 < Nn ? v[m + 1] : 0.f, m + 2 < Nn ? v[m + 2] : 0.f, 0.f);
    };
    auto st4 = [&](float* v, long long m, float4 x) {
        if (m + 3 < Nn) { *reinterpret_cast<float4*>(v + m) = x; return; }
        if (m < Nn) v[m] = x.x;
        if (m + 1 < Nn) v[m + 1] = x.y;
        if (m + 2 < Nn) v[m + 2] = x.z;
    };
    float4 dv[UV], pv[UV], ov[UV], qv[UV], rv[UV], iv[UV];
    for (int ul = 0; ul < rounds; ++ul) {
        const long long m0 = (round0 + ul) * UR + threadIdx.x * 4;
        double part[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const long long m = m0 + u * (RT * 4);
            qv[u] = ld4(I.Ap32, m); rv[u] = ld4(I.r32, m); iv[u] = ld4(I.dinv32, m);
            if (odd) { dv[u] = ld4(I.d32, m); pv[u] = ld4(I.p32b, m); ov[u] = ld4(I.p32a, m); }
        }
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const long long m = m0 + u * (RT * 4);
            float4 zv;
            if (odd) {
                auto add = [&](float& d, float po, float pk) { d = __fmaf_rn(alpha, pk, __fmaf_rn(alpha_prev, po, d)); };
                add(dv[u].x, ov[u].x, pv[u].x); add(dv[u].y, ov[u].y, pv[u].y);
                add(dv[u].z, ov[u].z, pv[u].z); add(dv[u].w, ov[u].w, pv[u].w);
                st4(I.d32, m, dv[u]);
            }
            auto one = [&](int k, float q, float& r, float inv, float& z) {
                r = __fmaf_rn(-alpha, q, r);
                if (fr && m + k == fi_idx) { r = flipf(r, st->fi_bit); st->fi_fired = 1; }
                z = __fmul_rn(r, inv);
                // products of FP32 values are exact in FP64; plain FP64 sums suffice
                // for the inner solve's 1e-4 relative tolerance
                part[0] = dfma((double)r, (double)r, part[0]);
                part[1] = dfma((double)r, (double)z, part[1]);
            };
            one(0, qv[u].x, rv[u].x, iv[u].x, zv.x);
            one(1, qv[u].y, rv[u].y, iv[u].y, zv.y);
            one(2, qv[u].z, rv[u].z, iv[u].z, zv.z);
            one(3, qv[u].w, rv[u].w, iv[u].w, zv.w);
            st4(I.r32, m, rv[u]); st4(I.z32, m, zv);
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
            for (int q = 0; q < 2; ++q) part[q] = dadd(part[q], __shfl_xor_sync(0xffffffffu, part[q], off));
        if (lane == 0) { shr[ul][0][warp] = part[0]; shr[ul][1][warp] = part[1]; }
    }
    __syncthreads();
    // the rounds' trees over the warp sums, two rounds of two quantities at a time; one
    // partial per round (a quarter of the flat blocks), from the instance's flat0 on
    double* const base = B.pf + I.flat0;
    if (warp == 0) {
        for (int h = 0; h < rounds; h += 2) {
            const int ul = h + (lane >> 4), q = (lane >> 3) & 1;
            double v = shr[ul][q][lane & 7];
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) v = dadd(v, __shfl_xor_sync(0xffffffffu, v, off));
            if ((lane & 7) == 0 && ul < rounds && round0 + ul < nround) base[q * B.nflat + round0 + ul] = v;
        }
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            s_last = atomicAdd(&st->tick_u, 1u) == (unsigned)(I.nchunk - 1) ? 1u : 0u;
        }
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const double bn_in = __ldcg(&st->bn_in), tol_in = __ldcg(&st->tol_in), rho = __ldcg(&st->rho);
    const long long total = __ldcg(&st->inner_total);
    const int iter = __ldcg(&st->iter);
    double part[2];
    inst_total<2, RT, 8>(part, base, B.nflat, nround, &st->tick_u, sh);
    if (threadIdx.x != 0) return;
    st->inner_total = total + 1;
    st->pend = iter & 1 ? 0 : 1;
    const double rel = __ddiv_rn(__dsqrt_rn(part[0]), bn_in);
    if (!isfinite(rel) || !isfinite(part[1])) { st->inner_bad = 1; st->done = 1; return; }
    if (rel < tol_in || iter + 1 >= B.max_inner) { st->done = 1; return; }
    st->beta = __ddiv_rn(part[1], rho);
    st->rho = part[1];
    st->iter = iter + 1;
}

// T += d (FP64) at the interior nodes, for the instances whose inner solve
// just finished; Dirichlet values are never changed, and a correction from an
// inner solve that went non-finite is discarded (the next correction re-solves)
__global__ void __launch_bounds__(RT) kb_correct(BatchArgs B) {
    const FlatPos f = flat_pos(B);
    if (f.slot < 0) return;
    const BInst& I = B.inst[f.slot];
    if (!I.active || I.st->odone || I.st->inner_bad) return;
    const int N = I.part.N;
    // an even last iteration's p is in p32a (a later p, if any, went to p32b)
    const bool pend = I.st->pend != 0;
    const float alpha = (float)I.st->alpha;
    for (int k = 0; k < f.cnt; ++k) {
        const long long m = f.m0 + k;
        if (is_bnd(m, N)) continue;
        const float d = pend ? __fmaf_rn(alpha, I.p32a[m], I.d32[m]) : I.d32[m];
        I.T[m] = dadd(I.T[m], (double)d);
    }
}

// count the discarded inner solves (one thread per instance, after kb_correct)
__global__ void kb_count_bad(BatchArgs B) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= B.n_inst) return;
    const BInst& I = B.inst[slot];
    if (!I.active || I.st->odone) return;
    if (I.st->inner_bad) I.st->inner_faults += 1;
}

// set-up helpers: FP32 reciprocal of the diagonal; the interior indicator
__global__ void k_recip32(long long n, const double* d, float* out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = (float)__ddiv_rn(1.0, d[i]);
}
// interleaved FP64 and FP32 element coefficients (rho*c, k); uniform rho*c: k alone in FP32
__global__ void k_pack_coef(long long ne, const double* rhoc, const double* k, double2* c64, float2* c32, float* k32) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += (long long)gridDim.x * blockDim.x) {
        const double r = rhoc[i], kk = k[i];
        c64[i] = make_double2(r, kk);
        if (k32) k32[i] = __double2float_rn(kk);
        else c32[i] = make_float2(__double2float_rn(r), __double2float_rn(kk));
    }
}
// fresh state of an added instance: checksum weight norms from their squared sums, nothing to iterate
__global__ void kb_init_state(BState* st, const double* sq) {
    BState s{};
    s.norm_wM = __dsqrt_rn(sq[0]);
    s.norm_wA = __dsqrt_rn(sq[2]);
    s.odone = 1; s.done = 1;
    *st = s;
}
__global__ void k_ones_interior(int N, double* v) {
    const long long NN = N + 1, Nn = NN * NN * NN;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < Nn; i += (long long)gridDim.x * blockDim.x)
        v[i] = is_bnd(i, N) ? 0.0 : 1.0;
}

// arm (vec > 0) or disarm (vec == 0) the vector fault of one instance
__global__ void kb_arm(BState* st, int vec, int outer, int iter, long long idx, int bit) {
    st->fi_vec = vec; st->fi_outer = outer; st->fi_iter = iter; st->fi_idx = idx; st->fi_bit = bit;
}

// step start: outer state of every active instance
__global__ void kb_step_begin(BatchArgs B) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= B.n_inst) return;
    const BInst& I = B.inst[slot];
    if (!I.active) return;
    BState* st = I.st;
    st->outer = 0; st->odone = 0; st->done = 1; st->iter = 0;
    st->extrap = B.extrapolate && st->has_prev;
    st->has_prev = 1;
}

// start of the step's solve (after b = M T): T <- 2 T - T_prev where a
// previous field exists, else T unchanged; T_prev <- T of this step's start
__global__ void __launch_bounds__(RT) kb_extrapolate(BatchArgs B) {
    const FlatPos f = flat_pos(B);
    if (f.slot < 0 || !B.extrapolate) return;
    const BInst& I = B.inst[f.slot];
    if (!I.active) return;
    const bool ex = I.st->extrap;
    for (int k = 0; k < f.cnt; ++k) {
        const long long m = f.m0 + k;
        const double t = I.T[m];
        if (ex) I.T[m] = dfma(2.0, t, -I.Tm1[m]);
        I.Tm1[m] = t;
    }
}

// loop conditions: any active instance still in its outer loop (WHICH 0) /
// in an inner solve (WHICH 1)
template <int WHICH>
__global__ void kb_cond(BatchArgs B, cudaGraphConditionalHandle h, int* flag) {
    int any = 0;
    for (int s = threadIdx.x; s < B.n_inst; s += blockDim.x) {
        const BInst& I = B.inst[s];
        if (!I.active) continue;
        const BState* st = I.st;
        if (WHICH == 0 ? !st->odone : (!st->odone && !st->done)) any = 1;
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        if (flag) *flag = any;                      // direct launches: the host reads the flag
        else cudaGraphSetConditional(h, any ? 1u : 0u);
    }
}

}  // namespace hs
