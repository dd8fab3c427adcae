// hs_pcg.cuh -- a whole PCG solve of a small grid as one cooperative kernel
// (included by hs_solver.cu).
//
// On a small grid a CG iteration's work takes a microsecond or two, and the
// two launches of the graph's while body 17 to 20 us (B200, N = 8..48): the
// time goes into the launches' ramp-up, the geometry and the loads that each
// launch repeats, and chains of memory latencies.  Here the CTAs stay: CTA c
// owns slab tile c (operator) and run c of the vector update, one flat block
// of 512 nodes (up to three runs where there are more runs than tiles), and
// keeps
//   * p on its tile and halo planes in shared memory, where the next iteration
//     forms p = z + beta p in place (halo values by the same operations as
//     their owner, so the same bits);
//   * r, d and x of its block's nodes in registers.
// Only z, Ap and p cross CTAs, through the L2.
//
// Two exchanges per iteration order the phases.  An exchange is not a barrier
// followed by loads of partial sums: each CTA publishes its partial sum and a
// tag in one 16-byte word after its vectors are visible, and every CTA polls
// the words it sums.  So a partial's arrival is the barrier.  Every CTA then
// finishes the reduction itself, in the canonical order: alpha, beta and the
// convergence decision are the same bits everywhere.  The solution update and
// the checksum run while the next exchange is in flight.
#pragma once
#include <type_traits>

#include "hs_kernels.cuh"

namespace hs {

// ---- exchange words ------------------------------------------------------------
struct __align__(16) XWord { double v; unsigned long long tag; };
__device__ __forceinline__ void xput(XWord* w, double v, unsigned long long tag) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(w),
                 "l"(__double_as_longlong(v)), "l"(tag)
                 : "memory");
}
__device__ __forceinline__ void xget(const XWord* w, double& v, unsigned long long& tag) {
    long long a;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(tag)
                 : "l"(w)
                 : "memory");
    v = __longlong_as_double(a);
}

// Before the words of many CTAs are read, one thread waits for their count:
// with 294 CTAs polling 294 words each, the polls themselves held the words up
// (N=48: 10 us of an 18 us iteration).  A solve with the gate | without it, us:
// N=16 (10 CTAs) 190 | 184, 24 (31) 280 | 279, 27 (43) 293 | 303, 29 (53) 310 | 344,
// 36 (99) 370 | 513, 47 (288) 597 | 886, 71 (252) 1175 | 1450.
constexpr int kGateCtas = 48;
__device__ __forceinline__ void xgate(const unsigned* count, unsigned target) {
    if (threadIdx.x == 0) {
        unsigned v, left = kPolls;
        do {
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        } while ((int)(v - target) < 0 && --left);
    }
    __syncthreads();
}

// Wait for n words per quantity (quantity q's at words + q * n), each thread for
// words tid, tid + RT, ... (at most FB), and add them up per thread in that
// order.  Afterwards everything their writers stored before publishing is
// visible to the CTA.  False: gave up.
template <int NQ, int FB>
__device__ __forceinline__ bool xwait(double (&v)[NQ], const XWord* words, int n, unsigned long long tag,
                                      unsigned* s_bad) {
    double t[NQ][FB];
    unsigned left = kPolls;
    bool ok;
    do {
        ok = true;
#pragma unroll
        for (int u = 0; u < FB; ++u) {
            const int k = threadIdx.x + u * RT;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                t[q][u] = 0.0;
                if (k < n) {
                    unsigned long long g;
                    xget(words + (long long)q * n + k, t[q][u], g);
                    ok = ok && g == tag;
                }
            }
        }
    } while (!ok && --left);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (!ok) *s_bad = 1u;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        v[q] = 0.0;
#pragma unroll
        for (int u = 0; u < FB; ++u)
            if ((int)threadIdx.x + u * RT < n) v[q] = dadd(v[q], t[q][u]);
    }
    __syncthreads();
    return *s_bad == 0u;
}
// The block tree over the RT values with the result in every thread: each warp
// runs the second stage itself on the eight warp sums (a xor butterfly gives
// every lane the same bits).  sh is free again after the next CTA barrier.
template <int NQ>
__device__ __forceinline__ void xtree(double (&v)[NQ], double (*sh)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = dadd(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) sh[q][warp] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = sh[q][lane & 7];
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = dadd(v[q], __shfl_xor_sync(0xffffffffu, v[q], off));
}

constexpr int kPcgRuns = 3;      // runs of one CTA at most

struct PcgArgs {
    Part part;
    double dt, dtF;
    const double2* coef;
    const double* wM;
    const double* wA;
    const double* F;         // source (null: none)
    const double* d;         // Jacobi diagonal
    double* x;               // T: start and solution
    double* b;
    double* r;               // (RU > 1)
    double* z;
    double* Ap;
    double* pbuf0;           // p_k in pbuf[k & 1]
    double* pbuf1;
    XWord* xa;               // tile words: [2 parities][nblk]
    XWord* xr;               // run words: [2 parities][3][nruns]
    unsigned* count;         // words published: [0] tiles, [32] runs (k_step_begin zeroes them)
    double* dparts;          // checksum partials: [3 sets][3][nblk]
    unsigned long long tag;  // this launch's first tag
    DevState* st;
    int with_rhs, nruns, d1;
    int fail_waits;          // every wait counts as given up (tests)
    ElemConsts ec;
};

// shared memory: PP planes xa-1..xb+1 of the operator's input vector, then the
// hand-over buffers (as SlabSmem's)
struct PcgSmem {
    double2 MK[64];                            // the dense form's (M^_ij, K^_ij)
    double2 Y1[SPOS], Y2[SPOS], Y3[SPOS];      // (a gather of a position without an element may read into Y1)
};
inline size_t pcg_smem(int CX) { return (size_t)(CX + 2) * SPOS * sizeof(double) + sizeof(PcgSmem); }

// elem_fast with the matrices in shared memory, outputs v[q] for Q0 <= q < Q1
// only.  One broadcast load per entry and element: as kernel parameters, or
// shared between elements, the compiler keeps the constants of the unrolled
// element in registers and spills them.
template <int Q0, int Q1>
__device__ __forceinline__ void elem_fast_smem(double* v, double rhoc, double dk, const double2* MK) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(MK);
    double xl[8], yl[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) xl[i] = v[q_of_local(i)];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (q_of_local(i) < Q0 || q_of_local(i) >= Q1) continue;
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            double m, kk;
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(m), "=d"(kk) : "r"(base + (i * 8 + j) * 16));
            acc = dfma(dfma(rhoc, m, dmul(dk, kk)), xl[j], acc);
        }
        yl[i] = acc;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (q_of_local(i) >= Q0 && q_of_local(i) < Q1) v[q_of_local(i)] = yl[i];
}

// Operator on the planes in shared memory (layers as in slab_march): y, the
// stored p (loop) and the thread's partial sums.  cf: the first layer's
// coefficients, loaded by the caller.  NK: positions per thread.
template <int FORM, int NK>
__device__ __forceinline__ void pcg_apply(const PcgArgs& a, double* PP, PcgSmem& S, const SlabTile& T, const SlabPos& G,
                                          double2 (&cf)[NK], double dt_eff, const double* w, const double* F,
                                          double* yout, double* pout, bool fi_ap, bool fi_r, int fi_bit,
                                          long long fi_idx, long long fi_elem, double (&part)[MAXQ]) {
    const Part& P = a.part;
    const int N = P.N, Cw = P.Cw, tid = threadIdx.x;
    const unsigned plane = (unsigned)P.NN * (unsigned)P.NN, eplane = (unsigned)N * (unsigned)N;
    const unsigned fl = G.fl;
    const bool d1 = a.d1 != 0;
    double ac[NK], an[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) ac[k] = 0.0;
    auto layer = [&](int ix, auto first_, auto last_) {
        // the first layer completes no node, the last starts none
        constexpr bool FIRST = decltype(first_)::value, LAST = decltype(last_)::value;
        const double* P0 = PP + (ix - T.xa + 1) * SPOS;
        const double* P1 = P0 + SPOS;
        double wv[NK], fv[NK];
        double2 cn[NK];
#pragma unroll
        for (int k = 0; k < NK; ++k) {
            const bool o = !FIRST && sp_out(fl, k);
            const unsigned n = (unsigned)ix * plane + (unsigned)G.noff[k];
            wv[k] = (o && d1) ? __ldg(w + n) : 0.0;
            fv[k] = (o && F) ? __ldg(F + n) : 0.0;
            const bool e = !LAST && ix + 1 < N && sp_elem(fl, k);
            cn[k] = e ? __ldg(a.coef + ((unsigned)(ix + 1) * eplane + (unsigned)G.eoff[k])) : make_double2(0.0, 0.0);
        }
        if (ix >= 0 && ix < N) {
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                const int j = tid + k * ST;
                double v[8];
                v[0] = P0[j]; v[1] = P0[j + 1]; v[2] = P0[j + Cw]; v[3] = P0[j + Cw + 1];
                v[4] = P1[j]; v[5] = P1[j + 1]; v[6] = P1[j + Cw]; v[7] = P1[j + Cw + 1];
                if constexpr (FORM == FORM_FAST) elem_fast_smem<FIRST ? 4 : 0, LAST ? 4 : 8>(v, cf[k].x, dmul(dt_eff, cf[k].y), S.MK);
                else elem_apply<FORM>(v, cf[k].x, cf[k].y, dt_eff, a.ec);
                if (fi_r && (long long)ix * eplane + G.eoff[k] == fi_elem) v[0] = flipbit(v[0], fi_bit);
                if (!FIRST) ac[k] = dadd(ac[k], v[0]);
                if (!LAST) an[k] = dadd(0.0, v[4]);
                if (sp_elem(fl, k)) {
                    if (FIRST) {          // only the upper corners' sums are this tile's
                        S.Y1[j + 1].y = v[5]; S.Y2[j + Cw].y = v[6]; S.Y3[j + Cw + 1].y = v[7];
                    } else if (LAST) {
                        S.Y1[j + 1].x = v[1]; S.Y2[j + Cw].x = v[2]; S.Y3[j + Cw + 1].x = v[3];
                    } else {
                        S.Y1[j + 1] = make_double2(v[1], v[5]);
                        S.Y2[j + Cw] = make_double2(v[2], v[6]);
                        S.Y3[j + Cw + 1] = make_double2(v[3], v[7]);
                    }
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < NK; ++k) an[k] = 0.0;
        }
        __syncthreads();
        const bool xbnd = ix == 0 || ix == N;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
            if (sp_out(fl, k)) {
                const int j = tid + k * ST;
                const bool yzin = !sp_yzb(fl, k);
                const double2 zero = make_double2(0.0, 0.0);
                double2 y3 = zero, y2 = zero, y1 = zero;
                if (yzin) { y3 = S.Y3[j]; y2 = S.Y2[j]; y1 = S.Y1[j]; }
                if (!FIRST) {
                    const unsigned n = (unsigned)ix * plane + (unsigned)G.noff[k];
                    const bool bnd = !yzin || xbnd;
                    double y = bnd ? 0.0 : dadd(dadd(dadd(ac[k], y3.x), y2.x), y1.x);
                    if (fi_ap && (long long)n == fi_idx) y = flipbit(y, fi_bit);
                    const double pv = P0[j];
                    if (pout) part[0] = dfma(pv, y, part[0]);
                    if (d1) {
                        part[1] = bnd ? dfma(0.0, y, part[1]) : dadd(part[1], y);
                        part[2] = dfma(wv[k], pv, part[2]);
                        part[3] = dfma(pv, pv, part[3]);
                    }
                    if (F) y = dfma(a.dtF, fv[k], y);
                    yout[n] = y;
                    if (pout) pout[n] = pv;
                }
                if (!LAST) ac[k] = yzin ? dadd(dadd(dadd(an[k], y3.y), y2.y), y1.y) : 0.0;
            }
            cf[k] = cn[k];
        }
        if (!LAST) __syncthreads();
    };
    using std::false_type; using std::true_type;
    layer(T.xa - 1, true_type{}, false_type{});
    for (int ix = T.xa; ix < T.xb; ++ix) layer(ix, false_type{}, false_type{});
    layer(T.xb, false_type{}, true_type{});
}

template <int FORM, int NK, int RU>
__global__ void __launch_bounds__(ST, FORM == FORM_GAUSS ? 1 : 2) k_pcg(PcgArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* const PP = reinterpret_cast<double*>(smem_raw);
    PcgSmem& S = *reinterpret_cast<PcgSmem*>(smem_raw + (size_t)(a.part.CX + 2) * SPOS * sizeof(double));
    __shared__ double sh[2][MAXQ][8];
    __shared__ unsigned s_bad;
    DevState* const st = a.st;
    const int c = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    const Part& P = a.part;
    const int nblk = (int)P.nblk, nruns = a.nruns;
    const bool det = a.d1 != 0;
    const bool tile = c < nblk, run = c < nruns;
    const bool d1_cta = det && c == G - 1;
    if (tid == 0) s_bad = a.fail_waits ? 1u : 0u;
    if (FORM == FORM_FAST && tid < 64) S.MK[tid] = make_double2(a.ec.M[tid], a.ec.K[tid]);
    const double tol = st->tol, norm_wA = st->norm_wA;
    const int max_iter = st->max_iter;
    const int fi_vec = st->fi_vec, fi_iter = st->fi_iter, fi_bit = st->fi_bit;
    const long long fi_idx = st->fi_idx;
    unsigned long long tag = a.tag;
    const bool gate = G > kGateCtas;
    unsigned want_a = 0, want_r = 0;        // counts of the gates

    // ---- the tile: geometry, and the input's planes --------------------------------
    SlabTile T{};
    SlabPos Q{};
    if (tile) { T = slab_tile(P, c); Q = slab_pos(P, T, tid); }
    const int N = P.N;
    const unsigned plane = (unsigned)P.NN * (unsigned)P.NN, eplane = (unsigned)N * (unsigned)N;
    const int npl = tile ? T.xb - T.xa + 3 : 0;          // planes xa-1 .. xb+1
    auto ld_z = [&](const double* src, int pl, double (&v)[NK]) {
        const int px = T.xa - 1 + pl;
        const bool pv = pl < npl && px >= 0 && px <= N;
#pragma unroll
        for (int k = 0; k < NK; ++k)
            v[k] = (pv && sp_valid(Q.fl, k)) ? __ldcg(src + ((unsigned)px * plane + (unsigned)Q.noff[k])) : 0.0;
    };
    auto ld_coef = [&](double2 (&cf)[NK]) {
        const int ex = T.xa - 1;
#pragma unroll
        for (int k = 0; k < NK; ++k)
            cf[k] = (tile && ex >= 0 && sp_elem(Q.fl, k)) ? __ldg(a.coef + ((unsigned)ex * eplane + (unsigned)Q.eoff[k]))
                                                          : make_double2(0.0, 0.0);
    };
    // ---- the runs c, c + G, ...: one flat block each, a pair of nodes per thread --------
    // r, d and x stay in registers for one run; for RU > 1 the thread's own
    // entries are re-read from the L2 (36 registers more would spill)
    constexpr bool KEEP = RU == 1;
    auto node0 = [&](int u) { return ((long long)(c + u * G) * RT + tid) * KF; };
    auto count = [&](int u) {
        const long long m = node0(u);
        return c + u * G >= nruns ? 0 : (m + 1 < P.Nn) ? 2 : (m < P.Nn ? 1 : 0);
    };
    auto ld2 = [&](const double* base, int u) {          // vectors written in this launch
        const long long m = node0(u);
        const int cnt = count(u);
        if (cnt == 2) return __ldcg(reinterpret_cast<const double2*>(base + m));
        return make_double2(cnt ? __ldcg(base + m) : 0.0, 0.0);
    };
    auto st2 = [&](double* base, int u, double2 v) {
        const long long m = node0(u);
        const int cnt = count(u);
        if (cnt == 2) *reinterpret_cast<double2*>(base + m) = v;
        else if (cnt) base[m] = v.x;
    };
    double2 dd[RU], xx[RU], rr[RU];
#pragma unroll
    for (int u = 0; u < RU; ++u) {
        rr[u] = make_double2(0.0, 0.0);
        if (KEEP) { dd[u] = ld2(a.d, u); xx[u] = ld2(a.x, u); }
    }
    // the tree of each run's sums, published (all runs of the CTA behind one fence)
    auto put_runs = [&](auto& part, int par) {
        constexpr int NQ = sizeof(part[0]) / sizeof(double);
#pragma unroll
        for (int u = 0; u < RU; ++u)
            if (u == 0 || c + u * G < nruns) cta_tree_sum<NQ>(part[u], sh[0]);
        if (tid == 0) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
            for (int u = 0; u < RU; ++u)
                if (c + u * G < nruns) {
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        xput(a.xr + (long long)(par * 3 + q) * nruns + c + u * G, part[u][q], tag);
                    if (gate) atomicAdd(a.count + 32, 1u);
                }
        }
    };

    // publish the tile's partials of an application / the run's sums
    auto put_tile = [&](double (&part)[MAXQ], int set, int par) {
        cta_tree_sum<MAXQ>(part, sh[0]);
        if (tid == 0) {
            if (det) {
#pragma unroll
                for (int q = 1; q < MAXQ; ++q) a.dparts[((long long)set * 3 + q - 1) * nblk + c] = part[q];
            }
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            xput(a.xa + (long long)par * nblk + c, part[0], tag);
            if (gate) atomicAdd(a.count, 1u);
        }
    };
    auto checksum = [&](int set, double nw) {
        double q[3];
        final_sums<3, 2>(q, a.dparts + (long long)set * 3 * nblk, nblk, sh[1]);
        if (tid == 0) {
            const double nx = __dsqrt_rn(q[2]);
            double rel = __ddiv_rn(fabs(dsub(q[0], q[1])), dfma(nw, nx, 1e-300));
            if (!isfinite(rel)) rel = 1e300;
            st->d1_last = rel;
            st->d1_step = fmax(st->d1_step, rel);
        }
    };
    auto stuck = [&]() { if (tid == 0) st->stuck = 1; };        // (k_step_end tells the host)

    // ---- b = M T + dt F and Ap = A T -------------------------------------------------
    double2 cf[NK];
    if (tile) {
        for (int pl = 0; pl < npl; ++pl) {
            double v[NK];
            ld_z(a.x, pl, v);
#pragma unroll
            for (int k = 0; k < NK; ++k) PP[pl * SPOS + tid + k * ST] = v[k];
        }
        __syncthreads();
        if (a.with_rhs) {
            double part[MAXQ] = {0.0, 0.0, 0.0, 0.0};
            ld_coef(cf);
            pcg_apply<FORM, NK>(a, PP, S, T, Q, cf, 0.0, a.wM, a.F, a.b, nullptr, false, false, 0, -1, -1, part);
            cta_tree_sum<MAXQ>(part, sh[0]);
            if (tid == 0) {
#pragma unroll
                for (int q = 1; q < MAXQ; ++q) a.dparts[((long long)2 * 3 + q - 1) * nblk + c] = part[q];
            }
        }
        double part[MAXQ] = {0.0, 0.0, 0.0, 0.0};
        const bool fi_r = st->fi_armR != 0;
        ld_coef(cf);
        pcg_apply<FORM, NK>(a, PP, S, T, Q, cf, a.dt, a.wA, nullptr, a.Ap, nullptr, false, fi_r, fi_bit, -1,
                            fi_r ? st->fi_elem : -1, part);
        ++tag;
        put_tile(part, 1, 1);
    } else {
        ++tag;
    }
    {
        double v[1];
        want_a += nblk;
        if (gate) xgate(a.count, want_a);
        if (!xwait<1, 2>(v, a.xa + nblk, nblk, tag, &s_bad)) { stuck(); return; }
    }
    // ---- prologue: r = b - Ap, z = r / d -----------------------------------------------
    ++tag;
    if (run) {
        double part[RU][3];
#pragma unroll
        for (int u = 0; u < RU; ++u) {
            const int cnt = count(u);
            const double2 bb = ld2(a.b, u), qq = ld2(a.Ap, u);
            if (!KEEP) dd[u] = ld2(a.d, u);
            double2 zz = make_double2(0.0, 0.0);
            part[u][0] = part[u][1] = part[u][2] = 0.0;
            auto one = [&](double b, double q, double d, double& r, double& z) {
                r = dfma(-1.0, q, b);
                z = __ddiv_rn(r, d);
                part[u][0] = dfma(b, b, part[u][0]);
                part[u][1] = dfma(r, z, part[u][1]);
                part[u][2] = dfma(r, r, part[u][2]);
            };
            if (cnt > 0) one(bb.x, qq.x, dd[u].x, rr[u].x, zz.x);
            if (cnt > 1) one(bb.y, qq.y, dd[u].y, rr[u].y, zz.y);
            st2(a.z, u, zz);
            if (!KEEP) st2(a.r, u, rr[u]);
        }
        put_runs(part, 1);
    }
    if (d1_cta) {
        if (a.with_rhs) checksum(2, st->norm_wM);
        checksum(1, norm_wA);
    }
    double bnorm, rho, beta = 0.0, alpha = 0.0, pAp = 0.0;
    {
        double v[3];
        want_r += nruns;
        if (gate) xgate(a.count + 32, want_r);
        if (!xwait<3, 3>(v, a.xr + (long long)3 * nruns, nruns, tag, &s_bad)) { stuck(); return; }
        xtree<3>(v, sh[1]);
        bnorm = __dsqrt_rn(v[0]);
        if (bnorm < 1e-30) bnorm = 1.0;
        rho = v[1];
        if (c == 0 && tid == 0) st->rel0 = __ddiv_rn(__dsqrt_rn(v[2]), bnorm);
    }

    // ---- CG iterations -------------------------------------------------------------------
    constexpr int ZP = 3;                       // planes of z loaded ahead of beta (all of them for CX = 1)
    double zv[ZP][NK];
#pragma unroll
    for (int pl = 0; pl < ZP; ++pl) ld_z(a.z, pl, zv[pl]);
    ld_coef(cf);
    int iter = 0, result = 0, broken = 0;
    bool done = max_iter <= 0;
    while (!done) {
        double* const p = (iter & 1) ? a.pbuf1 : a.pbuf0;
        const int par = iter & 1;
        const bool fi = fi_vec != 0 && fi_iter == iter;
        ++tag;
        if (tile) {
            // p = z + beta p on every plane (k = 0: p = z), in place
            auto form = [&](int pl, double (&v)[NK]) {
#pragma unroll
                for (int k = 0; k < NK; ++k) {
                    double* q = PP + pl * SPOS + tid + k * ST;
                    double pv = iter > 0 ? dfma(beta, *q, v[k]) : v[k];
                    if (fi && fi_vec == FI_P && sp_valid(Q.fl, k) &&
                        (long long)(T.xa - 1 + pl) * plane + Q.noff[k] == fi_idx)
                        pv = flipbit(pv, fi_bit);
                    *q = pv;
                }
            };
#pragma unroll
            for (int pl = 0; pl < ZP; ++pl) form(pl, zv[pl]);
            for (int pl = ZP; pl < npl; ++pl) {
                double v[NK];
                ld_z(a.z, pl, v);
                form(pl, v);
            }
            __syncthreads();
            double part[MAXQ] = {0.0, 0.0, 0.0, 0.0};
            pcg_apply<FORM, NK>(a, PP, S, T, Q, cf, a.dt, a.wA, nullptr, a.Ap, p, fi && fi_vec == FI_AP, false, fi_bit,
                                fi_idx, -1, part);
            put_tile(part, par, par);
            ld_coef(cf);                        // the next iteration's first layer
        }
        {
            if (!KEEP) {
#pragma unroll
                for (int u = 0; u < RU; ++u) { rr[u] = ld2(a.r, u); dd[u] = ld2(a.d, u); }
            }
            double v[1];
            want_a += nblk;
            if (gate) xgate(a.count, want_a);
            if (!xwait<1, 2>(v, a.xa + (long long)par * nblk, nblk, tag, &s_bad)) { stuck(); return; }
            double2 qq[RU];
#pragma unroll
            for (int u = 0; u < RU; ++u) qq[u] = ld2(a.Ap, u);
            xtree<1>(v, sh[1]);
            pAp = v[0];
            if (fabs(pAp) < 1e-30) {            // breakdown: the reference stops before the update
                if (d1_cta) { __syncthreads(); checksum(par, norm_wA); }
                broken = 1; result = iter;
                break;
            }
            alpha = __ddiv_rn(rho, pAp);
            ++tag;
            if (run) {
                const double nalpha = -alpha;
                const bool fr = fi && fi_vec == FI_RV;
                double part[RU][2];
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int cnt = count(u);
                    const long long m = node0(u);
                    double2 zz = make_double2(0.0, 0.0);
                    part[u][0] = part[u][1] = 0.0;
                    auto one = [&](double q, double d, long long n, double& r, double& z) {
                        r = dfma(nalpha, q, r);
                        if (fr && n == fi_idx) r = flipbit(r, fi_bit);
                        z = __ddiv_rn(r, d);
                        part[u][0] = dfma(r, r, part[u][0]);
                        part[u][1] = dfma(r, z, part[u][1]);
                    };
                    if (cnt > 0) one(qq[u].x, dd[u].x, m, rr[u].x, zz.x);
                    if (cnt > 1) one(qq[u].y, dd[u].y, m + 1, rr[u].y, zz.y);
                    st2(a.z, u, zz);
                    if (!KEEP) st2(a.r, u, rr[u]);
                }
                put_runs(part, par);
                // while the sums travel: x += alpha p
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int cnt = count(u);
                    const double2 pv = ld2(p, u);
                    if (!KEEP) xx[u] = ld2(a.x, u);
                    if (cnt > 0) xx[u].x = dfma(alpha, pv.x, xx[u].x);
                    if (cnt > 1) xx[u].y = dfma(alpha, pv.y, xx[u].y);
                    if (!KEEP) st2(a.x, u, xx[u]);
                }
            }
        }
        if (d1_cta) checksum(par, norm_wA);
        double v[2];
        want_r += nruns;
        if (gate) xgate(a.count + 32, want_r);
        if (!xwait<2, 3>(v, a.xr + (long long)par * 3 * nruns, nruns, tag, &s_bad)) { stuck(); return; }
#pragma unroll
        for (int pl = 0; pl < ZP; ++pl) ld_z(a.z, pl, zv[pl]);
        xtree<2>(v, sh[1]);
        const double rel = __ddiv_rn(__dsqrt_rn(v[0]), bnorm);
        const bool conv = rel < tol;
        beta = 0.0;
        if (!conv) { beta = __ddiv_rn(v[1], rho); rho = v[1]; }
        if (c == 0 && tid == 0 && st->log_rel && iter < st->log_cap) {
            st->log_rel[iter] = rel; st->log_alpha[iter] = alpha; st->log_beta[iter] = beta;
        }
        if (conv) { result = iter + 1; done = true; }
        else {
            ++iter;
            if (iter >= max_iter) { result = max_iter; done = true; }
        }
    }
    if (KEEP) st2(a.x, 0, xx[0]);
    if (c == 0 && tid == 0) {
        st->rho = rho; st->alpha = alpha; st->beta = beta; st->bnorm = bnorm; st->pAp = pAp;
        st->iter = iter; st->done = 1; st->broken = broken; st->result = result;
        st->x_pend = 0;
    }
}

}  // namespace hs
