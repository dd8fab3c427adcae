// hs_field.cu -- lognormal conductivity fields generated on the device
// (included by hs_solver.cu; used by hs_field_lognormal and by the batched
// solver's hs_batch_add_lognormal).
//
// The reference's generator (scripts/gen_field.py:29-61) draws white noise on
// the n^3 element grid, filters it in Fourier space by the square root of the
// spectrum of the periodic covariance exp(-r^2/L^2), standardises the result
// to mean 0 and variance 1 and sets k = exp(mu + sigma g).  The square-root
// spectrum exp(-|k|^2 L^2 / 8) is, in real space, the Gaussian kernel
// exp(-2 r^2 / L^2) (standard deviation L/2), so the same filtering is a
// periodic convolution that separates into three 1-D passes (z, y, x); the
// kernel is cut at 6 standard deviations (weights below 1.6e-8 of the
// centre) and wraps around the period like the FFT's.  The white noise comes
// from a counter-based generator: SplitMix64 (G. L. Steele, D. Lea and C. H.
// Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014) of
// the seed and the element index, turned into a normal by the Box-Muller
// transform.  This is not NumPy's stream, so a field is not the reference
// generator's field bit for bit (the host restatement in fields.py is); it
// is a field of the same law, a fixed function of (N, seed, L, mu, sigma):
// the standardisation uses the library's fixed-order reductions.
#include <cuda_runtime.h>

namespace hs {

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
// uniform in (0, 1]: the top 53 bits of a 64-bit word
__device__ __forceinline__ double u01(unsigned long long w) { return ((double)(w >> 11) + 1.0) * 0x1.0p-53; }

// g[e] ~ N(0, 1), independent over e, a fixed function of (seed, e)
__global__ void k_field_noise(long long ne, unsigned long long seed, double* g) {
    const unsigned long long key = splitmix64(seed);
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
        const unsigned long long c = key + 2ull * (unsigned long long)e;
        const double u1 = u01(splitmix64(c)), u2 = u01(splitmix64(c + 1ull));
        g[e] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    }
}

// The weights of a pass: w(t) = exp(-t^2 / (2 s^2)), t = -R..R (s in cells)
constexpr int kFieldMaxTaps = 4096;
__device__ __forceinline__ void field_weights(int R, double s, double* w) {
    for (int t = threadIdx.x; t < 2 * R + 1; t += blockDim.x) {
        const double d = (double)(t - R);
        w[t] = exp(-d * d / (2.0 * s * s));
    }
}

// one periodic 1-D Gaussian pass along axis (0: x, 1: y, 2: z) of an n^3
// grid: out[i] = sum_t w(t) in[i + t e_axis mod n], t = -R..R in order.
// A block takes FL lines and up to FO outputs of each: the inputs with their
// halo (wrapped) go to shared memory once, a lane works on one line and
// carries FU consecutive outputs with a sliding window, so a tap costs one
// shared load, one broadcast of its weight and FU multiply-adds.  Bound: the
// shared-memory pipe and FP64 issue about equally (N=128, 49 taps: 103 M
// multiply-adds a pass, 6 us of the FP64 pipe; 20 us measured, 38 us with the
// window loaded one row at a time).  With one thread per output, a global load
// and a wrap test per tap, the generator took 310 us of device time at N=128
// and 1300 at N=160 with 97 taps; now 130 and 290.
constexpr int FL = 32, FU = 8, FO = 8 * FU;      // one chunk of FU outputs per warp, 8 warps
constexpr int kFieldPitch = FL + 1;      // z pass: lanes load along the line, so an odd pitch
// outputs of a block along a line: the line in equal parts of at most FO, whole chunks
__host__ __device__ inline int field_outs(int n) {
    const int parts = (n + FO - 1) / FO;
    return ((n + parts - 1) / parts + FU - 1) / FU * FU;
}
inline size_t field_conv_smem(int n, int R) {
    return ((size_t)(field_outs(n) + 2 * R) * kFieldPitch + 2 * R + 1) * sizeof(double);
}
__global__ void __launch_bounds__(256) k_field_conv(int n, int axis, int R, double s, const double* in, double* out) {
    extern __shared__ __align__(16) double sm[];
    const int outs = field_outs(n);
    const int span = outs + 2 * R, taps = 2 * R + 1;
    double* S = sm;                                           // [span][kFieldPitch]
    double* w = sm + (size_t)span * kFieldPitch;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nn = (long long)n * n;
    const long long line0 = (long long)blockIdx.x * FL;
    const int o0 = blockIdx.y * outs;                         // first output
    const long long stride = axis == 0 ? nn : axis == 1 ? (long long)n : 1;
    // first element of line l (lines in the order of the other two axes)
    auto base = [&](long long l) { return axis == 0 ? l : axis == 1 ? (l / n) * nn + l % n : l * n; };
    field_weights(R, s, w);
    // rows of the window: z takes a warp per line with the lanes along it, the
    // other axes a warp per row with the lanes across the lines; BL loads in flight
    constexpr int BL = 7;
    const int step = axis == 2 ? 32 : 8, inc = step % n;
    for (int q = axis == 2 ? warp : lane; q < FL; q += axis == 2 ? 8 : FL) {
        const long long ln = line0 + q;
        const double* src = in + base(ln < nn ? ln : 0);
        int i = axis == 2 ? lane : warp;
        int c = (((o0 - R + i) % n) + n) % n;
        while (i < span) {
            double v[BL];
#pragma unroll
            for (int b = 0; b < BL; ++b) {
                v[b] = (i + b * step < span) ? __ldg(src + (long long)c * stride) : 0.0;
                c += inc;
                if (c >= n) c -= n;
            }
#pragma unroll
            for (int b = 0; b < BL; ++b, i += step)
                if (i < span) S[i * kFieldPitch + q] = v[b];
        }
    }
    __syncthreads();
    const int u0 = warp * FU;
    const long long l = line0 + lane;
    double acc[FU], win[FU];
    if (u0 < outs) {
        const double* L = S + (size_t)u0 * kFieldPitch + lane;
#pragma unroll
        for (int u = 0; u < FU; ++u) { acc[u] = 0.0; win[u] = L[u * kFieldPitch]; }
        // taps (odd) = whole groups of FU and a rest; the last tap needs no new input
        int t0 = 0;
        for (; t0 + FU < taps; t0 += FU) {
#pragma unroll
            for (int tt = 0; tt < FU; ++tt) {
                const double wt = w[t0 + tt], nx = L[(t0 + tt + FU) * kFieldPitch];
#pragma unroll
                for (int u = 0; u < FU; ++u) acc[u] = __fma_rn(wt, win[(u + tt) % FU], acc[u]);
                win[tt] = nx;
            }
        }
#pragma unroll
        for (int tt = 0; tt < FU; ++tt) {
            if (t0 + tt < taps) {
                const double wt = w[t0 + tt];
#pragma unroll
                for (int u = 0; u < FU; ++u) acc[u] = __fma_rn(wt, win[(u + tt) % FU], acc[u]);
                if (t0 + tt + 1 < taps) win[tt] = L[(t0 + tt + FU) * kFieldPitch];
            }
        }
        if (axis != 2 && l < nn) {
#pragma unroll
            for (int u = 0; u < FU; ++u)
                if (o0 + u0 + u < n) out[base(l) + (long long)(o0 + u0 + u) * stride] = acc[u];
        }
    }
    if (axis != 2) return;
    // z: turned in shared memory, so that the stores run along the lines
    __syncthreads();
    if (u0 < outs) {
#pragma unroll
        for (int u = 0; u < FU; ++u) S[(u0 + u) * kFieldPitch + lane] = acc[u];
    }
    __syncthreads();
    for (int q = warp; q < FL; q += 8) {
        if (line0 + q >= nn) break;
        for (int i = lane; i < outs && o0 + i < n; i += 32) out[base(line0 + q) + o0 + i] = S[i * kFieldPitch + q];
    }
}

// The same pass for kernels too wide for the window to fit in shared memory.
__global__ void k_field_conv_wide(int n, int axis, int R, double s, const double* in, double* out) {
    __shared__ double w[kFieldMaxTaps];
    const int taps = 2 * R + 1;
    field_weights(R, s, w);
    __syncthreads();
    const long long nn = (long long)n * n, ne = nn * n;
    const long long stride = axis == 0 ? nn : axis == 1 ? (long long)n : 1;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(axis == 0 ? e / nn : axis == 1 ? (e / n) % n : e % n);
        const long long base = e - (long long)c * stride;
        int j = ((c - R) % n + n) % n;
        double acc = 0.0;
        for (int t = 0; t < taps; ++t) {
            acc = __fma_rn(w[t], __ldg(in + base + (long long)j * stride), acc);
            j = (j + 1 == n) ? 0 : j + 1;
        }
        out[e] = acc;
    }
}

// block partials of sum(g) (pass 0) or sum((g - mean)^2) (pass 1, mean from stats[0])
__global__ void __launch_bounds__(RT) k_field_moment(long long ne, int pass, const double* g, const double* stats,
                                                     double* partials, long long nblk) {
    __shared__ double sh[MAXQ][8];
    const double mean = pass ? stats[0] : 0.0;
    double v[1] = {0.0};
    const long long e0 = ((long long)blockIdx.x * RT + threadIdx.x) * KF;
#pragma unroll
    for (int k = 0; k < KF; ++k) {
        const long long e = e0 + k;
        if (e >= ne) break;
        const double x = g[e];
        if (pass) { const double d = dsub(x, mean); v[0] = dfma(d, d, v[0]); }
        else v[0] = dadd(v[0], x);
    }
    store_partials<1>(v, partials, nblk, sh);
}
// stats[0] = mean (pass 0) or stats[1] = standard deviation (pass 1)
__global__ void __launch_bounds__(RT) k_field_moment_final(long long ne, int pass, const double* partials,
                                                           long long nblk, double* stats) {
    __shared__ double sh[MAXQ][8];
    double v[1];
    final_sums<1>(v, partials, nblk, sh);
    if (threadIdx.x != 0) return;
    if (pass == 0) stats[0] = __ddiv_rn(v[0], (double)ne);
    else stats[1] = __dsqrt_rn(__ddiv_rn(v[0], (double)ne));
}
// k = exp(mu + sigma (g - mean) / std), rho*c = rhoc (g is read from rh) for
// elements e0 .. e1-1.  stats may be elements of k: outside the launch's range,
// or in that of a launch of one block.
__global__ void k_field_finish(long long e0, long long e1, double mu, double sigma, double rhoc, const double* stats,
                               double* k, double* rh) {
    const double mean = stats[0], sd = stats[1];
    __syncthreads();
    for (long long e = e0 + (long long)blockIdx.x * blockDim.x + threadIdx.x; e < e1; e += (long long)gridDim.x * blockDim.x) {
        const double g = __ddiv_rn(dsub(rh[e], mean), sd);
        k[e] = exp(dfma(sigma, g, mu));
        rh[e] = rhoc;
    }
}

struct FieldSpecDev {
    int N;
    double mu, sigma, L, rhoc;
    unsigned long long seed;
};

// Taps of the 1-D pass for correlation length L (domain units) on an n-cell period
inline void field_taps(int n, double L, int* R, double* s) {
    *s = 0.5 * L * n;                       // L/2 in cells
    int r = (int)std::ceil(6.0 * *s);
    if (r < 1) r = 1;
    const int rmax = (kFieldMaxTaps - 1) / 2;
    *R = r > rmax ? rmax : r;
}

// Enqueue a lognormal field on stream st into k and rh (N^3 doubles each; rh
// is also the working buffer).  partials: ceil(N^3 / (RT*KF)) doubles;
// stats: 2 doubles; both null: k itself holds them until its values are written
// (N >= 2), so that no scratch memory is needed (allocating and freeing it took
// 600 us of a call).
inline cudaError_t enqueue_field_lognormal(const FieldSpecDev& f, double* k, double* rh, double* partials,
                                           double* stats, cudaStream_t st) {
    const int n = f.N;
    const long long ne = (long long)n * n * n;
    const long long nblk = (ne + (long long)RT * KF - 1) / ((long long)RT * KF);
    int R = 1;
    double s = 1.0;
    field_taps(n, f.L, &R, &s);
    const long long tail = stats ? 0 : 2;
    if (!stats) { partials = k; stats = k + ne - 2; }       // k is free after the last pass
    const int g = (int)std::min<long long>((ne + RT - 1) / RT, 148 * 32);
    k_field_noise<<<g, RT, 0, st>>>(ne, f.seed, k);
    // the window fits in shared memory up to a reach of 390 cells (a correlation of 130 cells)
    const size_t smem = field_conv_smem(n, R);
    constexpr size_t most = 220 * 1024;
    const bool fits = smem <= most;
    if (fits) {
        const cudaError_t e = cudaFuncSetAttribute(k_field_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
    }
    auto conv = [&](int axis, const double* in, double* out) {
        const dim3 grid((unsigned)(((long long)n * n + FL - 1) / FL), (unsigned)((n + field_outs(n) - 1) / field_outs(n)));
        if (fits) k_field_conv<<<grid, 256, smem, st>>>(n, axis, R, s, in, out);
        else k_field_conv_wide<<<g, RT, 0, st>>>(n, axis, R, s, in, out);
    };
    conv(2, k, rh);    // z
    conv(1, rh, k);    // y
    conv(0, k, rh);    // x
    for (int pass = 0; pass < 2; ++pass) {
        k_field_moment<<<(int)nblk, RT, 0, st>>>(ne, pass, rh, stats, partials, nblk);
        k_field_moment_final<<<1, RT, 0, st>>>(ne, pass, partials, nblk, stats);
    }
    k_field_finish<<<g, RT, 0, st>>>(0, ne - tail, f.mu, f.sigma, f.rhoc, stats, k, rh);
    if (tail) k_field_finish<<<1, 32, 0, st>>>(ne - tail, ne, f.mu, f.sigma, f.rhoc, stats, k, rh);
    return cudaGetLastError();
}

}  // namespace hs

extern "C" hs_status hs_field_lognormal(int N, double mu, double sigma, double L, unsigned long long seed,
                                        double rhoc, double* k_dev, double* rhoc_dev) {
    using namespace hs;
    if (N < 1 || N > 1200 || !(sigma >= 0) || !(L > 0) || !(rhoc > 0) || !k_dev || !rhoc_dev) {
        set_error("hs_field_lognormal: bad arguments");
        return HS_ERR_ARG;
    }
    double* scratch = nullptr;
    cudaError_t e = cudaSuccess;
    if (N == 1) e = cudaMalloc(&scratch, 3 * sizeof(double));      // one element holds no scratch
    FieldSpecDev f{N, mu, sigma, L, rhoc, seed};
    if (e == cudaSuccess)
        e = enqueue_field_lognormal(f, k_dev, rhoc_dev, scratch ? scratch + 2 : nullptr, scratch, 0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    if (scratch) cudaFree(scratch);
    if (e != cudaSuccess) { set_error(std::string("hs_field_lognormal: ") + cudaGetErrorString(e)); return HS_ERR_CUDA; }
    return HS_OK;
}
