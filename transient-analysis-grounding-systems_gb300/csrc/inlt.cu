// Numerical Laplace transform pair in FP64 on the device.
//
// Replaces laplace_trans / inv_laplace_trans (src/auxiliary.c:239-329) and the
// batched inverse of the examples (examples/three_grids.c:447-465), which use
// FFTW r2c/c2r:
//   forward  G[k] = sum_j f[j] dt e^{-c t_j} e^{-2 pi i jk/nt},   k < nt/2+1
//   inverse  f[j] = (sum_k sigma_k G[k] e^{+2 pi i jk/nt} over the Hermitian
//            extension) * e^{c t_j} / (nt dt),   c = Re s_0,
// with the reference's data windows sigma (src/auxiliary.c:279-317). The
// twiddles come from one table of nt-th roots indexed exactly by (j k mod nt).
//
// A few series are transformed by direct sums spread over all SMs. Many series
// take a mixed-radix transform (k_inlt_fft): one CTA per two series, whose
// real results are the real and imaginary part of one complex transform of any
// length that fits shared memory; the sums are radix by radix, so they are
// shorter than the direct ones (nt = 4094: 2 + 23 + 89 terms instead of 2047)
// and no less accurate.
#include "tags_common.cuh"
#include "tags_internal.h"
#include "../../include/tags_gpu.h"
#include "plan.h"

namespace {

// The nt-th root number q of unity: angle 2 pi q / nt in [0, 2 pi); sincospi keeps it
// exact at the quadrants.
TAGS_D double2 root_of_unity(long long q, long long nt) {
    double s, c;
    sincospi(2.0 * (double)q / (double)nt, &s, &c);
    return make_double2(c, s);
}

__device__ double window(int filter, double w, double omega) {
    double alpha;
    switch (filter) {
    case 1: alpha = TAGS_PI * w / omega; return 0.42 + 0.5 * cos(alpha) + 0.08 * cos(2 * alpha);
    case 2: return (1 + cos(TAGS_PI * w / omega)) / 2;
    case 3: alpha = TAGS_PI * w / omega; return sin(alpha) / alpha;
    case 4: return 1.0 - (w / omega) * (w / omega);
    default: return 1.0;
    }
}

// The roots of unity, sigma_k of the samples and the output scale e^{c t_j} / (nt dt),
// once per call.
__global__ void k_inlt_tables(const double2* __restrict__ s, long long ns, long long nt, double tmax, int filter,
                              double2* __restrict__ tw, double* __restrict__ sigma, double* __restrict__ scale) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < ns) sigma[q] = window(filter, s[q].y, s[ns - 1].y);
    if (q < nt) {
        tw[q] = root_of_unity(q, nt);
        const double dt = tmax / (double)(nt - 1);
        scale[q] = exp(s[0].x * (double)q * dt) / ((double)nt * dt);
    }
}

// The direct sum of one output: run `part` of `parts` of the terms k = 1 .. kmax
// (runs, not every parts-th term: at late times, where the whole sum is small,
// a run's is too, and so is its rounding). g: the series' samples at stride gk.
TAGS_D double inlt_sum(const double2* __restrict__ g, long long gk, const double* __restrict__ sigma,
                       const double2* __restrict__ tw, long long nt, long long j, int part, int parts) {
    const long long kmax = (nt - 1) / 2, len = (kmax + parts - 1) / parts, k0 = 1 + part * len;
    const long long k1 = k0 + len - 1 < kmax ? k0 + len - 1 : kmax;
    long long q = (j * k0) % nt;
    double acc = 0.0;
    for (long long k = k0; k <= k1; ++k) {
        const double2 t = tw[q], v = g[k * gk];
        acc += sigma[k] * (v.x * t.x - v.y * t.y);
        q += j;
        if (q >= nt) q -= nt;
    }
    return 2.0 * acc;
}

// The terms outside that sum: k = 0 and, for even nt, the Nyquist term.
TAGS_D double inlt_ends(const double2* __restrict__ g, long long gk, const double* __restrict__ sigma, long long nt,
                        long long j) {
    double a = g[0].x * sigma[0];
    if (nt % 2 == 0 && nt > 1) a += ((j & 1) ? -1.0 : 1.0) * g[nt / 2 * gk].x * sigma[nt / 2];
    return a;
}

// Direct inverse, 32 outputs of one series per CTA, eight threads per output
// over eight runs of the terms (added in order): one series of nt = 4094 fills 128
// CTAs. FP64-bound (three operations per term).
constexpr int DIR_PARTS = 8;
__global__ void __launch_bounds__(32 * DIR_PARTS) k_inlt_direct(const double2* __restrict__ g, long long gseries,
                                                                long long gk, const double* __restrict__ sigma,
                                                                const double* __restrict__ scale,
                                                                const double2* __restrict__ tw, long long nt,
                                                                double* __restrict__ f, long long fseries,
                                                                long long fj) {
    __shared__ double part[DIR_PARTS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long j = (long long)blockIdx.x * 32 + lane, srs = blockIdx.y;
    const double2* G = g + gseries * srs;
    part[w][lane] = j < nt ? inlt_sum(G, gk, sigma, tw, nt, j, w, DIR_PARTS) : 0.0;
    __syncthreads();
    if (w != 0 || j >= nt) return;
    double acc = inlt_ends(G, gk, sigma, nt, j);
    for (int q = 0; q < DIR_PARTS; ++q) acc += part[q][lane];
    f[fseries * srs + fj * j] = acc * scale[j];
}

// ---- mixed-radix inverse -----------------------------------------------------------

constexpr int FFT_THREADS = 512;
constexpr int FFT_NT_MAX = 7000;          // two buffers of nt complex values in shared memory
constexpr int FFT_STAGES = 13;            // 2^13 > FFT_NT_MAX
constexpr int FFT_LOW = 64;               // samples k = 1 .. FFT_LOW are summed directly

struct FftPlan {
    int stages;
    int radix[FFT_STAGES];
};

// One self-sorting stage of radix r after l = product of the earlier ones:
//   Y[a + l q + l r b] = sum_p X[a + l (b + m p)] W_{l r}^{a p} W_r^{q p},
// m = n / (l r). A thread forms Q of the r outputs of one (a, b): the inputs
// and their twiddles once for Q outputs.
template <int Q>
TAGS_D void fft_stage(const double2* X, double2* Y, const double2* __restrict__ tw, int n, int l, int r) {
    const int m = n / (l * r), groups = (r + Q - 1) / Q, items = m * l * groups;
    for (int t = threadIdx.x; t < items; t += FFT_THREADS) {
        const int gq = t / (m * l), u = t - gq * (m * l);      // neighbours share q, so W_r^{qp} is one broadcast
        const int b = u / l, a = u - b * l, q0 = gq * Q;
        double2 acc[Q], tot[Q];                                 // sums of eight terms, and of those: a long
#pragma unroll                                                  // chain's rounding grows with its length
        for (int i = 0; i < Q; ++i) acc[i] = tot[i] = cz(0.0, 0.0);
        int ap = 0;                                             // a p m mod n
        const int step = n / r;                                 // W_r = W_n^step
        int qp[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) qp[i] = 0;
        for (int p = 0; p < r; ++p) {
            double2 x = X[a + l * (b + m * p)];
            if (l > 1) x = cmul(x, tw[ap]);
            ap += a * m;
            if (ap >= n) ap -= n;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                acc[i] = cfma(x, tw[qp[i] * step], acc[i]);
                qp[i] += q0 + i;
                if (qp[i] >= r) qp[i] -= r;                     // q0 + i may pass r in the last group: those
                if (qp[i] >= r) qp[i] -= r;                     // outputs are dropped, the index stays in range
            }
            if ((p & 7) == 7) {
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    tot[i] = cadd(tot[i], acc[i]);
                    acc[i] = cz(0.0, 0.0);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if (q0 + i < r) Y[a + l * (q0 + i) + l * r * b] = cadd(tot[i], acc[i]);
    }
}

// Two series per CTA, both scaled to the same size (powers of two), so that
// neither's rounding reaches the other. A pair with a value that is not finite
// takes the direct sums instead, series by series. The lowest samples, where a
// transient's spectrum is largest, are left out of the transform and summed
// directly per output: a transform's rounding is the same at all times, and
// e^{c t} makes the late ones, where the undamped signal is smallest, the
// result's largest errors. FP64-bound: nt (5 sum r + 6 FFT_LOW) operations for
// two series; nt = 4094, 1417 series 65.8 -> 7.2 ms against the direct sums (with
// the host's copies 66.7 -> 8.2 ms). Errors against 128-bit sums, rms of 24
// series: 5.5e-12 of the result either way (FFT_LOW = 32: 5.7e-12, 0 and one
// chain of additions per output: 1.3e-11 at 3.5 ms), 4e-16 instead of 2.2e-15 of
// the undamped signal.
__global__ void __launch_bounds__(FFT_THREADS) k_inlt_fft(const double2* __restrict__ g, long long gseries,
                                                          long long gk, const double* __restrict__ sigma,
                                                          const double* __restrict__ scale,
                                                          const double2* __restrict__ tw, int nt, FftPlan plan,
                                                          double* __restrict__ f, long long fseries, long long fj,
                                                          long long nser) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* X = reinterpret_cast<double2*>(smem_raw);
    double2* Y = X + nt;
    __shared__ double red[2][FFT_THREADS / 32];
    __shared__ double2 low[2][FFT_LOW + 2];                  // k = 0 .. nlow, then the Nyquist sample
    const long long sa = 2LL * blockIdx.x, sb = sa + 1;
    const bool two = sb < nser;
    const double2* A = g + gseries * sa;
    const double2* B = g + gseries * sb;
    const int half = nt / 2, nlow = min(FFT_LOW, half / 2);
    // windowed samples to Y (series a) and X (series b), their largest magnitudes
    double ma = 0.0, mb = 0.0;
    bool bad = false;
    for (int k = threadIdx.x; k <= half; k += FFT_THREADS) {
        double2 va = A[k * gk], vb = two ? B[k * gk] : cz(0.0, 0.0);
        if (k == 0 || 2 * k == nt) va.y = vb.y = 0.0;          // a real signal's ends: the reference's c2r drops them
        const double sg = sigma[k];
        va = cscale(va, sg);
        vb = cscale(vb, sg);
        const double a1 = cabs1(va), b1 = cabs1(vb);
        bad = bad || !isfinite(a1) || !isfinite(b1);
        if (k <= nlow || 2 * k == nt) {
            const int q = k <= nlow ? k : nlow + 1;
            low[0][q] = va;
            low[1][q] = vb;
            va = vb = cz(0.0, 0.0);
        } else {
            ma = fmax(ma, a1);
            mb = fmax(mb, b1);
        }
        Y[k] = va;
        X[k] = vb;
    }
    if (__syncthreads_or(bad)) {
        for (int s = 0; s < (two ? 2 : 1); ++s) {
            const double2* G = s == 0 ? A : B;
            for (int j = threadIdx.x; j < nt; j += FFT_THREADS) {
                double acc = inlt_ends(G, gk, sigma, nt, j);
                acc += inlt_sum(G, gk, sigma, tw, nt, j, 0, 1);
                f[fseries * (sa + s) + fj * j] = acc * scale[j];
            }
        }
        return;
    }
    for (int o = 16; o > 0; o >>= 1) {
        ma = fmax(ma, __shfl_xor_sync(0xffffffffu, ma, o));
        mb = fmax(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = ma;
        red[1][threadIdx.x >> 5] = mb;
    }
    __syncthreads();
    for (int w = 0; w < FFT_THREADS / 32; ++w) {
        ma = fmax(ma, red[0][w]);
        mb = fmax(mb, red[1][w]);
    }
    const int ea = ma > 0.0 ? ilogb(ma) : 0, eb = mb > 0.0 ? ilogb(mb) : 0;
    const double da = scalbn(1.0, max(-1000, min(1000, -ea))), db = scalbn(1.0, max(-1000, min(1000, -eb)));
    // Hermitian extension of a + i b: k and nt - k by the same thread, in place
    for (int k = threadIdx.x; k <= half; k += FFT_THREADS) {
        const double2 va = cscale(Y[k], da), vb = cscale(X[k], db);
        const double2 lo = cz(va.x - vb.y, va.y + vb.x), hi = cz(va.x + vb.y, vb.x - va.y);
        Y[k] = lo;
        if (k > 0 && 2 * k != nt) Y[nt - k] = hi;
    }
    __syncthreads();
    int l = 1;
    for (int s = 0; s < plan.stages; ++s) {
        const int r = plan.radix[s];
        if (r > 4) fft_stage<4>(Y, X, tw, nt, l, r);
        else fft_stage<2>(Y, X, tw, nt, l, r);
        __syncthreads();
        double2* t = X;
        X = Y;
        Y = t;
        l *= r;
    }
    const double ua = scalbn(1.0, max(-1000, min(1000, ea))), ub = scalbn(1.0, max(-1000, min(1000, eb)));
    for (int j = threadIdx.x; j < nt; j += FFT_THREADS) {
        double a = 0.5 * low[0][0].x, b = 0.5 * low[1][0].x;    // largest first: at late times they cancel at once
        int q = 0;
        for (int k = 1; k <= nlow; ++k) {
            q += j;
            if (q >= nt) q -= nt;
            const double2 t = tw[q], va = low[0][k], vb = low[1][k];
            a += va.x * t.x - va.y * t.y;
            b += vb.x * t.x - vb.y * t.y;
        }
        a = 2.0 * a + Y[j].x * ua;
        b = 2.0 * b + Y[j].y * ub;
        if (nt % 2 == 0) {
            a += ((j & 1) ? -1.0 : 1.0) * low[0][nlow + 1].x;
            b += ((j & 1) ? -1.0 : 1.0) * low[1][nlow + 1].x;
        }
        const double sc = scale[j];
        f[fseries * sa + fj * j] = a * sc;
        if (two) f[fseries * sb + fj * j] = b * sc;
    }
}

FftPlan fft_plan(int nt, int* sum) {
    FftPlan p{};
    int n = nt;
    *sum = 0;
    auto take = [&](int r) {
        while (n % r == 0 && p.stages < FFT_STAGES) {
            p.radix[p.stages++] = r;
            *sum += r;
            n /= r;
        }
    };
    for (int r : {8, 4, 2, 9, 3}) take(r);
    for (int r = 5; n > 1; r += 2) {
        if (r * r > n) r = n;
        take(r);
    }
    return p;
}

// ---- forward -------------------------------------------------------------------

// The roots of unity and the damped samples f[j] dt e^{-c t_j}, once per call.
__global__ void k_nlt_damp(const double* __restrict__ f, long long nt, double tmax, double2* __restrict__ tw,
                           double* __restrict__ v) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nt) return;
    tw[j] = root_of_unity(j, nt);
    const double c = log((double)nt * (double)nt) / tmax, dt = tmax / (double)(nt - 1);
    v[j] = f[j] * dt * exp(-c * (double)j * dt);
}

// Forward transform of one damped series, 32 outputs per CTA, eight threads
// per output as in the direct inverse.
__global__ void __launch_bounds__(32 * DIR_PARTS) k_nlt(const double* __restrict__ v, long long nt,
                                                        const double2* __restrict__ tw, double2* __restrict__ g) {
    __shared__ double2 part[DIR_PARTS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long k = (long long)blockIdx.x * 32 + lane, ns = nt / 2 + 1;
    double re = 0.0, im = 0.0;
    if (k < ns) {
        long long q = (k * w) % nt;
        const long long dq = (k * DIR_PARTS) % nt;
        for (long long j = w; j < nt; j += DIR_PARTS) {
            const double2 t = tw[q];
            re += v[j] * t.x;
            im -= v[j] * t.y;
            q += dq;
            if (q >= nt) q -= nt;
        }
    }
    part[w][lane] = make_double2(re, im);
    __syncthreads();
    if (w != 0 || k >= ns) return;
    for (int q = 1; q < DIR_PARTS; ++q) {
        re += part[q][lane].x;
        im += part[q][lane].y;
    }
    g[k] = make_double2(re, im);
}

}  // namespace

size_t tags_inlt_workspace(long long nt) { return (sizeof(double2) + 2 * sizeof(double)) * (size_t)nt + 64; }

int tags_launch_inlt(const double2* d_g, long long gseries, long long gk, const double2* d_s, void* ws, long long nt,
                     double tmax, int filter, double* d_f, long long fseries, long long fj, long long nser,
                     cudaStream_t st) {
    const long long ns = nt / 2 + 1;
    double2* tw = reinterpret_cast<double2*>(ws);
    double* scale = reinterpret_cast<double*>(tw + nt);
    double* sigma = scale + nt;                                // ns <= nt values
    k_inlt_tables<<<(unsigned)((nt + 127) / 128), 128, 0, st>>>(d_s, ns, nt, tmax, filter, tw, sigma, scale);
    tags_note_launch();
    // SM cycles of either way (two FP64 multiply-adds per clock and SM): the
    // transform keeps a CTA's SM for nt (5 sum r + 6 FFT_LOW) / 2 and runs a pair per SM at a
    // time, the direct sums take three operations a term on all SMs. nt = 4094:
    // one series 60 us direct, the transform ~1.4 ms for up to 304.
    int sum = 0;
    const FftPlan plan = nt <= FFT_NT_MAX ? fft_plan((int)nt, &sum) : FftPlan{};
    const double pairs = 0.5 * (double)(nser + 1);
    const double sms = tags_num_sms();
    const double c_fft = ceil(pairs / sms) * (double)nt * (5.0 * sum + 6.0 * FFT_LOW) / 2.0;
    const double c_direct = (double)nser * (double)nt * (double)ns * 3.0 / (2.0 * sms);
    if (nt <= FFT_NT_MAX && nt > 2 && c_fft < c_direct) {
        static PerDevice state;
        const int err = tags_once_per_device(state, [] {
            if (cudaFuncSetAttribute(k_inlt_fft, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(2 * FFT_NT_MAX * sizeof(double2))) != cudaSuccess)
                return tags_fail(TAGS_E_CUDA, "cudaFuncSetAttribute(k_inlt_fft) failed");
            return 0;
        });
        if (err) return err;
        k_inlt_fft<<<(unsigned)((nser + 1) / 2), FFT_THREADS, 2 * sizeof(double2) * nt, st>>>(
            d_g, gseries, gk, sigma, scale, tw, (int)nt, plan, d_f, fseries, fj, nser);
        tags_note_launch();
    } else {
        for (long long s0 = 0; s0 < nser; s0 += 65535) {
            const long long n = nser - s0 < 65535 ? nser - s0 : 65535;
            k_inlt_direct<<<dim3((unsigned)((nt + 31) / 32), (unsigned)n), 32 * DIR_PARTS, 0, st>>>(
                d_g + gseries * s0, gseries, gk, sigma, scale, tw, nt, d_f + fseries * s0, fseries, fj);
            tags_note_launch();
        }
    }
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

int tags_launch_nlt(const double* d_f, long long nt, void* ws, double tmax, double2* d_g, cudaStream_t st) {
    double2* tw = reinterpret_cast<double2*>(ws);
    double* v = reinterpret_cast<double*>(tw + nt);
    k_nlt_damp<<<(unsigned)((nt + 127) / 128), 128, 0, st>>>(d_f, nt, tmax, tw, v);
    k_nlt<<<(unsigned)((nt / 2 + 1 + 31) / 32), 32 * DIR_PARTS, 0, st>>>(v, nt, tw, d_g);
    tags_note_launch(2);
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}
