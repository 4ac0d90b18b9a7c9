// FP64 solve of the immittance system in its structure (plain form).
//
// Same system as the reference's solve_immittance (src/linalg.c:112-139), in
// the static order [I_L, I_T, U]:
//     W = [ -ZL   0    A ]
//         [  0   -ZT   B ]      b = [0; 0; I_E]
//         [ A^T  B^T   0 ]
// The elimination meets the impedance blocks first and the node block last,
// so it needs no pivot search, and the coupling of ZL and ZT stays zero: an
// LDL^T takes 2 (4/3 m^3 + 4 m^2 n + 4 m n^2) + 4/3 n^3 real flops where the
// LU of the full matrix takes 8/3 N^3 (66.6 against 249 GFLOP at m = 1560,
// n = 1417). FP64 runs at two fused multiply-adds per clock and SM here, so
// the flops are the time. What the missing pivot search may cost in accuracy
// is recovered by FP64 refinement against the untouched impedance blocks; a
// sample whose corrections do not shrink until the next one would be below FP64
// rounding is handed to the pivoted LU (lu.cu) by its caller.
// Measured against that LU on GB300: 2 samples at m = 1560 714 -> 120 ms, 256
// samples at m = 100 24.3 -> 5.9 ms, 100 samples at m = 10 0.66 -> 0.25 ms.
//
// Layout: column-major N x N per sample, leading dimension ld. Lower triangle:
// the matrix, then L; the strict upper triangle keeps U = D L^T of the panels
// (the update's right operand) and, in the ZL/ZT coupling blocks that the
// elimination never touches, the full symmetric ZL (rows 0..m, columns m..2m)
// and ZT (rows m..2m, columns 0..m) that the residual reads. Panels are 32
// columns wide and never straddle m or 2m, so a ZL panel skips the ZT rows
// exactly. The inverses of the panels' factored diagonal blocks live in the
// workspace, so that a solve's diagonal step is a product (every CTA of a panel
// launch factors the block itself, which saves a launch per panel).
#include <algorithm>

#include "tags_common.cuh"
#include "tags_internal.h"
#include "../../include/tags_gpu.h"
#include "plan.h"

namespace {

constexpr int PB = 32;                    // panel width

// Columns [j0, j0 + jb) of panel p; the rows below it are base + v, v < cnt,
// plus `skip` from `lim` on (a ZL panel has no ZT rows).
struct Panel {
    int j0, jb, base, lim, skip, cnt;
    TAGS_HD int row(int v) const {
        const int r = base + v;
        return r >= lim ? r + skip : r;
    }
};

TAGS_HD int panel_count(int N, int m) {
    return m == 0 ? (N + PB - 1) / PB : 2 * ((m + PB - 1) / PB) + (N - 2 * m + PB - 1) / PB;
}

TAGS_HD Panel panel_at(int p, int N, int m) {
    Panel q;
    const int pm = (m + PB - 1) / PB;
    int end;
    if (m == 0) {
        q.j0 = PB * p;
        end = N;
    } else if (p < pm) {
        q.j0 = PB * p;
        end = m;
    } else if (p < 2 * pm) {
        q.j0 = m + PB * (p - pm);
        end = 2 * m;
    } else {
        q.j0 = 2 * m + PB * (p - 2 * pm);
        end = N;
    }
    q.jb = end - q.j0 < PB ? end - q.j0 : PB;
    q.base = q.j0 + q.jb;
    const bool zl = m > 0 && q.j0 < m;
    q.lim = zl ? m : N;
    q.skip = zl ? m : 0;
    q.cnt = N - q.base - q.skip;
    return q;
}

// All CTAs of the cluster; their shared memory's writes before it are seen after.
TAGS_D void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// *p of the cluster's CTA `rank`, p in shared memory.
TAGS_D double2 ld_cluster(const double2* p, int rank) {
    uint32_t a;
    double2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"((uint32_t)rank));
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}

TAGS_D double2 crecip(double2 d) {
    const double s = 1.0 / (d.x * d.x + d.y * d.y);      // out of range: not finite, the sample goes to the LU
    return make_double2(d.x * s, -d.y * s);
}

// Diagonal block and rows of one panel: L21 = A21 L11^-T D^-1 (stored in
// place) and U12 = D L21^T (stored in the upper triangle). Every CTA factors
// the 32 x 32 block first; the 32 rows after the last one are the identity's,
// whose result L11^-T goes to the workspace for the solves, with 1/D on the
// diagonal. A warp's FP64 instruction holds its quarter of the SM for 64
// cycles, so time is the FP64 instructions of the busiest warp. The block: its
// 496 elements right of column 0 are dealt to the threads column by column, four
// each in registers, so that a step's live ones fill whole warps (252
// instructions for the products instead of 544 with a lane per row and a warp
// per column); every warp forms the scaled column itself (15 a step); one
// barrier per step. The rows: LPR lanes share a row, 32 / LPR columns each: 576
// instructions with 4 lanes, 320 with 8, 192 with 16, which take more CTAs for
// the same rows (panel_split). The 11 panels and block inverses of one system at m
// = 100, n = 85 644 -> 400 us, the panels of the plain form's 256 samples 2.3 ->
// 1.9 ms.
template <int LPR>
__global__ void __launch_bounds__(128) k_ldl64_panel(double2* __restrict__ A0, long long ld, long long stride,
                                                     Panel q, int p, double2* __restrict__ ws0, long long wstride,
                                                     int passes) {
    constexpr int ROWS = 128 / LPR, NC = PB / LPR;
    double2* A = A0 + stride * blockIdx.y;
    double2* ws = ws0 + wstride * blockIdx.y + (long long)p * PB * PB;
    __shared__ double2 sL[PB][PB + 1];
    __shared__ double2 sdi[PB];
    const int tid = threadIdx.x, lane = tid & 31;
    for (int t = tid; t < PB * PB; t += 128) {
        const int r = t % PB, c = t / PB;
        double2 v = cz(r == c ? 1.0 : 0.0, 0.0);          // a short panel is padded with the identity
        if (r < q.jb && c <= r) v = A[(q.j0 + r) + ld * (q.j0 + c)];
        sL[r][c] = v;
    }
    __syncthreads();
    int er[4], ec[4];
    double2 ev[4];
    for (int i = 0, c = 1, first = 0; i < 4; ++i) {        // element tid + 128 i: column c starts at `first`
        const int e = tid + 128 * i;
        while (c < PB && e - first >= PB - c) first += PB - c++;
        ec[i] = c < PB ? c : 0;                             // 0: none
        er[i] = c < PB ? c + e - first : 0;
        ev[i] = sL[er[i]][ec[i]];
    }
    for (int k = 0; k < q.jb; ++k) {
        // -W / d as (-W conj(d)) / |d|^2: the product is formed while the reciprocal is
        const double2 d = sL[k][k], w = cmul(sL[lane][k], cz(-d.x, d.y));
        const double2 l = cscale(w, 1.0 / (d.x * d.x + d.y * d.y));     // rows up to k are not used
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!__any_sync(0xffffffffu, ec[i] > k)) continue;
            const double2 lr = cz(__shfl_sync(0xffffffffu, l.x, er[i]), __shfl_sync(0xffffffffu, l.y, er[i]));
            if (ec[i] > k) {
                ev[i] = cfma(lr, sL[ec[i]][k], ev[i]);
                if (ec[i] == k + 1) sL[er[i]][ec[i]] = ev[i];     // the next step's column
            }
        }
        __syncthreads();
    }
    if (tid < PB) sdi[tid] = crecip(sL[tid][tid]);         // 1 past jb
    __syncthreads();
    for (int t = tid; t < PB * PB; t += 128) {            // unscaled columns -> L11
        const int r = t % PB, c = t / PB;
        if (r > c && r < q.jb) sL[r][c] = cmul(sL[r][c], sdi[c]);
        if (blockIdx.x == 0 && r <= c) ws[c * PB + r] = r == c ? sdi[c] : cz(0.0, 0.0);
    }
    __syncthreads();
    const int g = tid % LPR;                                // lane of the row's LPR: columns g, g + LPR, ..
    for (int pass = 0; pass < passes; ++pass) {
        const int v0 = (blockIdx.x * passes + pass) * ROWS;
        if (v0 >= q.cnt + PB) return;                       // the whole CTA
        const int v = v0 + tid / LPR, unit = v - q.cnt;     // unit >= 0: row of the identity
        const bool on = v < q.cnt;
        const int row = on ? q.row(v) : 0;
        double2 w[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int c = LPR * i + g;
            w[i] = on && c < q.jb ? A[row + ld * (q.j0 + c)] : cz(c == unit ? 1.0 : 0.0, 0.0);
        }
#pragma unroll
        for (int k = 0; k < PB - 1; ++k) {
            if (k + 1 < q.jb) {                             // the same in every thread
                const double2 wk = cz(-__shfl_sync(0xffffffffu, w[k / LPR].x, k % LPR, LPR),
                                      -__shfl_sync(0xffffffffu, w[k / LPR].y, k % LPR, LPR));
#pragma unroll
                for (int i = k / LPR; i < NC; ++i) {
                    const int c = LPR * i + g;
                    if (c > k) w[i] = cfma(wk, sL[c][k], w[i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int c = LPR * i + g;
            if (on && c < q.jb) {
                A[row + ld * (q.j0 + c)] = cmul(w[i], sdi[c]);
                A[(q.j0 + c) + ld * row] = w[i];
            } else if (unit >= 0 && unit < c) {
                ws[unit * PB + c] = w[i];
            }
        }
    }
}

// Trailing update C -= L21 U12 over the lower triangle of the rows below the
// panel, TL x TL tiles of TT x TT values per thread. FP64-bound (a warp's FP64
// instruction holds its quarter of the SM for 64 cycles): a tile of 64 takes
// 262,144 SM cycles of multiply-adds against 131 KB of C, so one panel (K = 32)
// per update is enough. The tile size sets the work wasted on the diagonal and
// the edge, and with four or more warps per tile how long a launch of few
// tiles takes at least: 131, 33 and 8 us for 64, 32 and 16.
// The complex products as three real ones: with s = re + im of each operand,
//   re = sum ar br - sum ai bi,  im = sum as bs - sum ar br - sum ai bi,
// a quarter fewer FP64 instructions; the sums s are formed once per tile, in
// shared memory. The imaginary part's rounding is then that of the larger part:
// the refinement's residual takes the products in full.
template <int TL, int TT>
__global__ void __launch_bounds__(TL * TL / (TT * TT)) k_ldl64_update(double2* __restrict__ A0, long long ld,
                                                                   long long stride, Panel q) {
    double2* A = A0 + stride * blockIdx.y;
    constexpr int TH = TL / TT, NT = TH * TH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sA = reinterpret_cast<double*>(smem_raw);      // [3][PB][TL]: re, im, re + im
    double* sB = sA + 3 * PB * TL;                         // [3][PB][TL]
    const int t = blockIdx.x;
    int ty = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while (ty > 0 && ty * (ty + 1) / 2 > t) --ty;
    while ((ty + 1) * (ty + 2) / 2 <= t) ++ty;
    const int r0 = ty * TL, c0 = (t - ty * (ty + 1) / 2) * TL;
    for (int s = threadIdx.x; s < PB * TL; s += NT) {
        const int r = s % TL, k = s / TL;
        const double2 a = (k < q.jb && r0 + r < q.cnt) ? A[q.row(r0 + r) + ld * (q.j0 + k)] : cz(0.0, 0.0);
        sA[s] = a.x;
        sA[PB * TL + s] = a.y;
        sA[2 * PB * TL + s] = a.x + a.y;
        const int kk = s % PB, c = s / PB, o = kk * TL + c;
        const double2 b = (kk < q.jb && c0 + c < q.cnt) ? A[(q.j0 + kk) + ld * q.row(c0 + c)] : cz(0.0, 0.0);
        sB[o] = b.x;
        sB[PB * TL + o] = b.y;
        sB[2 * PB * TL + o] = b.x + b.y;
    }
    __syncthreads();
    const int tx = threadIdx.x % TH, tyy = threadIdx.x / TH;
    double acc[3][TT][TT];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int a = 0; a < TT; ++a)
#pragma unroll
            for (int b = 0; b < TT; ++b) acc[p][a][b] = 0.0;
    for (int k = 0; k < q.jb; ++k) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            double av[TT], bv[TT];
#pragma unroll
            for (int a = 0; a < TT; ++a) av[a] = sA[(p * PB + k) * TL + tx + TH * a];
#pragma unroll
            for (int b = 0; b < TT; ++b) bv[b] = sB[(p * PB + k) * TL + tyy + TH * b];
#pragma unroll
            for (int a = 0; a < TT; ++a)
#pragma unroll
                for (int b = 0; b < TT; ++b) acc[p][a][b] = fma(av[a], bv[b], acc[p][a][b]);
        }
    }
#pragma unroll
    for (int b = 0; b < TT; ++b) {
        const int gc = c0 + tyy + TH * b;
        if (gc >= q.cnt) continue;
        const long long col = ld * q.row(gc);
#pragma unroll
        for (int a = 0; a < TT; ++a) {
            const int gr = r0 + tx + TH * a;
            if (gr < q.cnt && gr >= gc) {
                const long long idx = q.row(gr) + col;
                const double rr = acc[0][a][b], ii = acc[1][a][b];
                A[idx] = csub(A[idx], cz(rr - ii, acc[2][a][b] - rr - ii));
            }
        }
    }
}

// y = L11^-1 x (upper = 0) or L11^-T x (upper = 1) for a panel's 32 values,
// eight terms per thread in the CTA's first four warps; raw, y and part in
// shared memory. Ends with a barrier.
TAGS_D void block_apply(const double2* __restrict__ ws, const double2* raw, double2* y, double2 (*part)[PB], int upper) {
    const int r = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < 4) {
        double2 a = w == 0 ? raw[r] : cz(0.0, 0.0);
        for (int k = 8 * w; k < 8 * w + 8; ++k)
            if (upper ? k > r : k < r) a = cfma(ws[upper ? r * PB + k : k * PB + r], raw[k], a);
        part[w][r] = a;
    }
    __syncthreads();
    if (threadIdx.x < PB) y[r] = cadd(cadd(part[0][r], part[1][r]), cadd(part[2][r], part[3][r]));
    __syncthreads();
}

// One panel of the forward sweep: y = L11^-1 x_p (to Z), then x_r -= L_rp y
// below it. 32 rows per CTA, eight columns per warp; x_p itself is left, so the
// CTAs agree on it.
__global__ void __launch_bounds__(128) k_ldl64_fwd(const double2* __restrict__ A0, long long ld, long long stride,
                                                   Panel q, int p, const double2* __restrict__ ws0, long long wstride,
                                                   double2* __restrict__ X0, double2* __restrict__ Z0, int N,
                                                   const int* __restrict__ active) {
    const int b = blockIdx.y;
    if (!active[b]) return;
    const double2* A = A0 + stride * b;
    double2* X = X0 + (long long)N * b;
    __shared__ double2 raw[PB], y[PB], part[4][PB];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < PB) raw[lane] = lane < q.jb ? X[q.j0 + lane] : cz(0.0, 0.0);
    __syncthreads();
    block_apply(ws0 + wstride * b + (long long)p * PB * PB, raw, y, part, 0);
    if (blockIdx.x == 0 && (int)threadIdx.x < q.jb) Z0[(long long)N * b + q.j0 + threadIdx.x] = y[threadIdx.x];
    const int v = blockIdx.x * 32 + lane;
    const int row = v < q.cnt ? q.row(v) : 0;
    double2 acc = cz(0.0, 0.0);
    if (v < q.cnt)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = 8 * w + i;
            if (c < q.jb) acc = cfma(A[row + ld * (q.j0 + c)], y[c], acc);
        }
    part[w][lane] = acc;
    __syncthreads();
    if (w == 0 && v < q.cnt)
        X[row] = csub(X[row], cadd(cadd(part[0][lane], part[1][lane]), cadd(part[2][lane], part[3][lane])));
}

// One panel of the backward sweep on T (which starts as D^-1 z): y = L11^-T
// T_p (to S), then T_c -= L_pc^T y for the columns c0 .. j0 left of it.
__global__ void __launch_bounds__(128) k_ldl64_bwd(const double2* __restrict__ A0, long long ld, long long stride,
                                                   Panel q, int p, int c0, const double2* __restrict__ ws0,
                                                   long long wstride, double2* __restrict__ T0,
                                                   double2* __restrict__ S0, int N, const int* __restrict__ active) {
    const int b = blockIdx.y;
    if (!active[b]) return;
    const double2* A = A0 + stride * b;
    double2* T = T0 + (long long)N * b;
    __shared__ double2 raw[PB], y[PB], part[4][PB];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < PB) raw[lane] = lane < q.jb ? T[q.j0 + lane] : cz(0.0, 0.0);
    __syncthreads();
    block_apply(ws0 + wstride * b + (long long)p * PB * PB, raw, y, part, 1);
    if (blockIdx.x == 0 && (int)threadIdx.x < q.jb) S0[(long long)N * b + q.j0 + threadIdx.x] = y[threadIdx.x];
    const int c = c0 + blockIdx.x * 32 + lane;
    double2 acc = cz(0.0, 0.0);
    if (c < q.j0)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 8 * w + i;
            if (r < q.jb) acc = cfma(A[(q.j0 + r) + ld * c], y[r], acc);
        }
    part[w][lane] = acc;
    __syncthreads();
    if (w == 0 && c < q.j0)
        T[c] = csub(T[c], cadd(cadd(part[0][lane], part[1][lane]), cadd(part[2][lane], part[3][lane])));
}

// T = D^-1 z (in place).
__global__ void k_ldl64_dscale(double2* __restrict__ Z0, int N, int m, const double2* __restrict__ ws0,
                               long long wstride, const int* __restrict__ active) {
    const int b = blockIdx.y;
    if (!active[b]) return;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const int pm = (m + PB - 1) / PB;
    const int blk = m == 0 || j < m ? 0 : j < 2 * m ? 1 : 2, o = j - blk * m;
    const double2* ws = ws0 + wstride * b + (long long)(blk * pm + o / PB) * PB * PB;
    double2* z = Z0 + (long long)N * b + j;
    *z = cmul(*z, ws[(o % PB) * (PB + 1)]);
}

// Both sweeps of one sample by one CTA, the vector in shared memory: for
// systems whose sweeps are shorter than the panel-by-panel launches (N up to
// ~300: 81,000 SM cycles per sweep at N = 285), or batches that fill the SMs.
constexpr int SOLVE_THREADS = 256;
__global__ void __launch_bounds__(SOLVE_THREADS) k_ldl64_solve_cta(
    const double2* __restrict__ A0, long long ld, long long stride, int N, int m, const double2* __restrict__ ws0,
    long long wstride, const double2* __restrict__ X0, double2* __restrict__ S0, int p0,
    const int* __restrict__ active) {
    const int b = blockIdx.x;
    if (!active[b]) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* xs = reinterpret_cast<double2*>(smem_raw);     // N
    __shared__ double2 raw[PB], y[PB], part[4][PB];
    const double2* A = A0 + stride * b;
    const double2* ws = ws0 + wstride * b;
    const int P = panel_count(N, m);
    for (int j = threadIdx.x; j < N; j += blockDim.x) xs[j] = X0[(long long)N * b + j];
    __syncthreads();
    for (int p = p0; p < P; ++p) {                           // the right-hand side is zero above panel p0
        const Panel q = panel_at(p, N, m);
        if (threadIdx.x < PB) raw[threadIdx.x] = (int)threadIdx.x < q.jb ? xs[q.j0 + threadIdx.x] : cz(0.0, 0.0);
        __syncthreads();
        block_apply(ws + (long long)p * PB * PB, raw, y, part, 0);
        if ((int)threadIdx.x < q.jb) xs[q.j0 + threadIdx.x] = cmul(y[threadIdx.x],
                                                                   ws[(long long)p * PB * PB + threadIdx.x * (PB + 1)]);
        for (int v = threadIdx.x; v < q.cnt; v += blockDim.x) {
            const int row = q.row(v);
            double2 acc = cz(0.0, 0.0);
#pragma unroll 8
            for (int c = 0; c < q.jb; ++c) acc = cfma(A[row + ld * (q.j0 + c)], y[c], acc);
            xs[row] = csub(xs[row], acc);
        }
        __syncthreads();
    }
    for (int p = P - 1; p >= 0; --p) {
        const Panel q = panel_at(p, N, m);
        const int c0 = m > 0 && q.j0 >= m && q.j0 < 2 * m ? m : 0;
        if (threadIdx.x < PB) raw[threadIdx.x] = (int)threadIdx.x < q.jb ? xs[q.j0 + threadIdx.x] : cz(0.0, 0.0);
        __syncthreads();
        block_apply(ws + (long long)p * PB * PB, raw, y, part, 1);
        if ((int)threadIdx.x < q.jb) xs[q.j0 + threadIdx.x] = y[threadIdx.x];
        for (int c = c0 + threadIdx.x; c < q.j0; c += blockDim.x) {
            double2 acc = cz(0.0, 0.0);
#pragma unroll 8
            for (int r = 0; r < q.jb; ++r) acc = cfma(A[(q.j0 + r) + ld * c], y[r], acc);
            xs[c] = csub(xs[c], acc);
        }
        __syncthreads();
    }
    for (int j = threadIdx.x; j < N; j += blockDim.x) S0[(long long)N * b + j] = xs[j];
}

// The same of one sample by a cluster of 8 CTAs, for a few samples of up to 1024
// unknowns, whose sweeps leave the SMs idle in the kernels above: CTA g owns the
// rows whose 32-row chunk is g mod 8. Per panel every CTA gathers the panel's 32
// values from their owners' shared memory, forms the diagonal step itself and
// updates its own rows, eight columns per warp; one cluster barrier. The matrix's
// values do not wait for the vector, so a step's first two chunks are on their
// way before the barrier. The forward sweep works in xs and leaves its values in
// zs, the backward sweep the other way round, so nothing is overwritten that
// another CTA has still to gather. The backward sweep reads U = D L^T, whose rows
// lie side by side, with 1/D at the diagonal step. One sample at N = 285 195 ->
// 118 us; at N = 801 six samples' solves 0.31 -> 0.22 ms each. Where the line lies:
// N <= 64 gains nothing from eight CTAs (280 against 267 us for a whole nodal
// chain of 4 segments); up to N = 320 two waves of clusters still beat a CTA per
// sample, above that one wave beats the launches per panel.
constexpr int SCL_G = 8, SCL_N = 1024, SCL_UNITS = (SCL_N / 32 + SCL_G - 1) / SCL_G + 1;
constexpr size_t scl_smem(int N) { return sizeof(double2) * 2 * (size_t)N; }

__global__ void __cluster_dims__(SCL_G, 1, 1) __launch_bounds__(128) k_ldl64_solve_cl(
    const double2* __restrict__ A0, long long ld, long long stride, int N, int m, const double2* __restrict__ ws0,
    long long wstride, const double2* __restrict__ X0, double2* __restrict__ S0, int p0,
    const int* __restrict__ active) {
    const int b = blockIdx.y, g = blockIdx.x;
    if (!active[b]) return;                                  // the whole cluster
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* xs = reinterpret_cast<double2*>(smem_raw);      // N, own rows
    double2* zs = xs + N;                                    // N, own rows
    __shared__ double2 raw[PB], y[PB], part[4][PB], sum[SCL_UNITS][4][PB];
    const double2* A = A0 + stride * b;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, P = panel_count(N, m);
    auto own = [&](int i) { return ((i >> 5) & (SCL_G - 1)) == g; };
    for (int i = tid; i < N; i += 128)
        if (own(i)) {
            xs[i] = X0[(long long)N * b + i];
            zs[i] = cz(0.0, 0.0);                            // the sweep is zero above panel p0
        }
    for (int s = p0; s < 2 * P; ++s) {
        const int bwd = s >= P, p = bwd ? 2 * P - 1 - s : s;
        const Panel q = panel_at(p, N, m);
        const double2* ws = ws0 + wstride * b + (long long)p * PB * PB;
        double2 *work = bwd ? zs : xs, *fin = bwd ? xs : zs;
        // the rows to update: [lo, hi) without [q.lim, q.lim + q.skip) below a ZL panel
        const int lo = bwd ? (m > 0 && q.j0 >= m && q.j0 < 2 * m ? m : 0) : q.base, hi = bwd ? q.j0 : N;
        const int b0 = bwd ? N : q.lim, b1 = bwd ? N : q.lim + q.skip;
        auto live = [&](int i) { return i >= lo && i < hi && !(i >= b0 && i < b1); };
        const int c0 = (lo >> 5) + ((g - (lo >> 5)) & (SCL_G - 1));     // first own chunk
        const double2* col = A + ld * (q.j0 + 8 * warp);
        double2 pre[2][8];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = 32 * (c0 + SCL_G * u) + lane;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                pre[u][k] = live(i) && 8 * warp + k < q.jb ? col[i + ld * k] : cz(0.0, 0.0);
        }
        cluster_barrier();                                   // the panel's values are updated by all panels before
        if (tid < PB) {
            double2 v = cz(0.0, 0.0);
            if (tid < q.jb) {
                const int i = q.j0 + tid;
                v = ld_cluster(work + i, (i >> 5) & (SCL_G - 1));
                if (bwd) v = cmul(v, ws[tid * (PB + 1)]);
            }
            raw[tid] = v;
        }
        __syncthreads();
        block_apply(ws, raw, y, part, bwd);
        if (tid < q.jb && own(q.j0 + tid)) fin[q.j0 + tid] = y[tid];
        int nu = 0;
        for (int c = c0; 32 * c < hi; c += SCL_G, ++nu) {
            const int i = 32 * c + lane;
            double2 acc = cz(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double2 l = nu == 0 ? pre[0][k] : nu == 1 ? pre[1][k]
                                : live(i) && 8 * warp + k < q.jb ? col[i + ld * k] : cz(0.0, 0.0);
                acc = cfma(l, y[8 * warp + k], acc);
            }
            sum[nu][warp][lane] = acc;
        }
        __syncthreads();
        for (int u = warp; u < nu; u += 4) {
            const int i = 32 * (c0 + SCL_G * u) + lane;
            if (live(i))
                work[i] = csub(work[i], cadd(cadd(sum[u][0][lane], sum[u][1][lane]), cadd(sum[u][2][lane], sum[u][3][lane])));
        }
    }
    cluster_barrier();                                       // no CTA leaves while another gathers from it
    for (int i = tid; i < N; i += 128)
        if (own(i)) S0[(long long)N * b + i] = xs[i];
}

// Reordered index -> index of the original order [U, I_L, I_T] (m = 0: equal).
TAGS_D int orig_index(int ip, int m, int n) { return ip < 2 * m ? n + ip : ip - 2 * m; }

// Start of a solve: b and r = b in the static order, x = 0, every sample active.
__global__ void k_ldl64_start(const double2* __restrict__ rhs, long long rstride, int m, int n,
                              double2* __restrict__ B0, double2* __restrict__ R0, double2* __restrict__ X0,
                              int* __restrict__ active, int* __restrict__ conv) {
    const int N = n + 2 * m, b = blockIdx.y;
    const int ip = blockIdx.x * blockDim.x + threadIdx.x;
    if (ip == 0) {
        active[b] = 1;
        conv[b] = 0;
    }
    if (ip >= N) return;
    const double2 v = rhs[rstride * b + orig_index(ip, m, n)];
    const long long o = (long long)N * b + ip;
    B0[o] = v;
    R0[o] = v;
    X0[o] = cz(0.0, 0.0);
}

// The stopping rule, for the currents (amperes) and the potentials (volts), whose
// sizes have nothing to do with one another, each by itself. A correction dn after
// one of prev makes the next about dn^2 / prev; done when that is below 1e-16 of
// the unknowns, xn. (By dn <= 1e-8 xn alone a contraction of 1e-4 stopped after two
// refinements with 1e-12 left: 1200 random rods, wires and grids from |s| = 1e-4 / s
// on were off by up to 9e-12, now by up to 2e-14, at the same times.)
TAGS_D bool settled(double dn, double prev, double xn) { return dn <= 1e-8 * sqrt(prev) * sqrt(xn); }

// The rule's maxima of |Re| + |Im| as the values' upper words, which order as the
// values do (to 2^-20) and need no FP64 instruction; an infinity or a NaN is at
// least MAX_BAD. Of the currents' dx and x, then the potentials'.
constexpr unsigned MAX_BAD = 0x7ff00000u;
struct Maxima {
    unsigned v[4] = {0, 0, 0, 0};
    TAGS_D void take(bool current, double2 d, double2 x) {
        const unsigned a = (unsigned)__double2hiint(cabs1(d)), c = (unsigned)__double2hiint(cabs1(x));
        v[0] = max(v[0], current ? a : 0u);
        v[1] = max(v[1], current ? c : 0u);
        v[2] = max(v[2], current ? 0u : a);
        v[3] = max(v[3], current ? 0u : c);
    }
    TAGS_D double value(int q) const { return __hiloint2double((int)v[q], 0); }
    TAGS_D bool bad() const { return max(max(v[0], v[1]), max(v[2], v[3])) >= MAX_BAD; }
};
// Over a CTA of W warps; complete in thread 0. Ends with no barrier.
template <int W>
TAGS_D void maxima_reduce(Maxima& mx, unsigned (*sm)[W]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned r = __reduce_max_sync(0xffffffffu, mx.v[q]);
        if ((threadIdx.x & 31) == 0) sm[q][threadIdx.x >> 5] = r;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        for (int w = 0; w < W; ++w) mx.v[q] = max(mx.v[q], sm[q][w]);
}
// What a step's maxima mean after corrections of prev (volts and amperes, updated):
// 0 go on, 1 settled, 2 to the pivoted LU.
TAGS_D int step_state(const Maxima& mx, int step, bool last, double* prev) {
    bool done = true, stuck = last;
    for (int q = 0; q < 2; ++q) {
        const double dn = mx.value(2 * q);
        if (step > 0 && !settled(dn, prev[q], mx.value(2 * q + 1))) {
            done = false;
            stuck = stuck || dn > 0.5 * prev[q];
        }
        prev[q] = dn;
    }
    return mx.bad() ? 2 : step == 0 ? 0 : done ? 1 : stuck ? 2 : 0;
}

// x += dx and the stopping rule, one CTA per sample. Step 0's correction is x
// itself. Unknowns below nc are currents. A correction that has not settled and
// did not halve, or is the last step's, leaves the sample to the pivoted LU.
__global__ void __launch_bounds__(256) k_ldl64_apply(const double2* __restrict__ S0, double2* __restrict__ X0, int N,
                                                     int nc, int step, int last, int* __restrict__ active,
                                                     int* __restrict__ conv, double* __restrict__ prev) {
    const int b = blockIdx.x;
    if (!active[b]) return;
    __shared__ unsigned smx[4][8];
    Maxima mx;
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
        const long long o = (long long)N * b + j;
        const double2 d = S0[o], x = cadd(X0[o], d);
        X0[o] = x;
        mx.take(j < nc, d, x);
    }
    maxima_reduce<8>(mx, smx);
    if (threadIdx.x != 0) return;
    const int state = step_state(mx, step, last != 0, prev + 2 * b);
    if (state == 1) conv[b] = 1;
    if (state != 0) active[b] = 0;
}

// Solutions to the original order; info 0, or the mark of a sample that needs more
// corrections (its last one still contracted) or the pivoted LU.
__global__ void k_ldl64_out(const double2* __restrict__ X0, int m, int n, const int* __restrict__ active,
                            const int* __restrict__ conv, double2* __restrict__ out, long long ostride,
                            int* __restrict__ info) {
    const int N = n + 2 * m, b = blockIdx.y;
    const int ip = blockIdx.x * blockDim.x + threadIdx.x;
    if (ip == 0) info[b] = conv[b] ? 0 : active[b] ? TAGS_INFO_MORE : TAGS_INFO_RESOLVE;
    if (ip >= N) return;
    out[ostride * b + orig_index(ip, m, n)] = X0[(long long)N * b + ip];
}

// ---- the plan's system: impedance blocks in the coupling blocks, sparse incidence

// Lower triangle from the stored ZL, ZT (negated) and the incidence; a CTA
// writes one column of one sample.
__global__ void __launch_bounds__(128) k_ldl64_build(double2* __restrict__ W0, long long ld, long long stride,
                                                     const Incidence inc, int m, int n) {
    double2* W = W0 + stride * blockIdx.y;
    const int N = n + 2 * m, j = blockIdx.x;
    double2* col = W + ld * j;
    const double2 zero = cz(0.0, 0.0);
    if (j >= 2 * m) {
        for (int i = j + (int)threadIdx.x; i < N; i += blockDim.x) col[i] = zero;
        return;
    }
    const int bj = j < m ? 0 : 1, e = j - bj * m;
    // the stored block's column e, indexed by the matrix row: ZL (i, m + e), ZT (i, e)
    const double2* z = W + ld * (bj == 0 ? m + e : e);
    for (int i = j + (int)threadIdx.x; i < (bj + 1) * m; i += blockDim.x) col[i] = cneg(z[i]);
    for (int i = 2 * m + (int)threadIdx.x; i < N; i += blockDim.x) col[i] = zero;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int q = inc.seg_ptr[e]; q < inc.seg_ptr[e + 1]; ++q)
            col[2 * m + inc.seg_node[q]] = cz(bj == 0 ? (double)inc.seg_a[q] : 0.5, 0.0);
}

// r = b - W x: impedance rows (blockIdx.y 0: I_L, 1: I_T), a thread per row
// over the stored blocks' columns; FP64-bound (4 multiply-adds per 16 bytes).
__global__ void __launch_bounds__(64) k_ldl64_resid_z(const double2* __restrict__ W0, long long ld, long long stride,
                                                      const Incidence inc, int m, int n,
                                                      const double2* __restrict__ B0, const double2* __restrict__ X0,
                                                      double2* __restrict__ R0, const int* __restrict__ active) {
    const int b = blockIdx.z, blk = blockIdx.y;
    if (!active[b]) return;
    __shared__ double2 xs[64];
    const int N = n + 2 * m, k = blockIdx.x * blockDim.x + threadIdx.x;
    const double2* X = X0 + (long long)N * b;
    const double2* z = W0 + stride * b + (blk == 0 ? ld * m : (long long)m);
    double2 acc = cz(0.0, 0.0);
    for (int j0 = 0; j0 < m; j0 += 64) {
        const int nj = min(64, m - j0);
        __syncthreads();
        if ((int)threadIdx.x < nj) xs[threadIdx.x] = X[blk * m + j0 + threadIdx.x];
        __syncthreads();
        if (k < m) {
#pragma unroll 8
            for (int j = 0; j < nj; ++j) acc = cfma(z[k + ld * (j0 + j)], xs[j], acc);
        }
    }
    if (k >= m) return;
    double2 u = cz(0.0, 0.0);
    for (int q = inc.seg_ptr[k]; q < inc.seg_ptr[k + 1]; ++q)
        u = cadd(u, cscale(X[2 * m + inc.seg_node[q]], blk == 0 ? (double)inc.seg_a[q] : 0.5));
    const long long o = (long long)N * b + blk * m + k;
    R0[o] = cadd(csub(B0[o], u), acc);
}

__global__ void k_ldl64_resid_nodes(const Incidence inc, int m, int n, const double2* __restrict__ B0,
                                    const double2* __restrict__ X0, double2* __restrict__ R0,
                                    const int* __restrict__ active) {
    const int b = blockIdx.y;
    if (!active[b]) return;
    const int N = n + 2 * m, row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n) return;
    const double2* X = X0 + (long long)N * b;
    double2 acc = cz(0.0, 0.0);
    for (int q = inc.node_ptr[row]; q < inc.node_ptr[row + 1]; ++q) {
        const int e = inc.node_seg[q];
        const double a = inc.node_a[q];
        const double2 il = X[e], it = X[m + e];
        acc.x += a * il.x + 0.5 * it.x;
        acc.y += a * il.y + 0.5 * it.y;
    }
    const long long o = (long long)N * b + 2 * m + row;
    R0[o] = csub(B0[o], acc);
}

// ---- small systems: one CTA per sample does it all

constexpr int SMALL_N = 64;
constexpr size_t small_smem(int N) { return sizeof(double2) * ((size_t)N * (N | 1) + 5 * (size_t)N); }

// The whole solve of a sample with N <= 64 unknowns in shared memory: build,
// LDL^T column by column (the columns of a step go round the four warps),
// solves by one warp (a lane per row), refinement as in the launches above.
// Bound by the FP64 instructions of a step's pivot and columns, ~2000 SM
// cycles; 100 rods of 10 segments take 60 us where the panel launches took
// ~450.
__global__ void __launch_bounds__(128) k_ldl64_small(const double2* __restrict__ W0, long long ld, long long stride,
                                                     const Incidence inc, int m, int n,
                                                     const double2* rhs, double2* out,   // may be the same
                                                     double2* __restrict__ saved, int* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int N = n + 2 * m, P = N | 1, b = blockIdx.x;
    double2* A = reinterpret_cast<double2*>(smem_raw);     // (r, c) at c P + r
    double2* bv = A + (size_t)N * P;
    double2 *x = bv + N, *r = x + N, *dinv = r + N, *z = dinv + N;
    __shared__ unsigned smx[4][4];
    __shared__ int sstate;                                  // 0: go on, 1: done, 2: to the pivoted LU
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double2* W = W0 + stride * b;
    for (int t = tid; t < N * P; t += 128) A[t] = cz(0.0, 0.0);
    for (int i = tid; i < N; i += 128) {
        const double2 v = rhs[(long long)N * b + orig_index(i, m, n)];
        bv[i] = r[i] = v;
        x[i] = cz(0.0, 0.0);
        saved[(long long)N * b + i] = v;
    }
    __syncthreads();
    for (int t = tid; t < 2 * m * m; t += 128) {
        const int blk = t / (m * m), u = t - blk * m * m, c = u / m, i = u - c * m;
        if (i >= c) A[(blk * m + c) * P + blk * m + i] = cneg(blk == 0 ? W[i + ld * (m + c)] : W[m + i + ld * c]);
    }
    for (int e = tid; e < m; e += 128)
        for (int q = inc.seg_ptr[e]; q < inc.seg_ptr[e + 1]; ++q) {
            A[e * P + 2 * m + inc.seg_node[q]] = cz((double)inc.seg_a[q], 0.0);
            A[(m + e) * P + 2 * m + inc.seg_node[q]] = cz(0.5, 0.0);
        }
    __syncthreads();
    for (int k = 0; k < N; ++k) {
        const double2 di = crecip(A[k * P + k]);
        if (tid == 0) dinv[k] = di;
        // rows lane and lane + 32 of this warp's columns
        const int r1 = lane + 32;
        const double2 l0 = lane < N ? cneg(cmul(A[k * P + lane], di)) : cz(0.0, 0.0);
        const double2 l1 = r1 < N ? cneg(cmul(A[k * P + r1], di)) : cz(0.0, 0.0);
        for (int c = k + 1 + warp; c < N; c += 4) {
            if (k < m && c >= m && c < 2 * m) continue;     // the ZL/ZT coupling stays zero
            const double2 w = A[k * P + c];
            if (c < 32 && lane >= c && lane < N) A[c * P + lane] = cfma(l0, w, A[c * P + lane]);
            if (r1 >= c && r1 < N) A[c * P + r1] = cfma(l1, w, A[c * P + r1]);
        }
        __syncthreads();
    }
    for (int t = tid; t < N * N; t += 128) {
        const int c = t / N, i = t - c * N;
        if (i > c) A[c * P + i] = cmul(A[c * P + i], dinv[c]);
    }
    __syncthreads();
    double prev[2] = {0.0, 0.0};
    for (int step = 0; step < TAGS_RESOLVE_STEPS; ++step) {
        if (step > 0) {
            for (int i = tid; i < N; i += 128) {
                double2 a = cz(0.0, 0.0), u = cz(0.0, 0.0);
                if (i < 2 * m) {
                    const int blk = i < m ? 0 : 1, k = i - blk * m;
                    const double2* zc = W + (blk == 0 ? ld * m : (long long)m) + k;
                    for (int j = 0; j < m; ++j) a = cfma(zc[ld * j], x[blk * m + j], a);
                    for (int q = inc.seg_ptr[k]; q < inc.seg_ptr[k + 1]; ++q)
                        u = cadd(u, cscale(x[2 * m + inc.seg_node[q]], blk == 0 ? (double)inc.seg_a[q] : 0.5));
                } else {
                    const int k = i - 2 * m;
                    for (int q = inc.node_ptr[k]; q < inc.node_ptr[k + 1]; ++q)
                        u = cadd(u, cadd(cscale(x[inc.node_seg[q]], (double)inc.node_a[q]),
                                         cscale(x[m + inc.node_seg[q]], 0.5)));
                }
                r[i] = cadd(csub(bv[i], u), a);
            }
            __syncthreads();
        }
        if (warp == 0) {
            for (int k = 0; k < N; ++k) {
                const double2 rk = cneg(r[k]);
                if (lane > k && lane < N) r[lane] = cfma(A[k * P + lane], rk, r[lane]);
                if (lane + 32 > k && lane + 32 < N) r[lane + 32] = cfma(A[k * P + lane + 32], rk, r[lane + 32]);
                __syncwarp();
            }
            for (int i = lane; i < N; i += 32) z[i] = cmul(r[i], dinv[i]);
            __syncwarp();
            for (int k = N - 1; k > 0; --k) {
                const double2 zk = cneg(z[k]);
                if (lane < k) z[lane] = cfma(A[lane * P + k], zk, z[lane]);
                if (lane + 32 < k) z[lane + 32] = cfma(A[(lane + 32) * P + k], zk, z[lane + 32]);
                __syncwarp();
            }
        }
        __syncthreads();
        Maxima mx;
        for (int i = tid; i < N; i += 128) {
            const double2 d = z[i], v = cadd(x[i], d);
            x[i] = v;
            mx.take(i < 2 * m, d, v);
        }
        maxima_reduce<4>(mx, smx);
        if (tid == 0) sstate = step_state(mx, step, step + 1 == TAGS_RESOLVE_STEPS, prev);
        __syncthreads();
        if (sstate) break;
    }
    for (int i = tid; i < N; i += 128) out[(long long)N * b + orig_index(i, m, n)] = x[i];
    if (tid == 0) info[b] = sstate == 1 ? 0 : TAGS_INFO_RESOLVE;
}

// ---- a caller's symmetric matrix (full, original order)

// Lower triangle in the static order; *coupled is raised by a nonzero entry
// of the ZL/ZT coupling block.
__global__ void k_ldl64_permute(const double2* __restrict__ W, double2* __restrict__ A, int m, int n,
                                int* __restrict__ coupled) {
    const int N = n + 2 * m, j = blockIdx.x;
    const int i = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= N || i < j) return;
    const double2 v = W[orig_index(i, m, n) + (long long)N * orig_index(j, m, n)];
    A[i + (long long)N * j] = v;
    if (j < m && i >= m && i < 2 * m && (v.x != 0.0 || v.y != 0.0)) *coupled = 1;
}

// r = b - W x for the full symmetric W in the original order, x and r in the
// static order; a warp per row, read as the column (95 us with a thread per row
// at N = 285). The node columns are summed apart from the currents': an impedance
// row's potential difference is then exact in the incidence's two entries, as in
// k_ldl64_resid_z. In one sum the potentials' rounding, eps |U|, drowns ZL I_L
// towards DC: longitudinal currents of a 60 m grid at |s| = 0.01 / s, kappa = 1e-4
// S/m came out at 3.7e-7, now 2e-15.
__global__ void __launch_bounds__(128) k_ldl64_resid_full(const double2* __restrict__ W, int m, int n,
                                                          const double2* __restrict__ B,
                                                          const double2* __restrict__ X, double2* __restrict__ R,
                                                          const int* __restrict__ active) {
    if (!active[0]) return;
    const int N = n + 2 * m, ip = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (ip >= N) return;
    const double2* row = W + (long long)N * orig_index(ip, m, n);
    double2 cur = cz(0.0, 0.0), pot = cz(0.0, 0.0);
    for (int j = lane; j < N; j += 32) {
        const double2 w = row[orig_index(j, m, n)], x = X[j];
        if (j < 2 * m) cur = cfma(w, x, cur);
        else pot = cfma(w, x, pot);
    }
    for (int o = 16; o > 0; o >>= 1) {
        cur.x += __shfl_xor_sync(0xffffffffu, cur.x, o);
        cur.y += __shfl_xor_sync(0xffffffffu, cur.y, o);
        pot.x += __shfl_xor_sync(0xffffffffu, pot.x, o);
        pot.y += __shfl_xor_sync(0xffffffffu, pot.y, o);
    }
    if (lane == 0) R[ip] = csub(csub(B[ip], pot), cur);
}

// ---- many right-hand sides (the nodal admittance drop-ins)

// X = Z^-1 [rhs, I] for R = n + M right-hand sides, one refinement of each
// included. Columns do not depend on one another, so a CTA takes ct of them
// through everything in shared memory: both sweeps, the residual against Z,
// both sweeps again. A warp's unit of work is 32 rows of one column, a lane per
// row: one load of 16 bytes per four FP64 instructions, which hold the SM's
// quarter for 256 cycles, so L2 and the loads' latency are far from the bound;
// the CTAs take as many columns as give every SM the same number. The backward
// sweep reads U = D L^T from the upper triangle, whose rows lie side by side,
// and so needs 1/D only at the diagonal step. Sums over a panel first, then of
// those: less rounding than one chain. 16 warps, since 8 (two per quarter) leave
// the pipe waiting for L2 at M = 1560 (422 against 317 ms). calculate_yla_ytb
// against launches per panel over 32-column tiles: M = 4, n = 4 0.23 -> 0.11 ms,
// 220 and 121 2.74 -> 1.53, 600 and 400 24.2 -> 18.5, 1560 and 1417 362 -> 317.
constexpr int MCOLS_THREADS = 512;
constexpr int MCOLS_MAX = 8;              // columns of a CTA, at most
constexpr size_t MCOLS_SMEM = 227 * 1024 - 64;

// part -> X_p of the diagonal step: y = L11^-1 X_p (upper = 0), L11^-T (D^-1 X_p) (upper = 1).
// A unit is one column's sum over eight terms.
TAGS_D void mcols_block(const double2* __restrict__ ws, double2* x, int M, int ct, const Panel& q, int upper,
                        double2* raw, double2* part, double2* y) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < PB * ct; t += MCOLS_THREADS) {
        const int k = t % PB, c = t / PB;
        double2 v = k < q.jb ? x[c * M + q.j0 + k] : cz(0.0, 0.0);
        if (upper) v = cmul(v, ws[k * (PB + 1)]);
        raw[t] = v;
    }
    __syncthreads();
    for (int u = warp; u < 4 * ct; u += MCOLS_THREADS / 32) {
        const int c = u >> 2, k0 = 8 * (u & 3);
        double2 a = (u & 3) == 0 ? raw[c * PB + lane] : cz(0.0, 0.0);
        for (int k = k0; k < k0 + 8; ++k)
            if (upper ? k > lane : k < lane)
                a = cfma(ws[upper ? lane * PB + k : k * PB + lane], raw[c * PB + k], a);
        part[u * PB + lane] = a;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < PB * ct; t += MCOLS_THREADS) {
        const int k = t % PB, c = t / PB;
        const double2* pc = part + 4 * c * PB + k;
        const double2 a = cadd(cadd(pc[0], pc[PB]), cadd(pc[2 * PB], pc[3 * PB]));
        y[t] = a;
        if (k < q.jb) x[c * M + q.j0 + k] = a;
    }
    __syncthreads();
}

// x (M x ct in shared memory) <- Z^-1 x.
TAGS_D void mcols_sweeps(const double2* __restrict__ A, const double2* __restrict__ ws, double2* x, int M, int ct,
                         double2* raw, double2* part, double2* y) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, P = panel_count(M, 0);
    for (int s = 0; s < 2 * P; ++s) {
        const int bwd = s >= P, p = bwd ? 2 * P - 1 - s : s;
        const Panel q = panel_at(p, M, 0);
        mcols_block(ws + (long long)p * PB * PB, x, M, ct, q, bwd, raw, part, y);
        const int r0 = bwd ? 0 : q.base, nr = bwd ? q.j0 : q.cnt, groups = (nr + 31) / 32;
        const double2* L = A + r0 + (long long)M * q.j0;           // L21, or the rows of U above the block
        for (int u = warp; u < groups * ct; u += MCOLS_THREADS / 32) {
            const int c = u % ct, v = 32 * (u / ct) + lane;
            if (v >= nr) continue;
            double2 acc = cz(0.0, 0.0);
#pragma unroll 8
            for (int k = 0; k < q.jb; ++k) acc = cfma(L[v + (long long)M * k], y[c * PB + k], acc);
            x[c * M + r0 + v] = csub(x[c * M + r0 + v], acc);
        }
        __syncthreads();
    }
}

constexpr size_t mcols_smem(int M, int ct) { return sizeof(double2) * ((2 * (size_t)M + 6 * PB) * ct); }

__global__ void __launch_bounds__(MCOLS_THREADS) k_ldl64_mcols(const double2* __restrict__ Z0,
                                                               const double2* __restrict__ A0, int M,
                                                               const double2* __restrict__ ws0, long long wstride,
                                                               const double2* __restrict__ B0, int n, int R, int ct,
                                                               double2* __restrict__ X0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int b = blockIdx.y, c0 = blockIdx.x * ct, nc = min(ct, R - c0);
    const long long MM = (long long)M * M;
    const double2 *Z = Z0 + MM * b, *A = A0 + MM * b, *ws = ws0 + wstride * b, *B = B0 + (long long)M * n * b;
    double2* x = reinterpret_cast<double2*>(smem_raw);
    double2* e = x + (long long)M * ct;
    double2 *raw = e + (long long)M * ct, *y = raw + PB * ct, *part = y + PB * ct;
    auto rhs = [&](int i, int c) {
        return c0 + c < n ? B[i + (long long)M * (c0 + c)] : cz(c0 + c - n == i ? 1.0 : 0.0, 0.0);
    };
    for (int t = threadIdx.x; t < M * nc; t += MCOLS_THREADS) x[t] = rhs(t % M, t / M);
    __syncthreads();
    mcols_sweeps(A, ws, x, M, nc, raw, part, y);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int u = warp; u < (M + 31) / 32 * nc; u += MCOLS_THREADS / 32) {
        const int c = u % nc, i = 32 * (u / nc) + lane;
        if (i >= M) continue;
        double2 tot = cz(0.0, 0.0);
        for (int k0 = 0; k0 < M; k0 += PB) {
            double2 acc = cz(0.0, 0.0);
#pragma unroll 8
            for (int k = k0; k < min(k0 + PB, M); ++k) acc = cfma(Z[i + (long long)M * k], x[c * M + k], acc);
            tot = cadd(tot, acc);
        }
        e[c * M + i] = csub(rhs(i, c), tot);
    }
    __syncthreads();
    mcols_sweeps(A, ws, e, M, nc, raw, part, y);
    double2* X = X0 + (long long)M * R * b + (long long)M * c0;
    for (int t = threadIdx.x; t < M * nc; t += MCOLS_THREADS) X[t] = cadd(x[t], e[t]);
}

// Signs of the check's combination of right-hand sides.
TAGS_D double check_sign(int r) { return (((unsigned)r * 2654435761u) >> 15) & 1u ? 1.0 : -1.0; }

// Check of the whole solve on one random combination of its right-hand sides:
// v = sum_r sign_r X_r, u = sum_r sign_r B_r (B = [rhs, I]). Warp per row.
__global__ void __launch_bounds__(128) k_ldl64_check_sum(const double2* __restrict__ X0, const double2* __restrict__ B0,
                                                         int M, int n, long long xstride, long long bstride,
                                                         double2* __restrict__ vu0) {
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, b = blockIdx.y;
    if (row >= M) return;
    double2 v = cz(0.0, 0.0), u = cz(0.0, 0.0);
    for (int r = lane; r < n + M; r += 32) {
        const double sg = check_sign(r);
        const double2 x = X0[xstride * b + row + (long long)M * r];
        v.x += sg * x.x;
        v.y += sg * x.y;
        if (r < n) {
            const double2 w = B0[bstride * b + row + (long long)M * r];
            u.x += sg * w.x;
            u.y += sg * w.y;
        } else if (r - n == row) {
            u.x += sg;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        u.x += __shfl_xor_sync(0xffffffffu, u.x, o);
        u.y += __shfl_xor_sync(0xffffffffu, u.y, o);
    }
    if (lane == 0) {
        vu0[(2LL * b) * M + row] = v;
        vu0[(2LL * b + 1) * M + row] = u;
    }
}

// Row by row |Z v - u| against 1e-14 (sum |Z| |v| + |u|), the backward error
// of a stable solve with room for M ~ 50 eps; *bad is raised above it (or by a
// value that is not finite). Z: full symmetric. Warp per row.
__global__ void __launch_bounds__(128) k_ldl64_check(const double2* __restrict__ Z0, int M, long long zstride,
                                                     const double2* __restrict__ vu0, int* __restrict__ bad) {
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, b = blockIdx.y;
    if (row >= M) return;
    const double2* v = vu0 + 2LL * b * M;
    const double2 u = v[M + row];
    double2 acc = cz(0.0, 0.0);
    double mag = 0.0;
    for (int j = lane; j < M; j += 32) {
        const double2 z = Z0[zstride * b + j + (long long)M * row], x = v[j];
        acc = cfma(z, x, acc);
        mag = fma(cabs1(z), cabs1(x), mag);
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        mag += __shfl_xor_sync(0xffffffffu, mag, o);
    }
    if (lane == 0 && !(cabs1(csub(acc, u)) <= 1e-14 * (mag + cabs1(u)))) *bad = 1;
}

struct Ws {
    double2 *linv, *b, *x, *r, *z;
    double* prev;
    int *active, *conv;
    long long wstride;      // linv values per sample
};

Ws carve(void* p, int N, int batch) {
    Ws w;
    // the most panels any split of N into blocks can have
    w.wstride = (long long)((N + PB - 1) / PB + 2) * PB * PB;
    w.linv = reinterpret_cast<double2*>(p);
    w.b = w.linv + w.wstride * batch;
    w.x = w.b + (long long)N * batch;
    w.r = w.x + (long long)N * batch;
    w.z = w.r + (long long)N * batch;
    w.prev = reinterpret_cast<double*>(w.z + (long long)N * batch);
    w.active = reinterpret_cast<int*>(w.prev + 2 * batch);
    w.conv = w.active + batch;
    return w;
}

constexpr int SOLVE_N_MAX = 14000;        // 16 B per unknown in the one-CTA solve's shared memory

// Split of a panel's rows (the identity's 32 included): lanes per row, groups
// of rows per CTA, CTAs per sample. Taken is what leaves the busiest SM the
// least FP64 instructions per warp: 690 for a CTA's block and 576, 320 or 192
// per group of 32, 16 or 8 rows.
int panel_split(int rows, int nb, int& lpr, int& passes) {
    const int sms = tags_num_sms();
    long long best = -1;
    int ctas = 1;
    for (int l = 4, ins = 576; l <= 16; l *= 2, ins = l == 8 ? 320 : 192)
        for (int ps = 1, last = 0; ps <= 16; ++ps) {
            const int groups = (rows * l + 127) / 128, c = (groups + ps - 1) / ps;
            if (c == last) continue;                       // as many CTAs with fewer passes
            last = c;
            const long long cost = ((long long)nb * c + sms - 1) / sms * (690 + ins * ps);
            if (best < 0 || cost < best) {
                best = cost;
                lpr = l;
                passes = ps;
                ctas = c;
            }
        }
    return ctas;
}

int factor(double2* A, int N, long long ld, long long stride, int nb, int m, const Ws& w, cudaStream_t st) {
    const int P = panel_count(N, m), sms = tags_num_sms();
    for (int p = 0; p < P; ++p) {
        const Panel q = panel_at(p, N, m);
        int lpr, passes;
        const int ctas = panel_split(q.cnt + PB, nb, lpr, passes);
        int pf = tags_prof_begin(TAGS_PROF_LU64_OTHER, st);
        auto panel = lpr == 16 ? k_ldl64_panel<16> : lpr == 8 ? k_ldl64_panel<8> : k_ldl64_panel<4>;
        panel<<<dim3(ctas, nb), 128, 0, st>>>(A, ld, stride, q, p, w.linv, w.wstride, passes);
        tags_prof_end(TAGS_PROF_LU64_OTHER, pf, st, 0.0, 0.0);
        tags_note_launch();
        if (q.cnt <= 0) continue;
        // the largest tile that wastes little on the diagonal and the edge (ten
        // tile rows) and fills the SMs
        pf = tags_prof_begin(TAGS_PROF_LU64_GEMM, st);
        const long long t64 = (q.cnt + 63) / 64, t32 = (q.cnt + 31) / 32, t16 = (q.cnt + 15) / 16;
        if (t64 >= 10 && t64 * (t64 + 1) / 2 * nb >= 4 * sms)
            k_ldl64_update<64, 4><<<dim3((unsigned)(t64 * (t64 + 1) / 2), nb), 256, 6 * PB * 64 * sizeof(double), st>>>(
                A, ld, stride, q);
        else if (t32 >= 10 && t32 * (t32 + 1) / 2 * nb >= 2 * sms)
            k_ldl64_update<32, 2><<<dim3((unsigned)(t32 * (t32 + 1) / 2), nb), 256, 6 * PB * 32 * sizeof(double), st>>>(
                A, ld, stride, q);
        else
            k_ldl64_update<16, 1><<<dim3((unsigned)(t16 * (t16 + 1) / 2), nb), 256, 6 * PB * 16 * sizeof(double), st>>>(
                A, ld, stride, q);
        // the three real products' flops, 6 per complex multiply-add
        tags_prof_end(TAGS_PROF_LU64_GEMM, pf, st, 3.0 * q.cnt * (q.cnt + 1.0) * q.jb * nb,
                      (16.0 * q.cnt * (q.cnt + 1.0) + 32.0 * q.cnt * q.jb) * nb);
        tags_note_launch();
    }
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

// w.z = W^-1 w.r for the active samples (w.r is used up); the right-hand side
// is zero above row `lead`.
int solve(const double2* A, int N, long long ld, long long stride, int nb, int m, const Ws& w, int lead,
          cudaStream_t st) {
    const int P = panel_count(N, m);
    int p0 = 0;
    while (p0 + 1 < P && panel_at(p0, N, m).base <= lead) ++p0;
    int pf = tags_prof_begin(TAGS_PROF_LU64_OTHER, st);
    if (N > 64 && N <= SCL_N && nb <= tags_num_sms() / SCL_G * (N <= 320 ? 2 : 1)) {
        k_ldl64_solve_cl<<<dim3(SCL_G, nb), 128, scl_smem(N), st>>>(A, ld, stride, N, m, w.linv, w.wstride, w.r, w.z, p0,
                                                                    w.active);
        tags_prof_end(TAGS_PROF_LU64_OTHER, pf, st, 0.0, 0.0);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        return 0;
    }
    if (N <= 320 || (nb >= 128 && N <= SOLVE_N_MAX)) {
        k_ldl64_solve_cta<<<nb, SOLVE_THREADS, sizeof(double2) * N, st>>>(A, ld, stride, N, m, w.linv, w.wstride, w.r,
                                                                          w.z, p0, w.active);
        tags_prof_end(TAGS_PROF_LU64_OTHER, pf, st, 0.0, 0.0);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        return 0;
    }
    TAGS_CUDA_OK(cudaMemsetAsync(w.z, 0, sizeof(double2) * N * nb, st));
    for (int p = p0; p < P; ++p) {
        const Panel q = panel_at(p, N, m);
        k_ldl64_fwd<<<dim3(q.cnt > 0 ? (q.cnt + 31) / 32 : 1, nb), 128, 0, st>>>(A, ld, stride, q, p, w.linv,
                                                                                w.wstride, w.r, w.z, N, w.active);
    }
    k_ldl64_dscale<<<dim3((N + 127) / 128, nb), 128, 0, st>>>(w.z, N, m, w.linv, w.wstride, w.active);
    // the backward sweep runs on z and leaves the solution in r; then r -> z
    for (int p = P - 1; p >= 0; --p) {
        const Panel q = panel_at(p, N, m);
        const int c0 = m > 0 && q.j0 >= m && q.j0 < 2 * m ? m : 0, left = q.j0 - c0;
        k_ldl64_bwd<<<dim3(left > 0 ? (left + 31) / 32 : 1, nb), 128, 0, st>>>(A, ld, stride, q, p, c0, w.linv,
                                                                              w.wstride, w.z, w.r, N, w.active);
    }
    TAGS_CUDA_OK(cudaMemcpyAsync(w.z, w.r, sizeof(double2) * N * nb, cudaMemcpyDeviceToDevice, st));
    tags_prof_end(TAGS_PROF_LU64_OTHER, pf, st, 0.0, 0.0);
    tags_note_launch(2 * P - p0 + 1);
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

}  // namespace

// Kernel attributes, once per device, before any launch and any graph capture.
int tags_ldl64_prepare() {
    static PerDevice state;
    return tags_once_per_device(state, [] {
        if (cudaFuncSetAttribute(k_ldl64_mcols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MCOLS_SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_ldl64_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)small_smem(SMALL_N)) != cudaSuccess ||
            cudaFuncSetAttribute(k_ldl64_update<64, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(6 * PB * 64 * sizeof(double))) != cudaSuccess ||
            cudaFuncSetAttribute(k_ldl64_update<32, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(6 * PB * 32 * sizeof(double))) != cudaSuccess ||
            cudaFuncSetAttribute(k_ldl64_solve_cta, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(SOLVE_N_MAX * sizeof(double2))) != cudaSuccess)
            return tags_fail(TAGS_E_CUDA, "cudaFuncSetAttribute(k_ldl64) failed");
        return 0;
    });
}

size_t tags_ldl64_workspace(int N, int batch) {
    const size_t per = sizeof(double2) * (((size_t)(N + PB - 1) / PB + 2) * PB * PB + 4 * (size_t)N) +
                       2 * (sizeof(double) + sizeof(int));
    return per * batch + 64;
}

FillOut tags_ldl64_fill_out(double2* W, int m, int n) {
    const long long N = n + 2LL * m;
    FillOut out{};
    out.zl = W;
    out.zt = W;
    out.ld = N;
    out.batch_stride = N * N;
    out.col0_l = m;
    out.row0_t = m;
    out.sign = 1.0;
    out.mirror = 1;
    return out;
}

// Corrections [from, to) of the plan's system, then the solutions and info.
static int corrections(const double2* W, const Incidence& inc, int m, int n, int nb, const Ws& w, int from, int to,
                       double2* x, int* info, cudaStream_t st) {
    const int N = n + 2 * m;
    const long long NN = (long long)N * N;
    for (int step = from; step < to; ++step) {
        if (step > 0) {
            k_ldl64_resid_z<<<dim3((m + 63) / 64, 2, nb), 64, 0, st>>>(W, N, NN, inc, m, n, w.b, w.x, w.r, w.active);
            k_ldl64_resid_nodes<<<dim3((n + 127) / 128, nb), 128, 0, st>>>(inc, m, n, w.b, w.x, w.r, w.active);
            tags_note_launch(2);
        }
        if (int e = solve(W, N, N, NN, nb, m, w, step == 0 ? 2 * m : 0, st)) return e;
        k_ldl64_apply<<<nb, 256, 0, st>>>(w.z, w.x, N, 2 * m, step, step + 1 == TAGS_RESOLVE_STEPS, w.active, w.conv,
                                          w.prev);
        tags_note_launch();
    }
    k_ldl64_out<<<dim3((N + 127) / 128, nb), 128, 0, st>>>(w.x, m, n, w.active, w.conv, x, N, info);
    tags_note_launch();
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

int tags_ldl64_plan_solve(double2* W, const Incidence& inc, int m, int n, int nb, int batch, void* ws,
                          const double2* rhs, double2* x, int* info, int steps, cudaStream_t st) {
    if (int e = tags_ldl64_prepare()) return e;
    const int N = n + 2 * m;
    const long long NN = (long long)N * N;
    const Ws w = carve(ws, N, batch);
    if (N <= SMALL_N) {
        k_ldl64_small<<<nb, 128, small_smem(N), st>>>(W, N, NN, inc, m, n, rhs, x, w.b, info);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        return 0;
    }
    k_ldl64_start<<<dim3((N + 127) / 128, nb), 128, 0, st>>>(rhs, N, m, n, w.b, w.r, w.x, w.active, w.conv);
    k_ldl64_build<<<dim3(N, nb), 128, 0, st>>>(W, N, NN, inc, m, n);
    tags_note_launch(2);
    const int err = factor(W, N, N, NN, nb, m, w, st);
    return err ? err : corrections(W, inc, m, n, nb, w, 0, steps, x, info, st);
}

int tags_ldl64_plan_more(const double2* W, const Incidence& inc, int m, int n, int nb, int batch, void* ws, int* step,
                         double2* x, int* info, cudaStream_t st) {
    const int from = *step;
    *step = std::min(from + 2, TAGS_RESOLVE_STEPS);
    return corrections(W, inc, m, n, nb, carve(ws, n + 2 * m, batch), from, *step, x, info, st);
}

const double2* tags_ldl64_saved_rhs(void* ws, int N, int batch) { return carve(ws, N, batch).b; }

int tags_ldl64_sym_solve(const double2* W, double2* A, int m, int n, void* ws, int* d_words, double2* x, int* info,
                         cudaStream_t st) {
    if (int e = tags_ldl64_prepare()) return e;
    const int N = n + 2 * m;
    const Ws w = carve(ws, N, 1);
    TAGS_CUDA_OK(cudaMemsetAsync(d_words, 0, sizeof(int), st));
    k_ldl64_start<<<dim3((N + 127) / 128, 1), 128, 0, st>>>(x, N, m, n, w.b, w.r, w.x, w.active, w.conv);
    k_ldl64_permute<<<dim3(N, (N + 127) / 128), 128, 0, st>>>(W, A, m, n, d_words);
    tags_note_launch(2);
    int coupled = 0;
    TAGS_CUDA_OK(cudaMemcpyAsync(&coupled, d_words, sizeof(int), cudaMemcpyDeviceToHost, st));
    TAGS_CUDA_OK(cudaStreamSynchronize(st));
    const int zm = coupled ? 0 : m;          // the structure skipped by the elimination, if it is there
    int err = factor(A, N, N, 0, 1, zm, w, st);
    // three corrections, and where they still contract without having settled, more
    *info = TAGS_INFO_MORE;
    for (int step = 0; *info == TAGS_INFO_MORE && !err;) {
        for (const int end = step == 0 ? 3 : TAGS_RESOLVE_STEPS; step < end && !err; ++step) {
            if (step > 0) {
                k_ldl64_resid_full<<<(N + 3) / 4, 128, 0, st>>>(W, m, n, w.b, w.x, w.r, w.active);
                tags_note_launch();
            }
            err = solve(A, N, N, 0, 1, zm, w, 0, st);
            if (err) return err;
            k_ldl64_apply<<<1, 256, 0, st>>>(w.z, w.x, N, 2 * m, step, step + 1 == TAGS_RESOLVE_STEPS, w.active, w.conv,
                                             w.prev);
            tags_note_launch();
        }
        k_ldl64_out<<<dim3((N + 127) / 128, 1), 128, 0, st>>>(w.x, m, n, w.active, w.conv, x, N, d_words + 1);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        TAGS_CUDA_OK(cudaMemcpyAsync(info, d_words + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        TAGS_CUDA_OK(cudaStreamSynchronize(st));
    }
    return err;
}

bool tags_ldl64_multi_fits(int M) { return mcols_smem(M, 1) <= MCOLS_SMEM; }

size_t tags_ldl64_multi_workspace(int M) {
    return 2 * sizeof(double2) * (((size_t)(M + PB - 1) / PB + 2) * PB * PB + 2 * (size_t)M + (size_t)M * M) +
           64;
}

int tags_ldl64_multi_solve(const double2* Z, const double2* rhs, int M, int n, int nb, double2* X, void* wsp,
                           int* d_bad, cudaStream_t st) {
    if (int e = tags_ldl64_prepare()) return e;
    const int R = n + M;
    const long long MM = (long long)M * M, MR = (long long)M * R, MN = (long long)M * n;
    Ws w{};
    w.wstride = (long long)((M + PB - 1) / PB + 2) * PB * PB;
    w.linv = reinterpret_cast<double2*>(wsp);
    double2* vu = w.linv + w.wstride * nb;           // nb x 2 x M
    double2* A = vu + 2LL * M * nb;                  // nb x M x M, the factors
    TAGS_CUDA_OK(cudaMemsetAsync(d_bad, 0, sizeof(int), st));
    TAGS_CUDA_OK(cudaMemcpyAsync(A, Z, sizeof(double2) * MM * nb, cudaMemcpyDeviceToDevice, st));
    if (int e = factor(A, M, M, MM, nb, 0, w, st)) return e;
    // as many columns per CTA as leave the busiest SM the least to do
    const int sms = tags_num_sms();
    int ct = 1;
    long long best = 0;
    for (int t = 1; t <= MCOLS_MAX && mcols_smem(M, t) <= MCOLS_SMEM; ++t) {
        const long long ctas = (long long)((R + t - 1) / t) * nb, cost = (ctas + sms - 1) / sms * t;
        if (t == 1 || cost <= best) {
            best = cost;
            ct = t;
        }
    }
    // one refinement of every column: the factors were taken without pivoting
    // and the diagonal steps use inverses, so X alone is some times eps off
    k_ldl64_mcols<<<dim3((R + ct - 1) / ct, nb), MCOLS_THREADS, mcols_smem(M, ct), st>>>(Z, A, M, w.linv, w.wstride, rhs,
                                                                                    n, R, ct, X);
    k_ldl64_check_sum<<<dim3((M + 3) / 4, nb), 128, 0, st>>>(X, rhs, M, n, MR, MN, vu);
    k_ldl64_check<<<dim3((M + 3) / 4, nb), 128, 0, st>>>(Z, M, MM, vu, d_bad);
    tags_note_launch(3);
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}
