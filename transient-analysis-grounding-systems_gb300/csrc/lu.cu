// Batched dense complex FP64 LU factorisation and triangular solves (CUDA cores).
//
// Replaces the reference's dense solve of the immittance system,
// solve_immittance -> zsysv('L') (src/linalg.c:112-139), by LU with partial
// pivoting on the symmetrised W_G (row interchanges as in LAPACK's getrf: pivot =
// first index of max |Re|+|Im|): the allocation-free solve, and the systems that
// the FP64 LDL^T in the static order (ldl64.cu) hands over because its check asks
// for a pivot search. Right-looking blocked algorithm with a panel width NB:
// panel factorisation, row interchanges, triangular solve of the block row,
// trailing update C -= L21 * U12.
//
// Layout: column-major, leading dimension ld, one matrix per blockIdx.z
// (pointer + z * stride). ipiv is 0-based global row indices.
#include "tags_common.cuh"
#include "tags_internal.h"
#include "../../include/tags_gpu.h"
#include "plan.h"

namespace {

constexpr int NB = 32;                    // panel width
constexpr int PANEL_THREADS = 512;

// Factor the panel A[j0:n, j0:j0+jb] in place (unblocked, column by column).
// One CTA per matrix. Rows are interchanged inside the panel only; the rest of
// the matrix is swapped by k_laswp afterwards.
__global__ void __launch_bounds__(PANEL_THREADS) k_panel(double2* __restrict__ A0, int n, long long ld, long long stride,
                                                          int j0, int jb, int* __restrict__ ipiv0,
                                                          int* __restrict__ info0) {
    double2* A = A0 + stride * blockIdx.z;
    int* ipiv = ipiv0 + (long long)n * blockIdx.z;
    int* info = info0 + blockIdx.z;
    __shared__ double s_val[PANEL_THREADS / 32];
    __shared__ int s_idx[PANEL_THREADS / 32];
    __shared__ double2 s_row[128];
    __shared__ int s_p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int c = j0; c < j0 + jb; ++c) {
        double best = -1;
        int bi = n;
        for (int r = c + tid; r < n; r += blockDim.x) {
            double v = cabs1(A[r + ld * c]);
            if (v > best) { best = v; bi = r; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            double ov = __shfl_down_sync(0xffffffffu, best, o);
            int oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { s_val[warp] = best; s_idx[warp] = bi; }
        __syncthreads();
        if (tid == 0) {
            double b = s_val[0];
            int i = s_idx[0];
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
                if (s_val[w] > b || (s_val[w] == b && s_idx[w] < i)) { b = s_val[w]; i = s_idx[w]; }
            s_p = (i < n) ? i : c;
        }
        __syncthreads();
        const int p = s_p;
        if (tid == 0) ipiv[c] = p;
        if (p != c) {
            for (int cc = j0 + tid; cc < j0 + jb; cc += blockDim.x) {
                double2 t = A[c + ld * cc];
                A[c + ld * cc] = A[p + ld * cc];
                A[p + ld * cc] = t;
            }
        }
        __syncthreads();
        // pivot row of the panel to shared memory
        for (int cc = c + tid; cc < j0 + jb; cc += blockDim.x) s_row[cc - j0] = A[c + ld * cc];
        __syncthreads();
        double2 piv = s_row[c - j0];
        if (piv.x == 0.0 && piv.y == 0.0) {
            if (tid == 0 && *info == 0) *info = c + 1;
            __syncthreads();
            continue;
        }
        double2 ip = cdiv(cz(1.0, 0.0), piv);
        for (int r = c + 1 + tid; r < n; r += blockDim.x) {
            double2 l = cmul(A[r + ld * c], ip);
            A[r + ld * c] = l;
            double2 nl = cneg(l);
            for (int cc = c + 1; cc < j0 + jb; ++cc) A[r + ld * cc] = cfma(nl, s_row[cc - j0], A[r + ld * cc]);
        }
        __syncthreads();
    }
}

// Apply the interchanges ipiv[j0:j0+jb] to the columns outside the panel.
__global__ void k_laswp(double2* __restrict__ A0, int n, long long ld, long long stride, int j0, int jb,
                        const int* __restrict__ ipiv0) {
    double2* A = A0 + stride * blockIdx.z;
    const int* ipiv = ipiv0 + (long long)n * blockIdx.z;
    int col = blockIdx.x * blockDim.x + threadIdx.x;
    int ncols = n - jb;
    if (col >= ncols) return;
    int j = col < j0 ? col : col + jb;
    for (int c = j0; c < j0 + jb; ++c) {
        int p = ipiv[c];
        if (p != c) {
            double2 t = A[c + ld * j];
            A[c + ld * j] = A[p + ld * j];
            A[p + ld * j] = t;
        }
    }
}

// U12 = L11^{-1} A12, L11 = unit lower jb x jb at (j0, j0), columns j0+jb..n.
// One CTA per 32 columns; the block row tile lives in shared memory.
__global__ void __launch_bounds__(256) k_trsm_row(double2* __restrict__ A0, int n, long long ld, long long stride,
                                                  int j0, int jb) {
    double2* A = A0 + stride * blockIdx.z;
    __shared__ double2 sL[NB][NB + 1];
    __shared__ double2 sX[NB][33];
    const int c0 = j0 + jb + blockIdx.x * 32;
    const int ncol = min(32, n - c0);
    if (ncol <= 0) return;
    for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
        int r = t % jb, c = t / jb;
        sL[r][c] = A[(j0 + r) + ld * (j0 + c)];
    }
    for (int t = threadIdx.x; t < jb * 32; t += blockDim.x) {
        int r = t % jb, c = t / jb;
        sX[r][c] = c < ncol ? A[(j0 + r) + ld * (c0 + c)] : cz(0.0, 0.0);
    }
    __syncthreads();
    for (int k = 0; k < jb; ++k) {
        for (int t = threadIdx.x; t < (jb - k - 1) * 32; t += blockDim.x) {
            int r = k + 1 + t / 32, c = t % 32;
            sX[r][c] = cfma(cneg(sL[r][k]), sX[k][c], sX[r][c]);
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < jb * 32; t += blockDim.x) {
        int r = t % jb, c = t / jb;
        if (c < ncol) A[(j0 + r) + ld * (c0 + c)] = sX[r][c];
    }
}

// Trailing update C -= L21 * U12 over rows/cols [j0+jb, n). 64x64 output tile,
// 256 threads with a 4x4 register tile, K = jb <= NB in one shared stage.
__global__ void __launch_bounds__(256) k_gemm_update(double2* __restrict__ A0, int n, long long ld, long long stride,
                                                     int j0, int jb) {
    double2* A = A0 + stride * blockIdx.z;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* sA = reinterpret_cast<double2*>(smem_raw);          // [NB][64]  (k-major: sA[k*64 + r])
    double2* sB = sA + NB * 64;                            // [NB][64]  (sB[k*64 + c])
    const int base = j0 + jb;
    const int r0 = base + blockIdx.y * 64, c0 = base + blockIdx.x * 64;
    if (r0 >= n || c0 >= n) return;
    for (int t = threadIdx.x; t < jb * 64; t += blockDim.x) {
        int r = t & 63, k = t >> 6;
        int gr = r0 + r;
        sA[k * 64 + r] = gr < n ? A[gr + ld * (j0 + k)] : cz(0.0, 0.0);
        int c = t & 63, kk = t >> 6;
        int gc = c0 + c;
        // U12 row (j0+kk) read along columns: element (j0+kk, gc)
        sB[kk * 64 + c] = gc < n ? A[(j0 + kk) + ld * gc] : cz(0.0, 0.0);
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double2 acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = cz(0.0, 0.0);
    for (int k = 0; k < jb; ++k) {
        double2 av[4], bv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) av[a] = sA[k * 64 + ty + 16 * a];
#pragma unroll
        for (int b = 0; b < 4; ++b) bv[b] = sB[k * 64 + tx + 16 * b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = cfma(av[a], bv[b], acc[a][b]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        int gr = r0 + ty + 16 * a;
        if (gr >= n) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            int gc = c0 + tx + 16 * b;
            if (gc < n) {
                long long idx = gr + ld * gc;
                A[idx] = csub(A[idx], acc[a][b]);
            }
        }
    }
}

// ---- triangular solves with nrhs columns (x overwritten) ---------------------

// Apply ipiv forward (LAPACK laswp order) to the right-hand sides.
__global__ void k_rhs_swap(double2* __restrict__ X0, int n, int nrhs, long long ldx, long long xstride,
                           const int* __restrict__ ipiv0) {
    double2* X = X0 + xstride * blockIdx.z;
    const int* ipiv = ipiv0 + (long long)n * blockIdx.z;
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nrhs) return;
    for (int c = 0; c < n; ++c) {
        int p = ipiv[c];
        if (p != c) {
            double2 t = X[c + ldx * j];
            X[c + ldx * j] = X[p + ldx * j];
            X[p + ldx * j] = t;
        }
    }
}

// Solve the jb x jb diagonal block at j0 (lower unit or upper non-unit) for
// every right-hand side; one CTA per matrix.
__global__ void __launch_bounds__(256) k_trsv_diag(const double2* __restrict__ A0, int n, long long ld, long long stride,
                                                   double2* __restrict__ X0, int nrhs, long long ldx, long long xstride,
                                                   int j0, int jb, int upper) {
    const double2* A = A0 + stride * blockIdx.z;
    double2* X = X0 + xstride * blockIdx.z;
    __shared__ double2 sL[NB][NB + 1];
    __shared__ double2 sx[NB][9];
    for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
        int r = t % jb, c = t / jb;
        sL[r][c] = A[(j0 + r) + ld * (j0 + c)];
    }
    for (int j = 0; j < nrhs; j += 8) {
        int nj = min(8, nrhs - j);
        __syncthreads();
        for (int t = threadIdx.x; t < jb * nj; t += blockDim.x) {
            int r = t % jb, c = t / jb;
            sx[r][c] = X[(j0 + r) + ldx * (j + c)];
        }
        __syncthreads();
        if (!upper) {
            for (int k = 0; k < jb; ++k) {
                for (int t = threadIdx.x; t < (jb - k - 1) * nj; t += blockDim.x) {
                    int r = k + 1 + t / nj, c = t % nj;
                    sx[r][c] = cfma(cneg(sL[r][k]), sx[k][c], sx[r][c]);
                }
                __syncthreads();
            }
        } else {
            for (int k = jb - 1; k >= 0; --k) {
                if (threadIdx.x < nj) sx[k][threadIdx.x] = cmul(sx[k][threadIdx.x], cdiv(cz(1.0, 0.0), sL[k][k]));
                __syncthreads();
                for (int t = threadIdx.x; t < k * nj; t += blockDim.x) {
                    int r = t / nj, c = t % nj;
                    sx[r][c] = cfma(cneg(sL[r][k]), sx[k][c], sx[r][c]);
                }
                __syncthreads();
            }
        }
        for (int t = threadIdx.x; t < jb * nj; t += blockDim.x) {
            int r = t % jb, c = t / jb;
            X[(j0 + r) + ldx * (j + c)] = sx[r][c];
        }
    }
}

// X[rows] -= A[rows, j0:j0+jb] * X[j0:j0+jb]; rows = [j0+jb, n) (lower) or
// [0, j0) (upper). One thread per (row, rhs).
__global__ void k_trsv_update(const double2* __restrict__ A0, int n, long long ld, long long stride,
                              double2* __restrict__ X0, int nrhs, long long ldx, long long xstride, int j0, int jb,
                              int upper) {
    const double2* A = A0 + stride * blockIdx.z;
    double2* X = X0 + xstride * blockIdx.z;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    int j = blockIdx.y;
    int rbeg = upper ? 0 : j0 + jb, rend = upper ? j0 : n;
    r += rbeg;
    if (r >= rend || j >= nrhs) return;
    double2 acc = cz(0.0, 0.0);
    for (int k = 0; k < jb; ++k) acc = cfma(A[r + ld * (j0 + k)], X[(j0 + k) + ldx * j], acc);
    X[r + ldx * j] = csub(X[r + ldx * j], acc);
}

}  // namespace

// Kernel attributes of the LU, set once per device before any launch (and so
// before any graph capture).
int tags_lu_prepare() {
    static PerDevice state;
    return tags_once_per_device(state, [] {
        const int g64 = (int)(2 * NB * 64 * sizeof(double2));
        if (cudaFuncSetAttribute(k_gemm_update, cudaFuncAttributeMaxDynamicSharedMemorySize, g64) !=
            cudaSuccess)
            return tags_fail(TAGS_E_CUDA, "cudaFuncSetAttribute(k_gemm_update) failed");
        return 0;
    });
}

int tags_lu_z(double2* A, int n, long long ld, long long stride, int batch, int* ipiv, int* info, cudaStream_t st) {
    TAGS_CUDA_OK(cudaMemsetAsync(info, 0, sizeof(int) * batch, st));
    const size_t gsmem = 2 * NB * 64 * sizeof(double2);
    if (int e = tags_lu_prepare()) return e;
    for (int j0 = 0; j0 < n; j0 += NB) {
        int jb = min(NB, n - j0);
        k_panel<<<dim3(1, 1, batch), PANEL_THREADS, 0, st>>>(A, n, ld, stride, j0, jb, ipiv, info);
        tags_note_launch();
        int ncols = n - jb;
        if (ncols > 0) {
            k_laswp<<<dim3((ncols + 127) / 128, 1, batch), 128, 0, st>>>(A, n, ld, stride, j0, jb, ipiv);
            tags_note_launch();
        }
        int rest = n - j0 - jb;
        if (rest > 0) {
            k_trsm_row<<<dim3((rest + 31) / 32, 1, batch), 256, 0, st>>>(A, n, ld, stride, j0, jb);
            tags_note_launch();
            dim3 g((rest + 63) / 64, (rest + 63) / 64, batch);
            int pf = tags_prof_begin(TAGS_PROF_LU64_GEMM, st);
            k_gemm_update<<<g, 256, gsmem, st>>>(A, n, ld, stride, j0, jb);
            // rank-jb update of a rest x rest block: 8 rest^2 jb real flops
            tags_prof_end(TAGS_PROF_LU64_GEMM, pf, st, 8.0 * rest * (double)rest * jb * batch,
                          (32.0 * rest * (double)rest + 32.0 * rest * jb) * batch);
            tags_note_launch();
        }
    }
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

int tags_lu_solve_z(const double2* A, int n, long long ld, long long stride, int batch, const int* ipiv, double2* X,
                    int nrhs, long long ldx, long long xstride, cudaStream_t st) {
    k_rhs_swap<<<dim3((nrhs + 31) / 32, 1, batch), 32, 0, st>>>(X, n, nrhs, ldx, xstride, ipiv);
    tags_note_launch();
    for (int j0 = 0; j0 < n; j0 += NB) {
        int jb = min(NB, n - j0);
        k_trsv_diag<<<dim3(1, 1, batch), 256, 0, st>>>(A, n, ld, stride, X, nrhs, ldx, xstride, j0, jb, 0);
        tags_note_launch();
        int rest = n - j0 - jb;
        if (rest > 0) {
            k_trsv_update<<<dim3((rest + 127) / 128, nrhs, batch), 128, 0, st>>>(A, n, ld, stride, X, nrhs, ldx,
                                                                                 xstride, j0, jb, 0);
            tags_note_launch();
        }
    }
    int last = ((n - 1) / NB) * NB;
    for (int j0 = last; j0 >= 0; j0 -= NB) {
        int jb = min(NB, n - j0);
        k_trsv_diag<<<dim3(1, 1, batch), 256, 0, st>>>(A, n, ld, stride, X, nrhs, ldx, xstride, j0, jb, 1);
        tags_note_launch();
        if (j0 > 0) {
            k_trsv_update<<<dim3((j0 + 127) / 128, nrhs, batch), 128, 0, st>>>(A, n, ld, stride, X, nrhs, ldx,
                                                                               xstride, j0, jb, 1);
            tags_note_launch();
        }
    }
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}
