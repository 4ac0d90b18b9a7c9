// FP64 re-solves of a plan's samples, side by side: those whose refinement in the
// mixed form did not converge, and those whose structured FP64 solve has not
// settled yet (TAGS_INFO_MORE) or needs a pivot search (TAGS_INFO_RESOLVE). Three
// stages, each over all the samples that need it: the structured LDL^T with a pass's
// corrections, up to TAGS_RESOLVE_STEPS of them, and the LU with partial pivoting
// (lu.cu).
// Refinement that still contracts is cheaper than the LU (64 samples at 0.01 .. 1 Hz,
// 100 segments in 1e-4 S/m: 2.7 ms in all, 60 by the LU alone), and the LU's serial
// panels cost a batch little more than one sample: 64 samples at s = 0 66 -> 1.3 ms (N =
// 46) and 433 -> 11.6 ms (N = 285) against one LU after the other.
#include <algorithm>
#include <vector>

#include "tags_common.cuh"
#include "tags_internal.h"
#include "../../include/tags_gpu.h"
#include "plan.h"

int tags_plan_coef(tags_plan_s* p, const double2* d_s, const double2* d_kappa, double mur, int nb, cudaStream_t st);

namespace {

// Inputs of the samples idx[0..) side by side: their coefficients and right-hand
// sides in the original order (nc > 0: rhs is in the static order, nc currents
// first, and turned back).
__global__ void k_resolve_gather(const int* __restrict__ idx, const SampleCoef* __restrict__ coef,
                                 const double2* __restrict__ rhs, int N, int nc, SampleCoef* __restrict__ coef_out,
                                 double2* __restrict__ rhs_out) {
    const int b = blockIdx.y, q = idx[b], r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) coef_out[b] = coef[q];
    if (r >= N) return;
    const int o = nc == 0 ? r : r < nc ? N - nc + r : r - nc;
    rhs_out[(size_t)b * N + o] = rhs[(size_t)q * N + r];
}

// The same from a sweep's arrays: s and kappa, and the right-hand sides [ie; 0; 0]
// or a unit current at inj.
__global__ void k_resolve_inputs(const int* __restrict__ idx, const double2* __restrict__ s,
                                 const double2* __restrict__ kappa, const double2* __restrict__ ie, int inj, int n, int N,
                                 double2* __restrict__ s_out, double2* __restrict__ kappa_out,
                                 double2* __restrict__ rhs_out) {
    const int b = blockIdx.y, q = idx[b], r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) {
        s_out[b] = s[q];
        kappa_out[b] = kappa[q];
    }
    if (r >= N) return;
    double2 v = make_double2(0.0, 0.0);
    if (r < n) {
        if (ie) v = ie[(size_t)q * n + r];
        else if (r == inj) v = make_double2(1.0, 0.0);
    }
    rhs_out[(size_t)b * N + r] = v;
}

__global__ void k_resolve_scatter(const int* __restrict__ idx, const double2* __restrict__ x,
                                  const int* __restrict__ info, int N, double2* __restrict__ x_out,
                                  int* __restrict__ info_out) {
    const int b = blockIdx.y, q = idx[b], r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) info_out[q] = info[b];
    if (r < N) x_out[(size_t)q * N + r] = x[(size_t)b * N + r];
}

// The re-solves' buffers for `cap` samples at a time, in p->d_fb; a plain plan's
// matrices, LDL^T workspace and series tables serve here too (the pass is over).
struct View {
    double2* W;
    void* ldl;
    char* series;
    SampleCoef* coef;
    double2 *sk, *rhs;           // s and kappa (2 cap), right-hand sides and solutions (cap x N)
    int *info, *idx, *ipiv;      // cap, cap, cap x N
    int cap, ldl_batch;
};

size_t view_of(const tags_plan_s* p, int cap, View* v) {
    const size_t N = p->N;
    const bool plain = p->precision == TAGS_PLAIN_FP64;
    char* b = reinterpret_cast<char*>(p->d_fb);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char* r = b ? b + o : nullptr;
        o += (bytes + 255) / 256 * 256;
        return r;
    };
    View w{};
    w.W = plain ? p->d_W : reinterpret_cast<double2*>(take(sizeof(double2) * N * N * cap));
    w.ldl = plain ? p->d_ldl64 : take(tags_ldl64_workspace((int)N, cap));
    w.series = plain ? nullptr : take(tags_series_workspace(p->series, cap));
    w.coef = reinterpret_cast<SampleCoef*>(take(sizeof(SampleCoef) * cap));
    w.sk = reinterpret_cast<double2*>(take(sizeof(double2) * 2 * cap));
    w.rhs = reinterpret_cast<double2*>(take(sizeof(double2) * N * cap));
    w.info = reinterpret_cast<int*>(take(sizeof(int) * cap));
    w.idx = reinterpret_cast<int*>(take(sizeof(int) * cap));
    w.ipiv = reinterpret_cast<int*>(take(sizeof(int) * N * cap));
    w.cap = cap;
    w.ldl_batch = plain ? p->batch : cap;
    if (v) *v = w;
    return o;
}

// Room for up to `want` samples at a time: at most 64 (a plain plan: its batch),
// `most` bytes and an eighth of the free memory, at least one. Kept with the plan,
// grown when more is asked; the buffer that is there goes only when the larger one
// has been had.
int reserve(tags_plan_s* p, int want, size_t most) {
    const bool plain = p->precision == TAGS_PLAIN_FP64;
    want = std::min(want, plain ? p->batch : 64);
    if (p->fb_cap >= want || (p->fb_cap > 0 && p->fb_full)) return 0;
    if (!plain && p->series.nbk == 0)
        p->series = tags_series_geometry(p->h_elec.data(), p->m, p->h_img.data(), p->h_img.empty() ? 0 : p->m);
    size_t freeb = 0;
    TAGS_CUDA_OK(tags_free_memory(&freeb));
    const size_t one = view_of(p, 1, nullptr);
    int cap = (int)std::max<size_t>(1, std::min<size_t>((size_t)want, std::min(most, freeb / 8) / one));
    void* buf = nullptr;
    for (; cap > p->fb_cap; cap /= 2) {
        if (cudaMalloc(&buf, view_of(p, cap, nullptr)) == cudaSuccess) break;
        cudaGetLastError();
        buf = nullptr;
    }
    if (!buf) {
        p->fb_full = 1;
        return p->fb_cap > 0 ? 0 : tags_fail(TAGS_E_NOMEM, "device allocation failed (FP64 fallback)");
    }
    if (p->d_fb) {
        TAGS_CUDA_OK(cudaStreamSynchronize(p->stream));
        TAGS_CUDA_OK(cudaFree(p->d_fb));
    }
    p->d_fb = buf;
    p->fb_cap = cap;
    p->fb_full = cap < want;
    if (!plain && p->series.nbk) {
        View v;
        view_of(p, cap, &v);
        p->d_series = v.series;
        p->series_ns = cap;
    }
    return 0;
}

// Calls f(first, count) for the samples of idx in runs that fit, their numbers on
// the device in v.idx.
template <class F>
int for_runs(const View& v, const std::vector<int>& idx, int most, cudaStream_t st, F f) {
    const size_t step = (size_t)std::min(v.cap, most);
    for (size_t k = 0; k < idx.size(); k += step) {
        const int nf = (int)std::min(step, idx.size() - k);
        TAGS_CUDA_OK(cudaMemcpyAsync(v.idx, idx.data() + k, sizeof(int) * nf, cudaMemcpyHostToDevice, st));
        if (int e = f(nf)) return e;
    }
    return 0;
}

dim3 rows_grid(const tags_plan_s* p, int nf) { return dim3((unsigned)((p->N + 255) / 256), (unsigned)nf); }

int gather_pass(tags_plan_s* p, const View& v, const ResolveInputs& in, int nf, cudaStream_t st) {
    k_resolve_gather<<<rows_grid(p, nf), 256, 0, st>>>(v.idx, in.coef, in.rhs, p->N, in.currents_first, v.coef, v.rhs);
    tags_note_launch();
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

// The sweep's coefficients pass through the plan's, nf <= batch of them.
int gather_sweep(tags_plan_s* p, const View& v, const ResolveSweep& in, int nf, cudaStream_t st) {
    k_resolve_inputs<<<rows_grid(p, nf), 256, 0, st>>>(v.idx, in.s, in.kappa, in.ie, in.inj, p->n, p->N, v.sk, v.sk + v.cap,
                                                      v.rhs);
    tags_note_launch();
    if (int e = tags_plan_coef(p, v.sk, v.sk + v.cap, in.mur, nf, st)) return e;
    TAGS_CUDA_OK(cudaMemcpyAsync(v.coef, p->d_coef, sizeof(SampleCoef) * nf, cudaMemcpyDeviceToDevice, st));
    return 0;
}

int scatter(tags_plan_s* p, const View& v, int nf, double2* x, int* info, cudaStream_t st) {
    k_resolve_scatter<<<rows_grid(p, nf), 256, 0, st>>>(v.idx, v.rhs, v.info, p->N, x, info);
    tags_note_launch();
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

// v.rhs <- the solutions of the samples in v.coef and v.rhs [0, nf): the
// structured LDL^T (ldl64.cu), or the LU with partial pivoting.
int solve_ldl(tags_plan_s* p, const View& v, int nf, int steps, cudaStream_t st) {
    int err = tags_plan_fill_fp64(p, v.coef, nf, tags_ldl64_fill_out(v.W, p->m, p->n), st);
    if (!err)
        err = tags_ldl64_plan_solve(v.W, p->inc, p->m, p->n, nf, v.ldl_batch, v.ldl, v.rhs, v.rhs, v.info, steps, st);
    return err;
}

int solve_lu(tags_plan_s* p, const View& v, int nf, cudaStream_t st) {
    TagsRange range("tags FP64 re-solve");
    const long long N = p->N, NN = N * N;
    TAGS_CUDA_OK(cudaMemsetAsync(v.W, 0, sizeof(double2) * NN * nf, st));
    int err = tags_wg_incidence(v.W, N, NN, nf, p->d_cond, p->n, p->m, st);
    if (err) return err;
    FillOut out{};
    out.zl = v.W;
    out.zt = v.W;
    out.ld = N;
    out.batch_stride = NN;
    out.row0_l = out.col0_l = p->n;
    out.row0_t = out.col0_t = p->n + p->m;
    out.sign = -1.0;
    out.mirror = 1;
    err = tags_plan_fill_fp64(p, v.coef, nf, out, st);
    if (!err) err = tags_lu_z(v.W, (int)N, N, NN, nf, v.ipiv, v.info, st);
    return err ? err : tags_lu_solve_z(v.W, (int)N, N, NN, nf, v.ipiv, v.rhs, 1, N, N, st);
}

// The structured LDL^T of samples idx, which `gather` puts side by side. Where one
// run held them all, its state stays for `refine`.
template <class G>
int run_ldl(tags_plan_s* p, const View& v, const std::vector<int>& idx, int most, int steps, double2* x, int* info,
            cudaStream_t st, G gather) {
    p->fb_run = (int)idx.size() <= std::min(v.cap, most) ? (int)idx.size() : 0;
    p->fb_step = steps;
    return for_runs(v, idx, most, st, [&](int nf) {
        int e = gather(nf);
        if (!e) e = solve_ldl(p, v, nf, steps, st);
        return e ? e : scatter(p, v, nf, x, info, st);
    });
}

// The next corrections of samples `more` among the last run_ldl's: on its state, or
// all of them from the start where that is gone.
template <class G>
int refine(tags_plan_s* p, const View& v, const std::vector<int>& more, int most, double2* x, int* info, cudaStream_t st,
           G gather) {
    const int nf = p->fb_run;
    if (nf == 0) return run_ldl(p, v, more, most, TAGS_RESOLVE_STEPS, x, info, st, gather);
    const int e = tags_ldl64_plan_more(v.W, p->inc, p->m, p->n, nf, v.ldl_batch, v.ldl, &p->fb_step, v.rhs, v.info, st);
    return e ? e : scatter(p, v, nf, x, info, st);
}

template <class G>
int run_lu(tags_plan_s* p, const View& v, const std::vector<int>& idx, int most, double2* x, int* info, cudaStream_t st,
           G gather) {
    p->fb_run = 0;
    return for_runs(v, idx, most, st, [&](int nf) {
        int e = gather(nf);
        if (!e) e = solve_lu(p, v, nf, st);
        return e ? e : scatter(p, v, nf, x, info, st);
    });
}

int open_view(tags_plan_s* p, size_t want, size_t most, View* v) {
    if (int e = reserve(p, (int)want, most)) return e;
    view_of(p, p->fb_cap, v);
    return 0;
}

}  // namespace

int tags_resolve_pass(tags_plan_s* p, const std::vector<int>& first, const std::vector<int>& lu, const ResolveInputs& in,
                      double2* x, int* info, cudaStream_t st) {
    if (first.empty() && lu.empty()) return 0;
    TagsRange range("tags FP64 re-solve");
    View v;
    if (int e = open_view(p, std::max(first.size(), lu.size()), (size_t)512 << 20, &v)) return e;
    auto gather = [&](int nf) { return gather_pass(p, v, in, nf, st); };
    std::vector<int> todo = first, pivoted = lu;
    for (bool again = false; !todo.empty(); again = true) {
        const int e = again ? refine(p, v, todo, v.cap, x, info, st, gather)
                            : run_ldl(p, v, todo, v.cap, TAGS_FIRST_STEPS, x, info, st, gather);
        if (e) return e;
        std::vector<int> got(p->batch), more;
        TAGS_CUDA_OK(cudaMemcpyAsync(got.data(), info, sizeof(int) * p->batch, cudaMemcpyDeviceToHost, st));
        TAGS_CUDA_OK(cudaStreamSynchronize(st));
        for (int q : todo) {
            if (got[q] == TAGS_INFO_MORE) more.push_back(q);
            if (got[q] == TAGS_INFO_RESOLVE) pivoted.push_back(q);
        }
        todo = more;
    }
    return pivoted.empty() ? 0 : run_lu(p, v, pivoted, v.cap, x, info, st, gather);
}

int tags_resolve_sweep_ldl(tags_plan_s* p, const std::vector<int>& first, const ResolveSweep& in, int steps, double2* x,
                           int* info, size_t most, cudaStream_t st) {
    if (first.empty()) return 0;
    View v;
    if (int e = open_view(p, first.size(), most, &v)) return e;
    return run_ldl(p, v, first, p->batch, steps, x, info, st, [&](int nf) { return gather_sweep(p, v, in, nf, st); });
}

int tags_resolve_sweep_more(tags_plan_s* p, const std::vector<int>& more, const ResolveSweep& in, double2* x, int* info,
                            size_t most, cudaStream_t st) {
    if (more.empty()) return 0;
    View v;
    if (int e = open_view(p, more.size(), most, &v)) return e;
    return refine(p, v, more, p->batch, x, info, st, [&](int nf) { return gather_sweep(p, v, in, nf, st); });
}

int tags_resolve_sweep_lu(tags_plan_s* p, const std::vector<int>& idx, const ResolveSweep& in, double2* x, int* info,
                          size_t most, cudaStream_t st) {
    if (idx.empty()) return 0;
    View v;
    if (int e = open_view(p, idx.size(), most, &v)) return e;
    return run_lu(p, v, idx, p->batch, x, info, st, [&](int nf) { return gather_sweep(p, v, in, nf, st); });
}
