// Post-processing of solved currents on GB300: the scalar potential, the
// magnetic vector potential, the electric field and the path voltage of the
// reference (src/electrode.c:434-668), and the closed-form mHEM ground
// potential that its examples evaluate (examples/visacro57emc01.c:406-430),
// batched over points x Laplace samples x injections.
//
// Electrode integrals. The reference integrates e^{-gamma r}/r (and its
// gradient) along every electrode with an adaptive 1-D cubature
// (src/electrode.c:199-218 and :495-520). Here each (point, electrode) pair
// gets a fixed rule from its geometry: the substitution
//     u = u0 + (d'/L) sinh v,   d' = max(d, 1e-6 L)
// about the foot u0 of the point on the electrode's line (d the distance to
// that line, L the electrode length) turns du / r into (d'/L) cosh v dv / r,
// which is smooth (and exactly dv / L when d' = d), so the near-singularity
// of points close to an electrode disappears. Gauss-Legendre panels of unit
// width in v, split further wherever |gamma| grows r by more than 1.5 across a
// panel, integrate what is left with 8 nodes per panel; against 1e-14 adaptive
// integrals over random geometries, frequencies and distances (1e-4 L to 5 L)
// the rule stays within 1e-12 relative. Samples with |gamma| up to 2 / (L + 1/8 m) or
// so share the rule's moments and cost a series each (k_fields_series); the
// rule with an exponential per node (k_fields) serves the ones beyond.
//
// Path voltage. The reference integrates E . (p2 - p1) / |p2 - p1| over t in
// [0, 1] with a cubature whose integrand is itself a field cubature per
// electrode (src/electrode.c:599-668). The conservative part of E is exactly
// -grad u, so that part equals (u(p1) - u(p2)) / |p2 - p1|; the -s A part is a
// double integral of e^{-gamma r}/r between the path and each electrode, the
// pair integral of the impedance fill (fill.cu). Both are evaluated so here,
// without nesting; the result is the reference's (the path voltage divided by
// the path length).
//
// Layouts: currents il/it [sample][injection][electrode]; pot and gpd
// [sample][point][injection]; vecpot and efield [sample][point][injection][3];
// path voltages [sample][path][injection].
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <mutex>
#include <vector>

#include "tags_common.cuh"
#include "tags_internal.h"
#include "../../include/tags_gpu.h"
#include "plan.h"

using zd = std::complex<double>;

namespace {

constexpr int FQ = 8;             // Gauss-Legendre nodes per panel
constexpr double FC = 1.5;        // largest |gamma| * (r growth) across a panel
constexpr int NB = 256;           // node buffer per warp (shared memory)
constexpr int FW = 4;             // warps per CTA
constexpr int RMAX = 4;           // injections per pass of a warp
constexpr int KMAX = 64;          // subpanels per unit panel (cap)

__constant__ double c_fx[FQ];     // nodes on [0, 1]
__constant__ double c_fw[FQ];     // weights on [0, 1]

struct NodeRec {
    double r, spar, jw;
};

struct WarpSmem {
    NodeRec node[NB];
    double lo[32], hi[32];
    int k[32], pre[32];
};

enum { WANT_POT = 1, WANT_VEC = 2, WANT_EF = 4 };

struct FieldArgs {
    const double* pts;      // P x 3
    const Seg* elec;        // m
    const double2* cur_t;   // [m][R][S]
    const double2* cur_l;   // [m][R][S]
    const double2* gamma;   // S
    const double2* kappa;   // S
    double mur;
    int P, m, R, S, G;      // G samples per warp (power of two <= 32)
    int want;
    int skip_pot;           // skip |it| < DBL_EPSILON in the potential (field convention)
    double2* pot;           // [S][P][R]
    double2* vec;           // [S][P][R][3]
    double2* ef;            // [S][P][R][3]
    int* status;
    unsigned long long* evals;  // node x sample evaluations (work counter)
    int nchunk;             // electrode chunks (warps per point and sample group)
    double2* part;          // [nchunk][S][P][R][7] raw sums: pot, vec xyz, ef xyz
    const int* nt;          // S: terms of the moment series (0: the rule per sample serves this one)
    int schunk;             // the series' partial sums: [schunk][S][P][R][7]
    double2* spart;
};

TAGS_D double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

TAGS_D double2 shfl_xor2(double2 v, int o) {
    return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// One warp per (electrode chunk, point, group of G samples); lanes are
// (sample si = lane % G, node slice sub = lane / G). The rule's nodes of each
// electrode are built once per warp into shared memory and reused by all
// samples of the group. The electrode chunks spread one point's work over
// several warps so the grid fills the GPU evenly; k_fields_reduce adds them.
__global__ void __launch_bounds__(FW * 32) k_fields(FieldArgs a, int r0) {
    __shared__ WarpSmem sm_all[FW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpSmem& sm = sm_all[warp];
    const int G = a.G, NS = 32 / G;
    const int ngroups = (a.S + G - 1) / G;
    const long long per_chunk = (long long)a.P * ngroups;
    const long long item_all = (long long)blockIdx.x * FW + warp;
    if (item_all >= per_chunk * a.nchunk) return;     // whole warp leaves together
    const int chunk = (int)(item_all / per_chunk);
    const long long item = item_all - (long long)chunk * per_chunk;
    const int p = (int)(item / ngroups), grp = (int)(item % ngroups);
    const int e_begin = (int)((long long)chunk * a.m / a.nchunk);
    const int e_end = (int)((long long)(chunk + 1) * a.m / a.nchunk);
    const int si = lane % G, sub = lane / G;
    const int smp = grp * G + si;
    const bool valid = smp < a.S && a.nt[smp] == 0;   // the others take the moment series
    if (!__any_sync(0xffffffffu, valid)) return;
    const int nr = min(RMAX, a.R - r0);
    const double2 gam = valid ? a.gamma[smp] : cz(0.0, 0.0);
    const double gmax = warp_max(valid ? sqrt(cabs2(gam)) : 0.0);
    const double P0 = a.pts[3 * p], P1 = a.pts[3 * p + 1], P2 = a.pts[3 * p + 2];
    const bool wv = (a.want & (WANT_VEC | WANT_EF)) != 0;

    double2 pot[RMAX], vec[RMAX][3], ef[RMAX][3];
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        pot[r] = cz(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < 3; ++c) { vec[r][c] = cz(0.0, 0.0); ef[r][c] = cz(0.0, 0.0); }
    }

    for (int e = e_begin; e < e_end; ++e) {
        const Seg& S = a.elec[e];
        const double D[3] = {S.b[0] - S.a[0], S.b[1] - S.a[1], S.b[2] - S.a[2]};
        const double L2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2];
        const double Lg = sqrt(L2);
        const double w0[3] = {P0 - S.a[0], P1 - S.a[1], P2 - S.a[2]};
        const double u0 = (w0[0] * D[0] + w0[1] * D[1] + w0[2] * D[2]) / L2;
        const double wp[3] = {w0[0] - u0 * D[0], w0[1] - u0 * D[1], w0[2] - u0 * D[2]};
        const double d = sqrt(wp[0] * wp[0] + wp[1] * wp[1] + wp[2] * wp[2]);
        const double dp = fmax(d, 1e-6 * Lg);
        // distance from the point to the segment itself
        const double uc = fmin(fmax(u0, 0.0), 1.0);
        const double du = (u0 - uc) * Lg;
        const double va = asinh(-u0 * Lg / dp), vb = asinh((1.0 - u0) * Lg / dp);
        // a point on the electrode (or a zero-length or non-finite record):
        // the integral diverges, the reference's result is undefined
        const bool degenerate = !(sqrt(d * d + du * du) > 1e-12 * Lg) || !isfinite(va) || !isfinite(vb);

        // unit panels: [va, 0] and [0, vb] when the foot is inside, else [va, vb]
        const bool split = va < 0.0 && vb > 0.0;
        const double la = split ? -va : vb - va, lb = split ? vb : 0.0;
        const int na = degenerate ? 0 : max(1, (int)ceil(la - 1e-12));
        const int nb2 = (degenerate || !split) ? 0 : max(1, (int)ceil(lb - 1e-12));
        const int nu = na + nb2;                       // <= 30 with d' >= 1e-6 L
        int kj = 0;
        if (lane < nu) {
            double lo, hi;
            if (lane < na) {
                const double h = la / na, base = va;
                lo = base + lane * h;
                hi = (lane == na - 1) ? (split ? 0.0 : vb) : base + (lane + 1) * h;
            } else {
                const int j = lane - na;
                const double h = lb / nb2;
                lo = j * h;
                hi = (j == nb2 - 1) ? vb : (j + 1) * h;
            }
            const double slo = dp * sinh(lo), shi = dp * sinh(hi);
            const double rlo = sqrt(d * d + slo * slo), rhi = sqrt(d * d + shi * shi);
            kj = min(KMAX, max(1, (int)ceil(gmax * fabs(rhi - rlo) / FC)));
            sm.lo[lane] = lo;
            sm.hi[lane] = hi;
            sm.k[lane] = kj;
        }
        // exclusive prefix of the subpanel counts
        int incl = kj;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane < nu) sm.pre[lane] = incl - kj;
        const int ksum = __shfl_sync(0xffffffffu, incl, 31);
        const int nodes = ksum * FQ;
        if (lane == 0 && a.evals) atomicAdd(a.evals, (unsigned long long)nodes * (unsigned long long)min(G, a.S - grp * G));
        __syncwarp();

        double2 J1 = cz(0.0, 0.0), Ap = cz(0.0, 0.0), Bp = cz(0.0, 0.0);
        for (int base = 0; base < nodes; base += NB) {
            const int cnt = min(NB, nodes - base);
            for (int t = lane; t < cnt; t += 32) {
                const int nid = base + t, spn = nid / FQ, q = nid - spn * FQ;
                int lo_i = 0, hi_i = nu - 1;                 // panel j with pre[j] <= spn
                while (lo_i < hi_i) {
                    int mid = (lo_i + hi_i + 1) >> 1;
                    if (sm.pre[mid] <= spn) lo_i = mid; else hi_i = mid - 1;
                }
                const int j = lo_i, kk = sm.k[j], loc = spn - sm.pre[j];
                const double h = (sm.hi[j] - sm.lo[j]) / kk;
                const double v = sm.lo[j] + (loc + c_fx[q]) * h;
                const double sv = sinh(v), cv = cosh(v);
                NodeRec nr_;
                nr_.spar = dp * sv;
                nr_.r = sqrt(d * d + nr_.spar * nr_.spar);
                nr_.jw = c_fw[q] * h * (dp / Lg) * cv;
                sm.node[t] = nr_;
            }
            __syncwarp();
            if (valid) {
                for (int t = sub; t < cnt; t += NS) {
                    const NodeRec nd = sm.node[t];
                    const double2 ex = cexp_d(cz(-gam.x * nd.r, -gam.y * nd.r));
                    const double ir = 1.0 / nd.r;
                    J1.x = fma(nd.jw * ir, ex.x, J1.x);
                    J1.y = fma(nd.jw * ir, ex.y, J1.y);
                    if (wv) {
                        // (1 + gamma r) e^{-gamma r} / r^3
                        const double2 f = cmul(cz(1.0 + gam.x * nd.r, gam.y * nd.r), ex);
                        const double sc = nd.jw * ir * ir * ir;
                        Ap.x = fma(sc, f.x, Ap.x);
                        Ap.y = fma(sc, f.y, Ap.y);
                        Bp.x = fma(sc * nd.spar, f.x, Bp.x);
                        Bp.y = fma(sc * nd.spar, f.y, Bp.y);
                    }
                }
            }
            __syncwarp();
        }
        // reduce over the node slices (lane bits >= log2 G)
        for (int o = G; o < 32; o <<= 1) {
            J1 = cadd(J1, shfl_xor2(J1, o));
            if (wv) {
                Ap = cadd(Ap, shfl_xor2(Ap, o));
                Bp = cadd(Bp, shfl_xor2(Bp, o));
            }
        }
        if (degenerate) {
            if (lane == 0) raise_status(a.status, TAGS_ST_DEGENERATE_PAIR);
            J1 = Ap = Bp = cz(nan(""), nan(""));
        }
        if (valid && sub == 0) {
            const double Dh[3] = {D[0] / Lg, D[1] / Lg, D[2] / Lg};
#pragma unroll
            for (int r = 0; r < RMAX; ++r) {
                if (r >= nr) break;
                const long long ci = ((long long)e * a.R + r0 + r) * a.S + smp;
                if (a.want & (WANT_POT | WANT_EF)) {
                    const double2 ct = a.cur_t[ci];
                    const bool big = sqrt(cabs2(ct)) >= TAGS_DBL_EPSILON;
                    if (!a.skip_pot || big) pot[r] = cfma(ct, J1, pot[r]);
                    if ((a.want & WANT_EF) && big) {
                        const double2 ca = cmul(ct, Ap), cb = cmul(ct, Bp);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            ef[r][c].x += ca.x * wp[c] - cb.x * Dh[c];
                            ef[r][c].y += ca.y * wp[c] - cb.y * Dh[c];
                        }
                    }
                }
                if (a.want & WANT_VEC) {
                    const double2 cl = a.cur_l[ci];
                    if (sqrt(cabs2(cl)) >= TAGS_DBL_EPSILON) {
                        const double2 cj = cmul(cl, J1);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            vec[r][c].x = fma(cj.x, D[c], vec[r][c].x);
                            vec[r][c].y = fma(cj.y, D[c], vec[r][c].y);
                        }
                    }
                }
            }
        }
        __syncwarp();
    }

    if (!valid || sub != 0) return;
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        if (r >= nr) break;
        double2* o = a.part + ((((long long)chunk * a.S + smp) * a.P + p) * a.R + r0 + r) * 7;
        o[0] = pot[r];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            o[1 + c] = vec[r][c];
            o[4 + c] = ef[r][c];
        }
    }
}

// ---- moment series over the samples ------------------------------------------------
//
// With r = R + d about R = b h, the multiple of h nearest the distance to the
// electrode's midpoint, the three integrals of a (point, electrode) pair are
//   e^{-gamma R} sum_n p_n M_n,   p_n = (-gamma)^n / n!,
// for 1/r:                    N_n = \int d^n / r dt,
// for (1 + gamma r) / r^3:    A_n = \int (d^n - n d^(n-1) r) / r^3 dt
// (gamma r e^{-gamma d} contributes -n p_n d^(n-1) r), and B_n with the axial
// offset as a further factor. The moments are geometry only: one rule per pair
// serves all samples, a sample then costs 6 FP64 multiply-adds per term instead
// of a complex exponential and ~30 operations per node. |d| <= Lmax / 2 + h / 2 =
// dmax; terms up to x^n / n! <= 1e-17 at x = |gamma| dmax, at most FS_NT (x <= 2);
// samples beyond keep the rule of k_fields.
constexpr int FS_NT = 24;
constexpr double FS_XMAX = 2.0;
constexpr int FS_THREADS = 128;
// |c| >= DBL_EPSILON = 2^-52 (the square's rounded root), without FP64 work for
// the usual currents: a part of 2^-52 or more is seen in its exponent.
TAGS_D bool cur_big(double2 c) {
    const int hx = __double2hiint(c.x) & 0x7fffffff, hy = __double2hiint(c.y) & 0x7fffffff;
    const int lim = (1023 - 52) << 20;
    if (hx >= lim && hx < 0x7ff00000) return true;
    if (hy >= lim && hy < 0x7ff00000 && hx < 0x7ff00000) return true;
    return cabs2(c) >= 0x1.fffffffffffffp-105;      // the squares whose root rounds to 2^-52 or more
}
constexpr int FS_ORDERS[6] = {6, 7, 8, 9, 10, 12};
constexpr int FS_GL = 6 + 7 + 8 + 9 + 10 + 12, FS_8 = 6 + 7, FS_10 = 6 + 7 + 8 + 9;

// The rule's least order, as an index of FS_ORDERS, at y = |gamma| times half the range
// of r over the electrode, y2 / s2 = y^2: the distance leaves 1/r and 1/r^3 with 6 nodes
// from 16 and 7 from 8 lengths on below 1e-15, but the moments also carry e^{-gamma r},
// whose error is 3e-9 (y / 2)^12 with 6 nodes, 2e-11 (y / 2)^14 with 7 and 1e-13 (y / 2)^16
// with 8. Each stays up to where that passes 1e-15 to 4e-15 (6 nodes throughout: 6e-10 at the
// series' reach on the electrode's axis).
TAGS_D int fs_least_order(double y2, double s2) {
    return y2 <= 0.24 * s2 ? 0 : y2 <= 0.7 * s2 ? 1 : y2 <= 1.8 * s2 ? 2 : 3;
}
__constant__ double c_fsx[FS_GL], c_fsw[FS_GL];   // nodes and weights on [0, 1], order by order

struct SerArgs {
    FieldArgs f;
    const double2* pw;      // [FS_NT][S]
    const double2* tab;     // [bucket][S]: e^{-gamma b h} (null: formed per pair)
    double h;
    int nbk, ngc, echunk;   // buckets; sample groups per CTA (1, 2, 4); electrodes per CTA
    double ga2;             // a quarter of the largest |gamma|^2 among the series' samples
    int near;               // nodes per panel of the near points' rule: 8 or 10
};

// The samples' constants: a row of CTAs per bucket of the table (nbk of them, none
// where the pairs form theirs), one more for the powers.
__global__ void k_fser_tables(const double2* __restrict__ gamma, const int* __restrict__ nt, int S, int nbk, double h,
                              double2* __restrict__ pw, double2* __restrict__ tab) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    if (s >= S) return;
    const double2 g = nt[s] > 0 ? gamma[s] : cz(0.0, 0.0);
    if (b < nbk) {
        tab[(long long)b * S + s] = cexp_d(cz(-g.x * (b * h), -g.y * (b * h)));
        return;
    }
    double2 p = cz(1.0, 0.0);
    for (int n = 0; n < FS_NT; ++n) {
        pw[(long long)n * S + s] = n < nt[s] ? p : cz(0.0, 0.0);
        p = cscale(cmul(p, cneg(g)), 1.0 / (double)(n + 1));
    }
}

// What the samples need of a pair besides its moments.
struct SerPair {
    double D[3], wp[3], iL;     // electrode vector, offset of the point from its line, 1 / length
    int b, bad;
};

// Moments of one (point, electrode) pair by L lanes (g: this one), all of the
// warp's groups together, `on` or not: Gauss-Legendre in t where the point is at
// least two lengths away (6 to 12 nodes by the distance and |gamma|), else the sinh
// rule above, up to ~400 nodes, which one lane would take in a row: panels of 0.75 with
// 8 nodes, or of one with 10 where e^{-gamma r} asks for them (x > 1.1). 3000 random
// points within two lengths, 25 nodes each on average either way, stay within 8e-14 (6e-16
// in the median) and 4e-15; 8 nodes at x = 2: 1e-12. With 10 throughout, pairs of few
// lanes take a second round for one panel: path voltages of 40 paths 0.90 -> 0.92 ms.
template <int NT>
TAGS_D void fser_moments(const Seg& S, double P0, double P1, double P2, const SerArgs& sa, const double* gx,
                         const double* gw, bool on, int g, int L, SerPair& out, double* mom) {
    SerPair q;
    const double D[3] = {S.b[0] - S.a[0], S.b[1] - S.a[1], S.b[2] - S.a[2]};
    const double L2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2], Lg = sqrt(L2);
    const double w0[3] = {P0 - S.a[0], P1 - S.a[1], P2 - S.a[2]};
    const double u0 = (w0[0] * D[0] + w0[1] * D[1] + w0[2] * D[2]) / L2;
    double d2 = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        q.D[c] = D[c];
        q.wp[c] = w0[c] - u0 * D[c];
        d2 += q.wp[c] * q.wp[c];
    }
    q.iL = 1.0 / Lg;
    const double uc = fmin(fmax(u0, 0.0), 1.0), du = (u0 - uc) * Lg;
    const double dist = sqrt(d2 + du * du);
    const double dm = (u0 - 0.5) * Lg, rc = sqrt(d2 + dm * dm);
    q.b = min(sa.nbk - 1, max(0, (int)rint(rc / sa.h)));
    const double R = q.b * sa.h;
    double aN[NT], aA[NT], aB[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) aN[n] = aA[n] = aB[n] = 0.0;
    auto node = [&](double s, double r2, double w) {       // axial offset from the foot, r^2, weight
        const double ir = rsqrt(r2), r = r2 * ir, d = r - R, ir2 = ir * ir, ir3 = ir2 * ir;
        double pn = w, pm = 0.0, c = 0.0;                  // w d^n, w d^(n-1), n / r^2
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const double t = fma(-c, pm, pn * ir3);
            aN[n] = fma(pn, ir, aN[n]);
            aA[n] += t;
            aB[n] = fma(t, s, aB[n]);
            pm = pn;
            pn *= d;
            c += ir2;
        }
    };
    q.bad = !(dist > 1e-12 * Lg) || !isfinite(rc);
    if (!q.bad && dist >= 2.0 * Lg) {
        const double ratio = dist * q.iL;
        // r grows by L |dm| / rc over the electrode
        const int o = max(fs_least_order(sa.ga2 * L2 * (dm * dm), fma(dm, dm, d2)),
                          ratio >= 16.0 ? 0 : ratio >= 8.0 ? 1 : ratio >= 4.0 ? 3 : 5);
        const int nq = o == 5 ? 12 : 6 + o, off = o == 5 ? 40 : 6 * o + o * (o - 1) / 2;
        for (int i = g; i < nq; i += L) {
            const double s = (gx[off + i] - u0) * Lg;
            node(s, fma(s, s, d2), gw[off + i]);
        }
    } else if (!q.bad) {
        const double d = sqrt(d2), dp = fmax(d, 1e-6 * Lg);
        const double va = asinh(-u0 * Lg / dp), vb = asinh((1.0 - u0) * Lg / dp);
        const int nn = sa.near, off = nn == 8 ? FS_8 : FS_10, inv = nn == 8 ? 8193 : 6554;
        const double wide = nn == 8 ? 1.0 / 0.75 : 1.0;
        // panels on either side of the foot, or one range
        const bool split = va < 0.0 && vb > 0.0;
        for (int side = 0; side < (split ? 2 : 1); ++side) {
            const double lo = split && side == 1 ? 0.0 : va, hi = split && side == 0 ? 0.0 : vb;
            const int np = max(1, (int)ceil(fmin((hi - lo) * wide, 64.0)));
            const double ph = (hi - lo) / np;
            for (int t = g; t < nn * np; t += L) {
                const int p = (t * inv) >> 16, i = off + t - nn * p;        // p = t / nn up to 64 panels
                const double v = lo + (p + gx[i]) * ph, s = dp * sinh(v);
                node(s, fma(s, s, d2), gw[i] * ph * (dp * q.iL) * cosh(v));
            }
        }
    }
    for (int o = L >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            aN[n] += __shfl_xor_sync(0xffffffffu, aN[n], o);
            aA[n] += __shfl_xor_sync(0xffffffffu, aA[n], o);
            aB[n] += __shfl_xor_sync(0xffffffffu, aB[n], o);
        }
    if (!on || g != 0) return;
    out = q;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        mom[n] = aN[n];
        mom[NT + n] = aA[n];
        mom[2 * NT + n] = aB[n];
    }
}

// A CTA per (point, electrode chunk, four sample groups at most): FS_E electrodes
// at a time, a thread (or, with fewer electrodes, up to 32 lanes) forms a pair's
// moments, then the warps (sample group x
// share of the electrodes; lanes: G samples x 32 / G electrodes) sum the series
// and accumulate the currents' terms. FP64-bound: 6 nt + 24 multiply-adds per
// (pair, sample) and 20 per injection. The 1560-segment grid, 251 points, 64
// samples, 4 injections: 58.8 ms by the rule per sample, 13.1 ms so (14.4 with the
// vector potential's three components per pair; error of the field against 64-bit
// quadrature 1.6e-13 -> 2.2e-15). e^{-gamma R} comes from the table, or, where the
// call has fewer pairs than the table has buckets, is formed per pair and sample
// (TAB false): a point 1 km from ten electrodes needs 10 of 4002 buckets.
constexpr int FS_E = 128;                 // pairs per tile, a thread each
template <int NT, bool TAB>
__global__ void __launch_bounds__(FS_THREADS) k_fields_series(SerArgs sa, int r0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* mom = reinterpret_cast<double*>(smem_raw);              // [FS_E][3 NT]
    __shared__ SerPair pr[FS_E];
    __shared__ double gx[FS_GL], gw[FS_GL];
    const FieldArgs& a = sa.f;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p = blockIdx.x;
    if (tid < FS_GL) {
        gx[tid] = c_fsx[tid];
        gw[tid] = c_fsw[tid];
    }
    const int G = a.G, NS = 32 / G, ngroups = (a.S + G - 1) / G;
    const int nshare = (FS_THREADS / 32) / sa.ngc;
    const int grp = blockIdx.z * sa.ngc + warp % sa.ngc, share = warp / sa.ngc;
    const int si = lane % G, sub = lane / G, smp = grp * G + si;
    const bool valid = grp < ngroups && smp < a.S && a.nt[smp] > 0;
    const int nt = __reduce_max_sync(0xffffffffu, valid ? a.nt[smp] : 0);
    const int nr = min(RMAX, a.R - r0);
    const double2 gam = !TAB && valid ? a.gamma[smp] : cz(0.0, 0.0);
    const double P0 = a.pts[3 * p], P1 = a.pts[3 * p + 1], P2 = a.pts[3 * p + 2];
    const bool wv = (a.want & (WANT_VEC | WANT_EF)) != 0;
    const int e_begin = blockIdx.y * sa.echunk, e_end = min(a.m, e_begin + sa.echunk);

    double2 pot[RMAX], vec[RMAX][3], ef[RMAX][3];
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        pot[r] = cz(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < 3; ++c) { vec[r][c] = cz(0.0, 0.0); ef[r][c] = cz(0.0, 0.0); }
    }
    // the vector potential of electrodes in a row of one length and direction D
    // is summed as a multiple of D
    double D[3] = {0.0, 0.0, 0.0};
    double2 along[RMAX];
#pragma unroll
    for (int r = 0; r < RMAX; ++r) along[r] = cz(0.0, 0.0);
    auto flush = [&]() {
#pragma unroll
        for (int r = 0; r < RMAX; ++r) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                vec[r][c].x = fma(along[r].x, D[c], vec[r][c].x);
                vec[r][c].y = fma(along[r].y, D[c], vec[r][c].y);
            }
            along[r] = cz(0.0, 0.0);
        }
    };
    for (int e0 = e_begin; e0 < e_end; e0 += FS_E) {
        const int ne = min(FS_E, e_end - e0);
        __syncthreads();
        int L = 1;                                          // lanes per pair: a short tile shares out its nodes
        while (2 * L * ne <= FS_THREADS && L < 32) L *= 2;
        const int me = min(tid / L, ne - 1);
        const bool on = tid < L * ne;
        fser_moments<NT>(a.elec[e0 + me], P0, P1, P2, sa, gx, gw, on, tid % L, L, pr[me], mom + (size_t)me * 3 * NT);
        if (on && tid % L == 0 && pr[me].bad) raise_status(a.status, TAGS_ST_DEGENERATE_PAIR);
        __syncthreads();
        if (!valid) continue;
        for (int el = share * NS + sub; el < ne; el += nshare * NS) {
            const SerPair& q = pr[el];
            const double* mo = mom + (size_t)el * 3 * NT;
            double2 J1 = cz(0.0, 0.0), Ap = cz(0.0, 0.0), Bp = cz(0.0, 0.0);
            for (int n = 0; n < nt; ++n) {
                const double2 pn = sa.pw[(long long)n * a.S + smp];
                J1.x = fma(pn.x, mo[n], J1.x);
                J1.y = fma(pn.y, mo[n], J1.y);
                if (wv) {
                    Ap.x = fma(pn.x, mo[NT + n], Ap.x);
                    Ap.y = fma(pn.y, mo[NT + n], Ap.y);
                    Bp.x = fma(pn.x, mo[2 * NT + n], Bp.x);
                    Bp.y = fma(pn.y, mo[2 * NT + n], Bp.y);
                }
            }
            double2 ex;
            if (TAB) ex = sa.tab[(long long)q.b * a.S + smp];
            else ex = cexp_d(cz(-gam.x * (q.b * sa.h), -gam.y * (q.b * sa.h)));
            J1 = cmul(J1, ex);
            if (wv) {
                Ap = cmul(Ap, ex);
                Bp = cscale(cmul(Bp, ex), q.iL);
            }
            if (q.bad) J1 = Ap = Bp = cz(nan(""), nan(""));
            if ((a.want & WANT_VEC) && (__double_as_longlong(q.D[0]) != __double_as_longlong(D[0]) ||
                                        __double_as_longlong(q.D[1]) != __double_as_longlong(D[1]) ||
                                        __double_as_longlong(q.D[2]) != __double_as_longlong(D[2]))) {
                flush();
#pragma unroll
                for (int c = 0; c < 3; ++c) D[c] = q.D[c];
            }
            double2 F[3];                                   // the field of a unit current
            if (a.want & WANT_EF)
#pragma unroll
                for (int c = 0; c < 3; ++c) F[c] = cz(Ap.x * q.wp[c] - Bp.x * q.D[c], Ap.y * q.wp[c] - Bp.y * q.D[c]);
#pragma unroll
            for (int r = 0; r < RMAX; ++r) {
                if (r >= nr) break;
                const long long ci = ((long long)(e0 + el) * a.R + r0 + r) * a.S + smp;
                if (a.want & (WANT_POT | WANT_EF)) {
                    const double2 ct = a.cur_t[ci];
                    const bool big = cur_big(ct);
                    if (!a.skip_pot || big) pot[r] = cfma(ct, J1, pot[r]);
                    if ((a.want & WANT_EF) && big) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) ef[r][c] = cfma(ct, F[c], ef[r][c]);
                    }
                }
                if (a.want & WANT_VEC) {
                    const double2 cl = a.cur_l[ci];
                    if (cur_big(cl)) along[r] = cfma(cl, J1, along[r]);
                }
            }
        }
    }
    flush();
    // the electrode shares of a warp's lanes
    for (int o = G; o < 32; o <<= 1) {
#pragma unroll
        for (int r = 0; r < RMAX; ++r) {
            if (r >= nr) break;
            pot[r] = cadd(pot[r], shfl_xor2(pot[r], o));
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                vec[r][c] = cadd(vec[r][c], shfl_xor2(vec[r][c], o));
                ef[r][c] = cadd(ef[r][c], shfl_xor2(ef[r][c], o));
            }
        }
    }
    if (!valid || sub != 0) return;
    const long long chunk = (long long)blockIdx.y * nshare + share;
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        if (r >= nr) break;
        double2* o = a.spart + (((chunk * a.S + smp) * a.P + p) * a.R + r0 + r) * 7;
        o[0] = pot[r];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            o[1 + c] = vec[r][c];
            o[4 + c] = ef[r][c];
        }
    }
}

// Sum of the electrode chunks and the scale factors: 1 / (4 pi kappa) for the
// potential and field, mur mu0 / (4 pi) for the vector potential.
// A thread per output, or a warp (lanes over the chunks) where few outputs have
// many chunks each, which one thread would read one after the other (900
// electrodes, 1 point, 2 samples: 0.75 -> 0.22 ms for the whole call).
template <int W>
__global__ void k_fields_reduce(FieldArgs a) {
    const long long n = (long long)a.S * a.P * a.R;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / W;
    const int lane = (int)(t % W);
    if (i >= n) return;                                     // W = 32: the whole warp
    const int smp = (int)(i / ((long long)a.P * a.R));
    double2 v[7];
#pragma unroll
    for (int c = 0; c < 7; ++c) v[c] = cz(0.0, 0.0);
    const bool ser = a.nt[smp] > 0;
    const double2* part = ser ? a.spart : a.part;
    const int nchunk = ser ? a.schunk : a.nchunk;
    for (int ch = lane; ch < nchunk; ch += W) {
        const double2* q = part + ((long long)ch * n + i) * 7;
#pragma unroll
        for (int c = 0; c < 7; ++c) v[c] = cadd(v[c], q[c]);
    }
    if (W > 1) {
        for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 7; ++c) v[c] = cadd(v[c], shfl_xor2(v[c], o));
        if (lane != 0) return;
    }
    const double2 i4pk = cdiv(cz(1.0, 0.0), cscale(a.kappa[smp], TAGS_FOUR_PI));
    const double u4pi = a.mur * TAGS_MU0 / TAGS_FOUR_PI;
    if (a.pot && (a.want & WANT_POT)) a.pot[i] = cmul(v[0], i4pk);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (a.vec && (a.want & WANT_VEC)) a.vec[3 * i + c] = cscale(v[1 + c], u4pi);
        if (a.ef && (a.want & WANT_EF)) a.ef[3 * i + c] = cmul(v[4 + c], i4pk);
    }
}

// Closed-form mHEM ground potential: warp per (point, sample group); the
// electrode terms log((r1 + r2 + L) / (r1 + r2 - L)) / L and the midpoint
// distance are computed once per warp (a lane per electrode) and shuffled to
// the samples.
__global__ void __launch_bounds__(FW * 32) k_gpd_mhem(const double* __restrict__ pts, const Seg* __restrict__ elec,
                                                      const double2* __restrict__ cur_t,
                                                      const double2* __restrict__ gamma,
                                                      const double2* __restrict__ kappa, int P, int m, int R,
                                                      int S, int G, int r0, double2* __restrict__ gpd) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NS = 32 / G;
    const int ngroups = (S + G - 1) / G;
    const long long item = (long long)blockIdx.x * FW + warp;
    if (item >= (long long)P * ngroups) return;
    const int p = (int)(item / ngroups), grp = (int)(item % ngroups);
    const int si = lane % G, sub = lane / G;
    const int smp = grp * G + si;
    const bool valid = smp < S;
    const int nr = min(RMAX, R - r0);
    const double2 gam = valid ? gamma[smp] : cz(0.0, 0.0);
    const double x = pts[3 * p], y = pts[3 * p + 1], z = pts[3 * p + 2];
    double2 acc[RMAX];
#pragma unroll
    for (int r = 0; r < RMAX; ++r) acc[r] = cz(0.0, 0.0);
    for (int e0 = 0; e0 < m; e0 += 32) {
        double rbar = 0.0, gv = 0.0;
        if (e0 + lane < m) {
            const Seg& s = elec[e0 + lane];
            // examples/visacro57emc01.c:417-421 (vector_length = root of the summed squares)
            const double dm0 = x - s.mid[0], dm1 = y - s.mid[1], dm2 = z - s.mid[2];
            const double da0 = x - s.a[0], da1 = y - s.a[1], da2 = z - s.a[2];
            const double db0 = x - s.b[0], db1 = y - s.b[1], db2 = z - s.b[2];
            rbar = sqrt(dm0 * dm0 + dm1 * dm1 + dm2 * dm2);
            const double r1 = sqrt(da0 * da0 + da1 * da1 + da2 * da2);
            const double r2 = sqrt(db0 * db0 + db1 * db1 + db2 * db2);
            const double r0v = (r1 + r2 + s.len) / (r1 + r2 - s.len);
            gv = log(r0v) / s.len;
        }
        const int cnt = min(32, m - e0);
        // the same trip count in every lane, so the shuffles stay warp-uniform
        for (int jb = 0; jb < cnt; jb += NS) {
            const int j = jb + sub;
            const double rb = __shfl_sync(0xffffffffu, rbar, j & 31);
            const double g = __shfl_sync(0xffffffffu, gv, j & 31);
            if (!valid || j >= cnt) continue;
            const double2 ex = cexp_d(cz(-gam.x * rb, -gam.y * rb));
            const double2 eg = cscale(ex, g);
#pragma unroll
            for (int r = 0; r < RMAX; ++r) {
                if (r >= nr) break;
                acc[r] = cfma(cur_t[((long long)(e0 + j) * R + r0 + r) * S + smp], eg, acc[r]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < RMAX; ++r)
        for (int o = G; o < 32; o <<= 1) acc[r] = cadd(acc[r], shfl_xor2(acc[r], o));
    if (!valid || sub != 0) return;
    const double2 i4pk = cdiv(cz(1.0, 0.0), cscale(kappa[smp], TAGS_FOUR_PI));
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        if (r >= nr) break;
        gpd[((long long)smp * P + p) * R + r0 + r] = cmul(i4pk, acc[r]);
    }
}

// [S][R][m] -> [m][R][S]
__global__ void k_cur_transpose(const double2* __restrict__ in, double2* __restrict__ out, int S, int R, int m) {
    const long long n = (long long)S * R * m;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int e = (int)(i % m);
        const long long sr = i / m;
        const int r = (int)(sr % R), s = (int)(sr / R);
        out[((long long)e * R + r) * S + s] = in[i];
    }
}

// Path voltage from the end-point potentials and the path/electrode pair
// integrals jj[(s * NL + l) * m + e] (unscaled double integrals over [0,1]^2).
__global__ void k_voltage(const double* __restrict__ paths, int NL, const Seg* __restrict__ elec, int m,
                          const double2* __restrict__ cur_l, const double2* __restrict__ upts,
                          const double2* __restrict__ jj, const double2* __restrict__ svals, double mur, int R,
                          int S, double2* __restrict__ v) {
    const long long n = (long long)S * NL * R;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = (int)(i % R);
    const long long sl = i / R;
    const int l = (int)(sl % NL), s = (int)(sl / NL);
    const double* pa = paths + 6LL * l;
    const double dx[3] = {pa[3] - pa[0], pa[4] - pa[1], pa[5] - pa[2]};
    const double len2 = dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2];
    if (len2 < TAGS_DBL_EPSILON) {
        // src/electrode.c:612: the integrand fails for a path this short
        v[i] = cz(nan(""), nan(""));
        return;
    }
    const double len = sqrt(len2);
    // potentials of the two ends: upts[(s * 2NL + 2l + {0,1}) * R + r]
    const double2 u1 = upts[((long long)s * 2 * NL + 2 * l) * R + r];
    const double2 u2 = upts[((long long)s * 2 * NL + 2 * l + 1) * R + r];
    double2 out = cscale(csub(u1, u2), 1.0 / len);
    const double2 sv = svals[s];
    if (sqrt(cabs2(sv)) > TAGS_DBL_EPSILON) {
        double2 acc = cz(0.0, 0.0);
        const double2* jrow = jj + ((long long)s * NL + l) * m;
        for (int e = 0; e < m; ++e) {
            const double2 cl = cur_l[((long long)e * R + r) * S + s];
            if (sqrt(cabs2(cl)) < TAGS_DBL_EPSILON) continue;
            const Seg& g = elec[e];
            const double proj = ((g.b[0] - g.a[0]) * dx[0] + (g.b[1] - g.a[1]) * dx[1] + (g.b[2] - g.a[2]) * dx[2]) / len;
            acc = cfma(cscale(cl, proj), jrow[e], acc);
        }
        out = csub(out, cscale(cmul(sv, acc), mur * TAGS_MU0 / TAGS_FOUR_PI));
    }
    v[i] = out;
}

bool g_tables_ready[64] = {};
unsigned long long* g_evals[64] = {};   // per-device work counter

// The instance for nt terms, and its shared memory.
auto series_kernel(int nt, bool tab) {
    if (nt <= 12) return tab ? k_fields_series<12, true> : k_fields_series<12, false>;
    if (nt <= 16) return tab ? k_fields_series<16, true> : k_fields_series<16, false>;
    return tab ? k_fields_series<FS_NT, true> : k_fields_series<FS_NT, false>;
}
size_t series_smem(int nt) { return FS_E * 3 * sizeof(double) * (nt <= 12 ? 12 : nt <= 16 ? 16 : FS_NT); }

int fields_tables(int dev) {
    if (dev < 0 || dev >= 64) return TAGS_E_CUDA;
    if (g_tables_ready[dev]) return 0;
    double x[FQ], w[FQ];
    tags_gauss_legendre(FQ, x, w);
    TAGS_CUDA_OK(cudaMemcpyToSymbol(c_fx, x, sizeof(x)));
    TAGS_CUDA_OK(cudaMemcpyToSymbol(c_fw, w, sizeof(w)));
    double sx[FS_GL], sw[FS_GL];
    int off = 0;
    for (int q : FS_ORDERS) {
        tags_gauss_legendre(q, sx + off, sw + off);
        off += q;
    }
    TAGS_CUDA_OK(cudaMemcpyToSymbol(c_fsx, sx, sizeof(sx)));
    TAGS_CUDA_OK(cudaMemcpyToSymbol(c_fsw, sw, sizeof(sw)));
    for (int nt : {12, 16, FS_NT})
        for (bool tab : {true, false})
            if (cudaFuncSetAttribute(series_kernel(nt, tab), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)series_smem(nt)) != cudaSuccess)
                return tags_fail(TAGS_E_CUDA, "cudaFuncSetAttribute(k_fields_series) failed");
    TAGS_CUDA_OK(cudaMalloc(&g_evals[dev], sizeof(unsigned long long)));
    TAGS_CUDA_OK(cudaMemset(g_evals[dev], 0, sizeof(unsigned long long)));
    g_tables_ready[dev] = true;
    return 0;
}

int samples_per_warp(size_t S) {
    int g = 1;
    while (g < 32 && (size_t)g < S) g <<= 1;
    return g;
}

// Samples per device pass, so the buffers of one pass stay near 1.5 GB.
size_t chunk_samples(size_t S, size_t per_sample) {
    size_t c = per_sample ? (size_t)1.5e9 / per_sample : S;
    return std::max<size_t>(1, std::min(S, c));
}

inline double2 D2(tags_cdouble v) { return make_double2(v.re, v.im); }

// Electrode chunks per (point, sample group): enough warps for about six
// waves of two 4-warp CTAs per SM (the register-limited residency), at least
// 16 electrodes per chunk, and partial sums of at most `part_cap` bytes.
int field_chunks(size_t P, size_t ns, size_t R, size_t m, size_t part_cap) {
    const size_t G = (size_t)samples_per_warp(ns);
    const size_t warps = P * ((ns + G - 1) / G);
    const size_t target = (size_t)tags_num_sms() * 8 * 6;
    size_t c = warps ? (target + warps - 1) / warps : 1;
    c = std::min<size_t>(c, std::max<size_t>(1, m / 16));
    c = std::min<size_t>(c, 64);
    const size_t per = 7 * sizeof(double2) * P * R * ns;
    if (per) c = std::min<size_t>(c, std::max<size_t>(1, part_cap / per));
    return (int)std::max<size_t>(1, c);
}

// Geometry of the moment series over a call's points and electrodes.
struct SerGeo {
    double h = 0.0, dmax = 0.0;
    int nbk = 0;                  // 0: geometry that is not finite, no series
};

SerGeo series_geo(const double* pts, size_t P, const Seg* el, size_t m) {
    SerGeo g;
    double lo[3], hi[3], lmax = 0.0;
    bool fine = true;
    for (int c = 0; c < 3; ++c) {
        lo[c] = INFINITY;
        hi[c] = -INFINITY;
    }
    auto take = [&](const double* p) {
        for (int c = 0; c < 3; ++c) {
            fine = fine && std::isfinite(p[c]);
            lo[c] = std::min(lo[c], p[c]);
            hi[c] = std::max(hi[c], p[c]);
        }
    };
    for (size_t p = 0; p < P; ++p) take(pts + 3 * p);
    for (size_t e = 0; e < m; ++e) {
        take(el[e].a);
        take(el[e].b);
        double l2 = 0.0;
        for (int c = 0; c < 3; ++c) l2 += (el[e].b[c] - el[e].a[c]) * (el[e].b[c] - el[e].a[c]);
        lmax = std::max(lmax, sqrt(l2));
    }
    double d2 = 0.0;
    for (int c = 0; c < 3; ++c) d2 += (hi[c] - lo[c]) * (hi[c] - lo[c]);
    if (!fine || !std::isfinite(d2) || !(lmax > 0.0)) return g;
    g.h = std::max(lmax / 8.0, sqrt(d2) / 4000.0);
    g.dmax = 0.5 * (lmax + g.h);
    g.nbk = (int)(sqrt(d2) / g.h) + 2;
    return g;
}

// Terms of the series at |gamma|, 0 past its reach: x^(n-1) / (n-1)! <= 1e-17
// (one more than N_n alone needs, for the d^(n-1) of A_n).
int series_terms(const SerGeo& g, zd gamma) {
    const double x = std::abs(gamma) * g.dmax;
    if (g.nbk == 0 || !(x <= FS_XMAX)) return 0;
    double t = 1.0;
    int n = 1;
    while (n < FS_NT && t > 1e-17) t *= x / n++;
    return std::min(n + 1, FS_NT);
}

// Electrode chunks of the series: CTAs for four per SM, at least 4 electrodes
// each (a warp's lanes per pair then), partial sums of at most part_cap bytes.
void series_chunks(SerArgs* s, size_t part_cap) {
    FieldArgs& a = s->f;
    const int ngroups = (a.S + a.G - 1) / a.G;
    s->ngc = ngroups >= 3 ? 4 : ngroups;
    const long long ctas = (long long)a.P * ((ngroups + s->ngc - 1) / s->ngc);
    const size_t per = 7 * sizeof(double2) * a.P * a.R * (size_t)a.S * (4 / s->ngc);
    long long c = (tags_num_sms() * 4 + ctas - 1) / ctas;
    c = std::min<long long>(c, std::max<long long>(1, (long long)(part_cap / std::max<size_t>(per, 1))));
    c = std::min<long long>(c, (a.m + 3) / 4);
    s->echunk = (int)((a.m + c - 1) / c);
    a.schunk = (int)((a.m + s->echunk - 1) / s->echunk) * (4 / s->ngc);
}

// `direct`: samples past the series' reach are among these; `most`: the
// series' largest number of terms (0: none of these samples takes it).
int launch_fields(const SerArgs& sa, int most, double madds, bool direct, cudaStream_t st) {
    const FieldArgs& base = sa.f;
    const int ngroups = (base.S + base.G - 1) / base.G;
    const long long items = (long long)base.P * ngroups * base.nchunk;
    if (items == 0 || base.m == 0) return 0;
    const long long blocks = (items + FW - 1) / FW;
    if (blocks > 0x7fffffffLL) return tags_fail(TAGS_E_ARG, "too many points x samples for one launch");
    const int pf = tags_prof_begin(TAGS_PROF_FIELDS, st);
    if (most > 0) {
        const dim3 g((unsigned)base.P, (unsigned)(base.schunk / (4 / sa.ngc)), (unsigned)((ngroups + sa.ngc - 1) / sa.ngc));
        for (int r0 = 0; r0 < base.R; r0 += RMAX) {
            series_kernel(most, sa.tab != nullptr)<<<g, FS_THREADS, series_smem(most), st>>>(sa, r0);
            tags_note_launch();
            TAGS_CUDA_OK(cudaGetLastError());
        }
    }
    for (int r0 = 0; direct && r0 < base.R; r0 += RMAX) {
        k_fields<<<(unsigned)blocks, FW * 32, 0, st>>>(base, r0);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
    }
    const long long n = (long long)base.S * base.P * base.R;
    const int chunks = std::max(direct ? base.nchunk : 0, most > 0 ? base.schunk : 0);
    if (chunks >= 16 && n <= 32 * tags_num_sms())           // a warp each
        k_fields_reduce<32><<<(unsigned)((32 * n + 127) / 128), 128, 0, st>>>(base);
    else
        k_fields_reduce<1><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(base);
    // the series' multiply-adds (k_fields counts its rule's evaluations itself)
    tags_prof_end(TAGS_PROF_FIELDS, pf, st, 2.0 * madds * base.P * base.m, 0.0);
    tags_note_launch();
    TAGS_CUDA_OK(cudaGetLastError());
    return 0;
}

struct FieldsIn {
    const double* points;
    size_t P;
    const Electrode* elec;
    size_t m;
    const tags_cdouble* il;
    const tags_cdouble* it;
    size_t R, S;
    const tags_cdouble* gamma;
    const tags_cdouble* kappa;
    double mur;
    int want, skip_pot;
    tags_cdouble *pot, *vec, *ef;
};

// Host driver of k_fields over sample chunks (slots 10..14 of the context's
// scratch; the caller holds the drop-in lock).
int fields_run(const FieldsIn& in) {
    DeviceCtx* c = tags_ctx();
    if (!c) return tags_fail(TAGS_E_CUDA, "no usable CUDA device");
    if (int e = fields_tables(c->device)) return e;
    cudaStream_t st = c->stream;
    const size_t P = in.P, m = in.m, R = in.R, S = in.S;
    const SerGeo geo = series_geo(in.points, P, reinterpret_cast<const Seg*>(in.elec), m);
    // a table of e^{-gamma b h} where the pairs are no fewer than its buckets, or the
    // whole table is one warp per SM quarter (5 points, 24 electrodes, one sample: 160 us
    // with it, 166 with an exponential per pair)
    const bool few = (size_t)geo.nbk * S <= 32 * 4 * (size_t)tags_num_sms();
    const size_t rows = few || (size_t)geo.nbk <= P * m ? (size_t)geo.nbk : 0;
    const size_t per_sample = sizeof(double2) * (4 * R * m + P * R * 7 + 2 + FS_NT + rows) + sizeof(int);
    const size_t cs = chunk_samples(S, per_sample);
    // samples of the moment series, and those past its reach
    std::vector<int> nt(S);
    for (size_t k = 0; k < S; ++k) nt[k] = series_terms(geo, zd(in.gamma[k].re, in.gamma[k].im));
    // a warp of the rule costs the same for one of its samples as for all, so a
    // sample past the reach takes the warp's others along (42 electrodes, 126
    // points, 40 samples: 1.89 ms with the others in the series, 1.56 with none)
    for (size_t s0 = 0; s0 < S; s0 += cs) {
        const size_t ns = std::min(cs, S - s0), G = (size_t)samples_per_warp(ns);
        for (size_t g = s0; g < s0 + ns; g += G) {
            const auto b = nt.begin() + g, e = nt.begin() + std::min(g + G, s0 + ns);
            if (std::find(b, e, 0) != e) std::fill(b, e, 0);
        }
    }
    // where the series' samples are so few that the rule, bound by its own latency,
    // hardly notices them, it takes them all (its time grows by ~0.2 ms per 40,000
    // of points x electrodes x samples, what the series takes at least)
    const size_t far = (size_t)std::count(nt.begin(), nt.end(), 0);
    if (far > 0 && P * m * (S - far) <= 40000) std::fill(nt.begin(), nt.end(), 0);
    const bool any_direct = std::find(nt.begin(), nt.end(), 0) != nt.end();
    const bool any_series = std::any_of(nt.begin(), nt.end(), [](int t) { return t > 0; });
    const int nchunk = any_direct ? field_chunks(P, cs, R, m, (size_t)1e9) : 1;
    auto series_args = [&](size_t ns) {
        SerArgs s{};
        s.f.P = (int)P;
        s.f.m = (int)m;
        s.f.R = (int)R;
        s.f.S = (int)ns;
        s.f.G = samples_per_warp(ns);
        s.h = geo.h;
        s.nbk = geo.nbk;
        series_chunks(&s, (size_t)1e9);
        return s;
    };
    // partial sums of either kernel, for the largest pass
    size_t parts = any_direct ? (size_t)nchunk : 0;
    if (any_series)
        for (size_t s0 = 0; s0 < S; s0 += cs)
            parts = std::max(parts, (any_direct ? (size_t)nchunk : 0) + (size_t)series_args(std::min(cs, S - s0)).f.schunk);
    double* d_pts = (double*)c->scratch(10, sizeof(double) * 3 * P + 16);
    Seg* d_el = (Seg*)c->scratch(11, sizeof(Seg) * m + 16);
    double2* d_cur = (double2*)c->scratch(12, sizeof(double2) * 4 * R * m * cs + 16);
    double2* d_out = (double2*)c->scratch(13, sizeof(double2) * 7 * P * R * cs * (1 + parts) + 16);
    double2* d_gk = (double2*)c->scratch(14, sizeof(double2) * ((2 + FS_NT + rows) * cs) + sizeof(int) * cs + 16);
    if (!d_pts || !d_el || !d_cur || !d_out || !d_gk) return tags_fail(TAGS_E_NOMEM, "device allocation failed");
    TAGS_CUDA_OK(cudaMemcpyAsync(d_pts, in.points, sizeof(double) * 3 * P, cudaMemcpyHostToDevice, st));
    TAGS_CUDA_OK(cudaMemcpyAsync(d_el, in.elec, sizeof(Seg) * m, cudaMemcpyHostToDevice, st));
    TAGS_CUDA_OK(cudaMemsetAsync(c->status, 0, sizeof(int), st));
    for (size_t s0 = 0; s0 < S; s0 += cs) {
        const size_t ns = std::min(cs, S - s0);
        const size_t nc = R * m * ns;
        const bool turn = !((ns == 1) + (R == 1) + (m == 1) >= 2);    // else the transposed array is the same
        double2* raw_t = d_cur;               // [ns][R][m] as given
        double2* raw_l = d_cur + nc;
        double2* cur_t = turn ? d_cur + 2 * nc : raw_t;      // transposed [m][R][ns]
        double2* cur_l = turn ? d_cur + 3 * nc : raw_l;
        const bool need_t = (in.want & (WANT_POT | WANT_EF)) != 0, need_l = (in.want & WANT_VEC) != 0;
        const int tb = 256, tg = (int)std::min<size_t>((nc + tb - 1) / tb, (size_t)tags_num_sms() * 16);
        if (need_t) {
            TAGS_CUDA_OK(cudaMemcpyAsync(raw_t, in.it + s0 * R * m, sizeof(double2) * nc, cudaMemcpyHostToDevice, st));
            if (turn) {
                k_cur_transpose<<<tg, tb, 0, st>>>(raw_t, cur_t, (int)ns, (int)R, (int)m);
                tags_note_launch();
                TAGS_CUDA_OK(cudaGetLastError());
            }
        }
        if (need_l) {
            TAGS_CUDA_OK(cudaMemcpyAsync(raw_l, in.il + s0 * R * m, sizeof(double2) * nc, cudaMemcpyHostToDevice, st));
            if (turn) {
                k_cur_transpose<<<tg, tb, 0, st>>>(raw_l, cur_l, (int)ns, (int)R, (int)m);
                tags_note_launch();
                TAGS_CUDA_OK(cudaGetLastError());
            }
        }
        TAGS_CUDA_OK(cudaMemcpyAsync(d_gk, in.gamma + s0, sizeof(double2) * ns, cudaMemcpyHostToDevice, st));
        TAGS_CUDA_OK(cudaMemcpyAsync(d_gk + ns, in.kappa + s0, sizeof(double2) * ns, cudaMemcpyHostToDevice, st));
        SerArgs sa = series_args(ns);
        FieldArgs& a = sa.f;
        double2* pw = d_gk + 2 * ns;
        double2* tab = pw + (size_t)FS_NT * ns;
        int* d_nt = reinterpret_cast<int*>(tab + rows * ns);
        TAGS_CUDA_OK(cudaMemcpyAsync(d_nt, nt.data() + s0, sizeof(int) * ns, cudaMemcpyHostToDevice, st));
        const int most = *std::max_element(nt.begin() + s0, nt.begin() + s0 + ns);
        double ga = 0.0;
        for (size_t k = s0; k < s0 + ns; ++k)
            if (nt[k] > 0) ga = std::max(ga, std::abs(zd(in.gamma[k].re, in.gamma[k].im)));
        sa.ga2 = 0.25 * ga * ga;
        sa.near = ga * geo.dmax <= 1.1 ? 8 : 10;
        if (most > 0) {
            k_fser_tables<<<dim3((unsigned)((ns + 31) / 32), (unsigned)rows + 1), 32, 0, st>>>(
                d_gk, d_nt, (int)ns, (int)rows, geo.h, pw, tab);
            tags_note_launch();
            TAGS_CUDA_OK(cudaGetLastError());
        }
        sa.pw = pw;
        sa.tab = rows ? tab : nullptr;
        a.pts = d_pts;
        a.elec = d_el;
        a.cur_t = cur_t;
        a.cur_l = cur_l;
        a.gamma = d_gk;
        a.kappa = d_gk + ns;
        a.mur = in.mur;
        a.want = in.want;
        a.skip_pot = in.skip_pot;
        a.pot = d_out;
        a.vec = d_out + P * R * ns;
        a.ef = d_out + 4 * P * R * ns;
        a.status = c->status;
        a.evals = g_evals[c->device];
        a.nchunk = nchunk;
        a.part = d_out + 7 * P * R * ns;
        a.nt = d_nt;
        a.spart = a.part + 7 * P * R * ns * (any_direct ? (size_t)nchunk : 0);
        double madds = 0.0;                                  // per (point, electrode), as the series kernel's comment counts
        const bool wv = (in.want & (WANT_VEC | WANT_EF)) != 0;
        for (size_t k = s0; k < s0 + ns; ++k)
            if (nt[k] > 0)
                madds += (wv ? 6.0 : 2.0) * nt[k] + (wv ? 24.0 : 4.0) +
                         (double)R * ((in.want & WANT_EF ? 12 : 0) + (in.want & WANT_VEC ? 4 : 0) + 4);
        if (int e = launch_fields(sa, most, madds, any_direct, st)) return e;
        if (in.pot && (in.want & WANT_POT))
            TAGS_CUDA_OK(cudaMemcpyAsync(in.pot + s0 * P * R, a.pot, sizeof(double2) * P * R * ns,
                                         cudaMemcpyDeviceToHost, st));
        if (in.vec && (in.want & WANT_VEC))
            TAGS_CUDA_OK(cudaMemcpyAsync(in.vec + 3 * s0 * P * R, a.vec, sizeof(double2) * 3 * P * R * ns,
                                         cudaMemcpyDeviceToHost, st));
        if (in.ef && (in.want & WANT_EF))
            TAGS_CUDA_OK(cudaMemcpyAsync(in.ef + 3 * s0 * P * R, a.ef, sizeof(double2) * 3 * P * R * ns,
                                         cudaMemcpyDeviceToHost, st));
        TAGS_CUDA_OK(cudaStreamSynchronize(st));
    }
    int status = 0;
    TAGS_CUDA_OK(cudaMemcpyAsync(&status, c->status, sizeof(int), cudaMemcpyDeviceToHost, st));
    TAGS_CUDA_OK(cudaStreamSynchronize(st));
    return status & TAGS_ST_DEGENERATE_PAIR ? TAGS_E_GEOMETRY : 0;
}

bool bad_sizes(size_t P, size_t m, size_t R, size_t S) {
    return P > 0x7fffffffu || m > 0x7fffffffu || R > 0x7fffffffu || S > 0x7fffffffu;
}

}  // namespace

// ---- batched API -------------------------------------------------------------

extern "C" int tags_fields_batch(const double* points, size_t num_points, const Electrode* electrodes,
                                 size_t num_electrodes, const tags_cdouble* il, const tags_cdouble* it, size_t nrhs,
                                 size_t nsamples, const tags_cdouble* gamma, const tags_cdouble* kappa, double mur,
                                 tags_cdouble* pot, tags_cdouble* vecpot, tags_cdouble* efield) {
    if (num_points == 0 || nrhs == 0 || nsamples == 0) return 0;
    if (!points || !gamma || !kappa || (num_electrodes && !electrodes))
        return tags_fail(TAGS_E_ARG, "null pointer argument");
    if (bad_sizes(num_points, num_electrodes, nrhs, nsamples)) return tags_fail(TAGS_E_ARG, "size out of range");
    int want = (pot ? WANT_POT : 0) | (vecpot ? WANT_VEC : 0) | (efield ? WANT_EF : 0);
    if (((want & (WANT_POT | WANT_EF)) && !it) || ((want & WANT_VEC) && !il))
        return tags_fail(TAGS_E_ARG, "null current array");
    if (num_electrodes == 0) {
        const size_t n = num_points * nrhs * nsamples;
        if (pot) memset(pot, 0, sizeof(tags_cdouble) * n);
        if (vecpot) memset(vecpot, 0, sizeof(tags_cdouble) * 3 * n);
        if (efield) memset(efield, 0, sizeof(tags_cdouble) * 3 * n);
        return 0;
    }
    std::lock_guard<std::mutex> lk(tags_dropin_mutex());
    FieldsIn in{points, num_points, electrodes, num_electrodes, il, it, nrhs, nsamples, gamma, kappa, mur,
                want, 0, pot, vecpot, efield};
    return fields_run(in);
}

extern "C" int tags_gpd_mhem_batch(const double* points, size_t num_points, const Electrode* electrodes,
                                   size_t num_electrodes, const tags_cdouble* it, size_t nrhs, size_t nsamples,
                                   const tags_cdouble* gamma, const tags_cdouble* kappa, tags_cdouble* gpd) {
    if (num_points == 0 || nrhs == 0 || nsamples == 0) return 0;
    if (!points || !gamma || !kappa || !gpd || (num_electrodes && (!electrodes || !it)))
        return tags_fail(TAGS_E_ARG, "null pointer argument");
    if (bad_sizes(num_points, num_electrodes, nrhs, nsamples)) return tags_fail(TAGS_E_ARG, "size out of range");
    if (num_electrodes == 0) {
        memset(gpd, 0, sizeof(tags_cdouble) * num_points * nrhs * nsamples);
        return 0;
    }
    std::lock_guard<std::mutex> lk(tags_dropin_mutex());
    DeviceCtx* c = tags_ctx();
    if (!c) return tags_fail(TAGS_E_CUDA, "no usable CUDA device");
    cudaStream_t st = c->stream;
    const size_t P = num_points, m = num_electrodes, R = nrhs, S = nsamples;
    const size_t cs = chunk_samples(S, sizeof(double2) * (2 * R * m + P * R + 2));
    double* d_pts = (double*)c->scratch(10, sizeof(double) * 3 * P + 16);
    Seg* d_el = (Seg*)c->scratch(11, sizeof(Seg) * m + 16);
    double2* d_cur = (double2*)c->scratch(12, sizeof(double2) * 2 * R * m * cs + 16);
    double2* d_out = (double2*)c->scratch(13, sizeof(double2) * P * R * cs + 16);
    double2* d_gk = (double2*)c->scratch(14, sizeof(double2) * 2 * cs + 16);
    if (!d_pts || !d_el || !d_cur || !d_out || !d_gk) return tags_fail(TAGS_E_NOMEM, "device allocation failed");
    TAGS_CUDA_OK(cudaMemcpyAsync(d_pts, points, sizeof(double) * 3 * P, cudaMemcpyHostToDevice, st));
    TAGS_CUDA_OK(cudaMemcpyAsync(d_el, electrodes, sizeof(Seg) * m, cudaMemcpyHostToDevice, st));
    for (size_t s0 = 0; s0 < S; s0 += cs) {
        const size_t ns = std::min(cs, S - s0), nc = R * m * ns;
        TAGS_CUDA_OK(cudaMemcpyAsync(d_cur, it + s0 * R * m, sizeof(double2) * nc, cudaMemcpyHostToDevice, st));
        const int tb = 256, tg = (int)std::min<size_t>((nc + tb - 1) / tb, (size_t)tags_num_sms() * 16);
        k_cur_transpose<<<tg, tb, 0, st>>>(d_cur, d_cur + nc, (int)ns, (int)R, (int)m);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        TAGS_CUDA_OK(cudaMemcpyAsync(d_gk, gamma + s0, sizeof(double2) * ns, cudaMemcpyHostToDevice, st));
        TAGS_CUDA_OK(cudaMemcpyAsync(d_gk + ns, kappa + s0, sizeof(double2) * ns, cudaMemcpyHostToDevice, st));
        const int G = samples_per_warp(ns);
        const long long items = (long long)P * ((ns + G - 1) / G);
        const long long blocks = (items + FW - 1) / FW;
        if (blocks > 0x7fffffffLL) return tags_fail(TAGS_E_ARG, "too many points x samples for one launch");
        for (int r0 = 0; r0 < (int)R; r0 += RMAX) {
            k_gpd_mhem<<<(unsigned)blocks, FW * 32, 0, st>>>(d_pts, d_el, d_cur + nc, d_gk, d_gk + ns, (int)P, (int)m,
                                                             (int)R, (int)ns, G, r0, d_out);
            tags_note_launch();
            TAGS_CUDA_OK(cudaGetLastError());
        }
        TAGS_CUDA_OK(cudaMemcpyAsync(gpd + s0 * P * R, d_out, sizeof(double2) * P * R * ns, cudaMemcpyDeviceToHost, st));
        TAGS_CUDA_OK(cudaStreamSynchronize(st));
    }
    return 0;
}

extern "C" int tags_voltage_batch(const double* paths, size_t num_paths, const Electrode* electrodes,
                                  size_t num_electrodes, const tags_cdouble* il, const tags_cdouble* it, size_t nrhs,
                                  size_t nsamples, const tags_cdouble* gamma, const tags_cdouble* s,
                                  const tags_cdouble* kappa, double mur, tags_cdouble* v) {
    if (num_paths == 0 || nrhs == 0 || nsamples == 0) return 0;
    if (!paths || !gamma || !s || !kappa || !v || (num_electrodes && (!electrodes || !il || !it)))
        return tags_fail(TAGS_E_ARG, "null pointer argument");
    if (bad_sizes(2 * num_paths, num_electrodes, nrhs, nsamples)) return tags_fail(TAGS_E_ARG, "size out of range");
    const size_t NL = num_paths, m = num_electrodes, R = nrhs, S = nsamples;
    // potentials of the path ends with the field's convention (|it| below
    // DBL_EPSILON skipped, src/electrode.c:542)
    std::vector<tags_cdouble> upts(2 * NL * R * S);
    std::lock_guard<std::mutex> lk(tags_dropin_mutex());
    if (m > 0) {
        FieldsIn in{paths, 2 * NL, electrodes, m, il, it, R, S, gamma, kappa, mur, WANT_POT, 1,
                    upts.data(), nullptr, nullptr};
        int e = fields_run(in);
        if (e && e != TAGS_E_GEOMETRY) return e;
    }
    DeviceCtx* c = tags_ctx();
    if (!c) return tags_fail(TAGS_E_CUDA, "no usable CUDA device");
    if (int e = fields_tables(c->device)) return e;
    cudaStream_t st = c->stream;
    // paths as segment records after the electrodes (radius 0)
    std::vector<Seg> segs(m + NL);
    if (m) memcpy(segs.data(), electrodes, sizeof(Seg) * m);
    for (size_t l = 0; l < NL; ++l) {
        Seg& g = segs[m + l];
        const double* pa = paths + 6 * l;
        double len2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            g.a[k] = pa[k];
            g.b[k] = pa[3 + k];
            g.mid[k] = (pa[k] + pa[3 + k]) / 2.0;
            len2 += (pa[3 + k] - pa[k]) * (pa[3 + k] - pa[k]);
        }
        g.len = sqrt(len2);
        g.radius = 0.0;
    }
    const SeriesGeo geo = tags_series_geometry(segs[0].a, (int)(m + NL), nullptr, 0);
    const size_t cs = std::min<size_t>(65535, chunk_samples(S, sizeof(double2) * (2 * R * m + NL * m + 3 * NL * R + 4) +
                                                                   tags_series_workspace(geo, 1)));
    Seg* d_el = (Seg*)c->scratch(11, sizeof(Seg) * (m + NL) + 16);
    double* d_paths = (double*)c->scratch(10, sizeof(double) * 6 * NL + 16);
    double2* d_cur = (double2*)c->scratch(12, sizeof(double2) * 2 * R * m * cs + 16);
    double2* d_jj = (double2*)c->scratch(13, sizeof(double2) * (NL * m + 3 * NL * R) * cs + 16);
    double2* d_gk = (double2*)c->scratch(14, sizeof(double2) * 3 * cs + 16);
    SampleCoef* d_coef = (SampleCoef*)c->scratch(15, sizeof(SampleCoef) * cs + 16);
    if (!d_el || !d_paths || !d_cur || !d_jj || !d_gk || !d_coef)
        return tags_fail(TAGS_E_NOMEM, "device allocation failed");
    void* series = geo.nbk ? c->scratch(16, tags_series_workspace(geo, (int)cs)) : nullptr;
    TAGS_CUDA_OK(cudaMemcpyAsync(d_el, segs.data(), sizeof(Seg) * (m + NL), cudaMemcpyHostToDevice, st));
    TAGS_CUDA_OK(cudaMemcpyAsync(d_paths, paths, sizeof(double) * 6 * NL, cudaMemcpyHostToDevice, st));
    TAGS_CUDA_OK(cudaMemsetAsync(c->status, 0, sizeof(int), st));
    for (size_t s0 = 0; s0 < S; s0 += cs) {
        const size_t ns = std::min(cs, S - s0), nc = R * m * ns;
        double2* cur_l = d_cur + nc;
        double2* jj = d_jj;
        double2* d_u = d_jj + NL * m * ns;
        double2* d_v = d_u + 2 * NL * R * ns;
        if (m) {
            TAGS_CUDA_OK(cudaMemcpyAsync(d_cur, il + s0 * R * m, sizeof(double2) * nc, cudaMemcpyHostToDevice, st));
            const int tb = 256, tg = (int)std::min<size_t>((nc + tb - 1) / tb, (size_t)tags_num_sms() * 16);
            k_cur_transpose<<<tg, tb, 0, st>>>(d_cur, cur_l, (int)ns, (int)R, (int)m);
            tags_note_launch();
            TAGS_CUDA_OK(cudaGetLastError());
            std::vector<SampleCoef> coef(ns);
            for (size_t k = 0; k < ns; ++k) {
                coef[k] = SampleCoef{};
                coef[k].gamma = D2(gamma[s0 + k]);
            }
            TAGS_CUDA_OK(cudaMemcpyAsync(d_coef, coef.data(), sizeof(SampleCoef) * ns, cudaMemcpyHostToDevice, st));
            if (int e = tags_launch_path_pairs((const double*)d_el, (int)m, (const double*)(d_el + m), (int)NL, d_coef,
                                               (int)ns, jj, c->status, st, &geo, series))
                return e;
        }
        TAGS_CUDA_OK(cudaMemcpyAsync(d_u, upts.data() + s0 * 2 * NL * R, sizeof(double2) * 2 * NL * R * ns,
                                     cudaMemcpyHostToDevice, st));
        TAGS_CUDA_OK(cudaMemcpyAsync(d_gk, s + s0, sizeof(double2) * ns, cudaMemcpyHostToDevice, st));
        const long long n = (long long)ns * NL * R;
        k_voltage<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(d_paths, (int)NL, d_el, (int)m, cur_l, d_u, jj, d_gk, mur,
                                                               (int)R, (int)ns, d_v);
        tags_note_launch();
        TAGS_CUDA_OK(cudaGetLastError());
        TAGS_CUDA_OK(cudaMemcpyAsync(v + s0 * NL * R, d_v, sizeof(double2) * n, cudaMemcpyDeviceToHost, st));
        TAGS_CUDA_OK(cudaStreamSynchronize(st));
    }
    return 0;
}

extern "C" int tags_fields_evaluations(unsigned long long* count, int reset) {
    if (!count) return tags_fail(TAGS_E_ARG, "null pointer argument");
    std::lock_guard<std::mutex> lk(tags_dropin_mutex());
    DeviceCtx* c = tags_ctx();
    if (!c) return tags_fail(TAGS_E_CUDA, "no usable CUDA device");
    if (int e = fields_tables(c->device)) return e;
    TAGS_CUDA_OK(cudaMemcpyAsync(count, g_evals[c->device], sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 c->stream));
    if (reset) TAGS_CUDA_OK(cudaMemsetAsync(g_evals[c->device], 0, sizeof(unsigned long long), c->stream));
    TAGS_CUDA_OK(cudaStreamSynchronize(c->stream));
    return 0;
}

// ---- drop-ins with the reference's signatures -----------------------------------
// The reference's tolerance arguments (max_eval, req_abs_error, req_rel_error)
// are accepted and unused: the GPU rules are fixed at ~1e-12 relative.

extern "C" tags_cdouble electric_potential(const double* point, const Electrode* electrodes, size_t num_electrodes,
                                           const tags_cdouble* it, tags_cdouble gamma, tags_cdouble kappa,
                                           size_t max_eval, double req_abs_error, double req_rel_error) {
    (void)max_eval, (void)req_abs_error, (void)req_rel_error;
    tags_cdouble out{0.0, 0.0};
    // a point on an electrode leaves NaN in out (TAGS_E_GEOMETRY)
    int e = tags_fields_batch(point, 1, electrodes, num_electrodes, nullptr, it, 1, 1, &gamma, &kappa, 1.0, &out,
                              nullptr, nullptr);
    if (e && e != TAGS_E_GEOMETRY) out.re = out.im = nan("");
    return out;
}

extern "C" int magnetic_potential(const double* point, const Electrode* electrodes, size_t num_electrodes,
                                  const tags_cdouble* il, tags_cdouble gamma, double mur, size_t max_eval,
                                  double req_abs_error, double req_rel_error, tags_cdouble* va) {
    (void)max_eval, (void)req_abs_error, (void)req_rel_error;
    if (!va) return tags_fail(TAGS_E_ARG, "null pointer argument");
    const tags_cdouble kappa{1.0, 0.0};
    return tags_fields_batch(point, 1, electrodes, num_electrodes, il, nullptr, 1, 1, &gamma, &kappa, mur, nullptr,
                             va, nullptr);
}

extern "C" int electric_field(const double* point, const Electrode* electrodes, size_t num_electrodes,
                              const tags_cdouble* il, const tags_cdouble* it, tags_cdouble gamma, tags_cdouble s,
                              double mur, tags_cdouble kappa, size_t max_eval, double req_abs_error,
                              double req_rel_error, tags_cdouble* ve) {
    (void)max_eval, (void)req_abs_error, (void)req_rel_error;
    if (!ve) return tags_fail(TAGS_E_ARG, "null pointer argument");
    tags_cdouble va[3] = {}, ec[3] = {};
    const bool mag = std::abs(zd(s.re, s.im)) > TAGS_DBL_EPSILON;
    int e = tags_fields_batch(point, 1, electrodes, num_electrodes, il, it, 1, 1, &gamma, &kappa, mur, nullptr,
                              mag ? va : nullptr, ec);
    if (e && e != TAGS_E_GEOMETRY) return e;
    // src/electrode.c:530-535: with |s| > DBL_EPSILON ve is overwritten by
    // -s A, otherwise the conservative part is added to what ve holds
    for (int k = 0; k < 3; ++k) {
        zd base = mag ? -zd(s.re, s.im) * zd(va[k].re, va[k].im) : zd(ve[k].re, ve[k].im);
        zd r = base + zd(ec[k].re, ec[k].im);
        ve[k] = {r.real(), r.imag()};
    }
    return e;
}

extern "C" tags_cdouble voltage(const double* point1, const double* point2, const Electrode* electrodes,
                                size_t num_electrodes, const tags_cdouble* il, const tags_cdouble* it,
                                tags_cdouble gamma, tags_cdouble s, double mur, tags_cdouble kappa, size_t max_eval,
                                double req_abs_error, double req_rel_error) {
    (void)max_eval, (void)req_abs_error, (void)req_rel_error;
    double path[6];
    tags_cdouble out{nan(""), nan("")};
    if (!point1 || !point2) return out;
    memcpy(path, point1, sizeof(double) * 3);
    memcpy(path + 3, point2, sizeof(double) * 3);
    if (tags_voltage_batch(path, 1, electrodes, num_electrodes, il, it, 1, 1, &gamma, &s, &kappa, mur, &out))
        out.re = out.im = nan("");
    return out;
}
