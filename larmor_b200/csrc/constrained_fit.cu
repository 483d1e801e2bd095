// The constrained re-fit of log-signal fits that break a constraint (DKI's D(n) >= 0,
// K(n) >= 0, K(n) <= 3 / (b_max D(n)) on 256 directions), one warp per violating voxel.
//
// Follows constrained_fit (cpp/src/dwi/log_fit.cpp:170-216): the weighted design
// W^(1/2) X = Q R (Householder, unpivoted), the least-distance problem min ||z|| subject to
// A z >= c with A = G R^-1 and c = -G p_free, solved as the NNLS problem
// min ||[A^T; c^T] u - e|| over u >= 0 by the Lawson-Hanson active-set method with the
// least-squares fits by column-pivoted Householder QR on the active columns
// (cpp/src/sd/nnls.cpp:119-139, :187-221), at most 50 inner steps per constraint, then the
// feasibility margin, the back substitution and the check that the result meets the
// constraints up to rounding. Where any step fails the voxel keeps its unconstrained fit, as
// in the reference.
//
// DKI's own constraints take fast_refit_kernel (below); the kernels described here take every other
// constraint matrix, and what the fast kernel hands on.
//
// The NNLS matrix C = [R^-T G^T; -(G p_free)^T] ((p+1) x m) is never formed whole. Its
// gradient C^T r is G t with t = R^-1 r[:p] - r[p] p_free (G, shared by every voxel, stays in
// L2), and only the columns that join the active set are formed, each once per voxel, into a
// column cache. So a voxel moves its design's QR and the few columns it uses, not the 768-column
// system (which made the kernel move ~300x its algorithmic bytes).
//
// Work distribution: the violators were compacted into a list by the unconstrained fit; a
// fixed number of warps take them from a device work counter (no host round trip, so the pair
// of launches can be captured in a CUDA graph). Each warp owns a slot of global scratch
// memory: the QR of the weighted design (n x p), the column cache (m x (p+1), touched only for
// the columns used), the active columns' QR ((p+1) x 64), and the NNLS vectors. Lanes split
// the rows of the design for the reflections, the m constraint columns for gradients and
// steps, and the active columns for the small QR.

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "batch.cuh"
#include "common.cuh"
#include "log_fit.cuh"
#include "log_fit_warp.cuh"
#include "warp_nnls.cuh"

namespace lar {

namespace {

constexpr int kCWarps = 4;
constexpr double kEps = kEps64;
constexpr double kFeasibilityMargin = 1e-12;
constexpr int kInnerStepsPerConstraint = 50;
constexpr double kConstraintTolerance = 1e-9;

__device__ __forceinline__ double wsum(double v) { return warp_sum(v); }
__device__ __forceinline__ double wmax(double v) { return warp_max(v); }

// Per-warp shared state (p + 1 <= 32).
struct WarpState {
    double vec[4][32];  // p- or (p+1)-sized vectors: unconstrained and free solutions, scratch
    double tau[32];     // reflectors of the weighted design
    double qtau[kMaxActive], qnu[kMaxActive], qnd[kMaxActive], rv[32], res[32];
    double t[32];       // R^-1 r[:p] - r[p] p_free of the gradient
    int qperm[kMaxActive];
    int act[kMaxActive];
    int n_act;
};

// With the column sums' forward substitutions (one per lane, entry i at [i * 32 + lane]).
struct WarpShared : WarpState {
    double ysub[31 * 32];
};

constexpr int kSmemActive = 32;  // active NNLS columns whose QR fits can run in shared memory

// Where a violator's re-fit keeps its arrays: the weighted design's QR (n, p), the log signals and
// root weights (n each), the column sums' substitutions (31 x 32), the NNLS system's formed
// columns (m, p + 1), the QR of the active columns (kMaxActive, p + 1; ssub, when set, holds
// that of up to kSmemActive columns in shared memory), the NNLS vectors and flags (m each).
struct RefitMem {
    double *qr, *ys, *rw, *ysub, *ssub, *cache, *sub, *u, *z;
    uint8_t *flag, *ready;
};

// The slot layout of a warp (constrained_slot_doubles), with qr, ys and rw in it.
__device__ __forceinline__ RefitMem slot_refit_mem(double* slot, int n, int p, int m) {
    RefitMem r;
    const int rows = p + 1;
    r.qr = slot;
    r.cache = r.qr + size_t(n) * p;
    r.sub = r.cache + size_t(rows) * m;
    r.u = r.sub + size_t(rows) * kMaxActive;
    r.z = r.u + m;
    r.ys = r.z + m;
    r.rw = r.ys + n;
    r.flag = reinterpret_cast<uint8_t*>(r.rw + n);
    r.ready = r.flag + m;
    r.ysub = nullptr;
    r.ssub = nullptr;
    return r;
}

// Whether the column sums' substitutions fit in the QR's rows below R (dead by then).
__host__ __device__ inline bool refit_ysub_aliased(int n, int p) { return size_t(n - p) * p >= 31 * 32; }

// A warp's shared-memory doubles when its QR, signals, weights and small NNLS fits live there.
__host__ __device__ inline size_t refit_smem_doubles(int n, int p) {
    return size_t(n) * p + 2 * size_t(n) + size_t(p + 1) * kSmemActive + (refit_ysub_aliased(n, p) ? 0 : 31 * 32);
}

// The NNLS system C = [R^-T G^T; -(G p_free)^T] of one voxel, formed column by column on demand.
struct ImplicitSystem {
    const double* g;      // (m, p) constraints
    const double* gt;     // (p, m) the same, transposed
    const double* qr;     // (n, p): R in its upper triangle
    const double* pfree;  // (p,)
    double* cache;        // (m, p + 1)
    uint8_t* ready;       // (m,)
    int p, m;
    // Column c into the cache, unless it is there: the forward substitution R^T y = g_c with
    // lane i holding entry i (column-oriented: entry k is final once the rows above it are
    // subtracted), then y_p = -g_c p_free.
    __device__ void form(int c, int lane) const {
        if (ready[c]) return;
        const double* gc = g + size_t(c) * p;
        double* col = cache + size_t(c) * (p + 1);
        const double gi = lane < p ? gc[lane] : 0.0;
        double si = gi;
        for (int k = 0; k < p; ++k) {
            const double yk = __shfl_sync(0xffffffffu, si, k) / qr[size_t(k) * p + k];
            if (lane > k && lane < p) si -= qr[size_t(k) * p + lane] * yk;
            if (lane == k) si = yk;
        }
        const double gf = warp_sum(lane < p ? gi * pfree[lane] : 0.0);
        if (lane < p) col[lane] = si;
        if (lane == 0) {
            col[p] = -gf;
            ready[c] = 1;
        }
        __syncwarp();
    }
};

struct CachedColumns {
    const double* cache;
    int rows;
    __device__ __forceinline__ double operator()(int r, int col, int /*q*/) const {
        return cache[size_t(col) * rows + r];
    }
};

// Lawson-Hanson with QR fits on C (rows = p + 1, m columns) and d, as warp_nnls_explicit, with
// C's gradient C^T (d - C u) = G t and the active columns from the cache. Returns 1 when the
// method ended by its rule, 0 when the inner-step limit ran out, -1 past acap active columns.
__device__ int implicit_nnls(const ImplicitSystem& sys, const double* d, double tol, int max_inner, NnlsScratch s,
                             double* t, double* ssub, int lane) {
    const int m = sys.m, p = sys.p, rows = p + 1;
    const CachedColumns cols{sys.cache, rows};
    // The fit on the active columns, its QR in shared memory (ssub) when given and large enough.
    auto fit = [&]() {
        QrScratch q = s.qr;
        if (ssub != nullptr && *s.n_act <= kSmemActive) q.sub = ssub;
        warp_qr_least_squares_cols(cols, rows, s.act, *s.n_act, d, q, s.z, lane);
    };
    for (int j = lane; j < m; j += 32) {
        s.u[j] = 0.0;
        s.z[j] = 0.0;
        s.flag[j] = 0;
    }
    if (lane == 0) *s.n_act = 0;
    __syncwarp();
    int inner = 0;
    for (;;) {
        const int na = *s.n_act;
        for (int r = lane; r < rows; r += 32) {
            double acc = d[r];
            for (int q = 0; q < na; ++q) acc -= sys.cache[size_t(s.act[q]) * rows + r] * s.u[s.act[q]];
            s.res[r] = acc;
        }
        __syncwarp();
        // t = R^-1 res[:p] - res[p] p_free: column-oriented back substitution, lane i holding
        // entry i (entry k is final once the columns right of it are subtracted).
        {
            double yi = lane < p ? s.res[lane] : 0.0;
            for (int k = p - 1; k >= 0; --k) {
                const double tk = __shfl_sync(0xffffffffu, yi, k) / sys.qr[size_t(k) * p + k];
                if (lane < k) yi -= sys.qr[size_t(lane) * p + k] * tk;
                if (lane == k) yi = tk;
            }
            if (lane < p) t[lane] = yi - s.res[p] * sys.pfree[lane];
        }
        __syncwarp();
        // The gradient of every inactive column, g_c . t, lanes over the columns (each lane in
        // increasing order: the first on a tie).
        double bv = 0.0;
        int bi = -1;
        for (int c = lane; c < m; c += 32) {
            if (s.flag[c]) continue;
            double w = 0.0;
            for (int a = 0; a < p; ++a) w += sys.gt[size_t(a) * m + c] * t[a];
            if (bi < 0 || w > bv) {
                bv = w;
                bi = c;
            }
        }
        const int e = warp_argmax_first(bv, bi);
        const double ge = e >= 0 ? __shfl_sync(0xffffffffu, bv, e & 31) : 0.0;
        if (e < 0 || ge <= tol) return 1;
        if (na >= s.acap) return -1;
        sys.form(e, lane);
        if (lane == 0) {
            int q = na;
            while (q > 0 && s.act[q - 1] > e) {
                s.act[q] = s.act[q - 1];
                --q;
            }
            s.act[q] = e;
            *s.n_act = na + 1;
            s.flag[e] = 1;
        }
        __syncwarp();
        fit();
        for (;;) {
            const int n2 = *s.n_act;
            bool any = false;
            for (int q = lane; q < n2; q += 32) any |= s.z[s.act[q]] <= 0.0;
            if (!__any_sync(0xffffffffu, any)) break;
            if (++inner > max_inner) {
                for (int j = lane; j < m; j += 32) s.u[j] = s.flag[j] ? s.z[j] : 0.0;
                __syncwarp();
                return 0;
            }
            double sv = 0.0;
            int si = -1;
            for (int q = lane; q < n2; q += 32) {
                const int col = s.act[q];
                if (s.z[col] > 0.0) continue;
                const double dist = s.u[col] - s.z[col];
                const double st = dist > 0.0 ? s.u[col] / dist : 0.0;
                if (si < 0 || st < sv || (st == sv && col < si)) {
                    sv = st;
                    si = col;
                }
            }
            double step;
            const int bcol = warp_argmin_first(sv, si, &step);
            for (int j = lane; j < m; j += 32) {
                const double zj = s.flag[j] ? s.z[j] : 0.0;
                s.u[j] += step * (zj - s.u[j]);
            }
            __syncwarp();
            if (lane == 0) {
                s.u[bcol] = 0.0;
                int w = 0;
                for (int q = 0; q < n2; ++q) {
                    const int col = s.act[q];
                    if (col == bcol || !(fabs(s.u[col]) >= tol)) {
                        s.flag[col] = 0;
                        continue;
                    }
                    s.act[w++] = col;
                }
                *s.n_act = w;
            }
            __syncwarp();
            fit();
        }
        for (int j = lane; j < m; j += 32) s.u[j] = s.flag[j] ? s.z[j] : 0.0;
        __syncwarp();
    }
}

// The constrained re-fit of one violator on a warp (its unconstrained scaled parameters in
// pin): where every step succeeds, out (p) gets the constrained parameters.
template <class Src>
__device__ __forceinline__ void refit_violator(const LogDesignDevice<double>& d, const Src& src, int weighted,
                                               int64_t voxel, const double* pin, const RefitMem& mem, WarpState& sh,
                                               double* out, int lane) {
    const int n = d.n, p = d.p, m = d.m, rows = p + 1;
    double* const qr = mem.qr;
    double* const cache = mem.cache;
    double* const sub = mem.sub;
    double* const u = mem.u;
    double* const z = mem.z;
    double* const ys = mem.ys;
    double* const rw = mem.rw;
    uint8_t* const flag = mem.flag;
    uint8_t* const ready = mem.ready;
    double* pu = sh.vec[0];
    if (lane < p) pu[lane] = pin[lane];
    src.template warp_stage<double>(voxel, ys, lane);
    __syncwarp();
    // Root weights exp(pred - max pred) of the unconstrained solution (:259-263).
    double mx = -INFINITY;
    for (int j = lane; j < n; j += 32) {
        double pred = 0.0;
        for (int a = 0; a < p; ++a) pred += d.x[size_t(j) * p + a] * pu[a];
        rw[j] = pred;
        mx = fmax(mx, pred);
    }
    mx = wmax(mx);
    __syncwarp();
    for (int j = lane; j < n; j += 32) rw[j] = weighted ? exp(rw[j] - mx) : 1.0;
    __syncwarp();
    // W^(1/2) X and W^(1/2) y.
    for (int i = lane; i < n * p; i += 32) qr[i] = rw[i / p] * d.x[i];
    for (int j = lane; j < n; j += 32) ys[j] = rw[j] * ys[j];
    __syncwarp();
    // Householder QR (unpivoted), rotating ys along.
    double* tau = sh.tau;
    for (int k = 0; k < p; ++k) {
        const double c0 = qr[size_t(k) * p + k];
        double tail = 0.0;
        for (int r = k + 1 + lane; r < n; r += 32) tail += qr[size_t(r) * p + k] * qr[size_t(r) * p + k];
        tail = wsum(tail);
        double tk, beta;
        if (tail <= DBL_MIN) {
            tk = 0.0;
            beta = c0;
            for (int r = k + 1 + lane; r < n; r += 32) qr[size_t(r) * p + k] = 0.0;
        } else {
            beta = sqrt(c0 * c0 + tail);
            if (c0 >= 0.0) beta = -beta;
            const double den = c0 - beta;
            for (int r = k + 1 + lane; r < n; r += 32) qr[size_t(r) * p + k] /= den;
            tk = (beta - c0) / beta;
        }
        __syncwarp();
        if (lane == 0) {
            qr[size_t(k) * p + k] = beta;
            tau[k] = tk;
        }
        __syncwarp();
        if (tk != 0.0) {
            // Columns j > k and the data (column p), eight at a time: the dot products of a
            // group in one pass over the rows and independent warp reductions, then the
            // updates. Each dot keeps its rows' order and its reduction's.
            for (int j0 = k + 1; j0 <= p; j0 += 8) {
                double dv[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) dv[q] = 0.0;
                for (int r = k + 1 + lane; r < n; r += 32) {
                    const double vr = qr[size_t(r) * p + k];
                    const double* row = qr + size_t(r) * p;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int j = j0 + q;
                        if (j < p) dv[q] += vr * row[j];
                        else if (j == p) dv[q] += vr * ys[r];
                    }
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int j = j0 + q;
                    if (j <= p) dv[q] = wsum(dv[q]) + (j < p ? qr[size_t(k) * p + j] : ys[k]);
                }
                __syncwarp();
                if (lane == 0) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int j = j0 + q;
                        if (j < p) qr[size_t(k) * p + j] -= tk * dv[q];
                        else if (j == p) ys[k] -= tk * dv[q];
                    }
                }
                for (int r = k + 1 + lane; r < n; r += 32) {
                    double* row = qr + size_t(r) * p;
                    const double vr = row[k];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int j = j0 + q;
                        if (j < p) row[j] -= tk * vr * dv[q];
                        else if (j == p) ys[r] -= tk * vr * dv[q];
                    }
                }
                __syncwarp();
            }
        }
    }
    // Rank check on the diagonal of R (:183-188).
    double dmax = 0.0, dmin = INFINITY;
    for (int k = 0; k < p; ++k) {
        dmax = fmax(dmax, fabs(qr[size_t(k) * p + k]));
        dmin = fmin(dmin, fabs(qr[size_t(k) * p + k]));
    }
    if (!(dmin > double(n) * kEps * dmax)) return;
    // p_free = R^-1 (Q^T W^(1/2) y)[:p].
    double* pfree = sh.vec[1];
    if (lane == 0) {
        for (int i = p - 1; i >= 0; --i) {
            double s = ys[i];
            for (int j = i + 1; j < p; ++j) s -= qr[size_t(i) * p + j] * pfree[j];
            pfree[i] = s / qr[size_t(i) * p + i];
        }
    }
    __syncwarp();
    // The NNLS tolerance 10 eps norm1(C) max(p + 1, m) needs every column's absolute sum:
    // sum_i |(R^-T g_c)_i| + |g_c p_free|. Lanes over constraints, each substitution's
    // entries in the warp's shared column of ysub; the columns themselves are not kept.
    double colsum_max = 0.0;
    double* ysub = mem.ysub;
    for (int c = lane; c < m; c += 32) {
        const double* gc = d.g + size_t(c) * p;
        double acc_abs = 0.0, gf = 0.0;
        for (int i = 0; i < p; ++i) {
            double s0 = gc[i], s1 = 0.0;
            int k = 0;
            for (; k + 1 < i; k += 2) {
                s0 -= qr[size_t(k) * p + i] * ysub[k * 32 + lane];
                s1 -= qr[size_t(k + 1) * p + i] * ysub[(k + 1) * 32 + lane];
            }
            if (k < i) s0 -= qr[size_t(k) * p + i] * ysub[k * 32 + lane];
            const double si = (s0 + s1) / qr[size_t(i) * p + i];
            ysub[i * 32 + lane] = si;
            acc_abs += fabs(si);
            gf += gc[i] * pfree[i];
        }
        acc_abs += fabs(gf);
        colsum_max = fmax(colsum_max, acc_abs);
    }
    colsum_max = wmax(colsum_max);
    const double tol = 10.0 * kEps * colsum_max * double(max(rows, m));
    for (int c = lane; c < m; c += 32) ready[c] = 0;
    __syncwarp();
    // Lawson-Hanson (cpp/src/sd/nnls.cpp:187-221) on C u ~ e_p.
    double* unit = sh.vec[2];
    for (int r = lane; r < rows; r += 32) unit[r] = (r == p) ? 1.0 : 0.0;
    __syncwarp();
    const ImplicitSystem sys{d.g, d.gt, qr, pfree, cache, ready, p, m};
    NnlsScratch ns{u, z, flag, sh.act, &sh.n_act, sh.res,
                   QrScratch{sub, sh.qtau, sh.qnu, sh.qnd, sh.qperm, sh.rv}, kMaxActive};
    const int outcome = implicit_nnls(sys, unit, tol, kInnerStepsPerConstraint * m, ns, sh.t, mem.ssub, lane);
    if (outcome != 1) return;
    double* res = sh.vec[2];
    // Residual C u - e_p over the active columns (u is zero elsewhere).
    if (lane < rows) {
        double s = (lane == p) ? -1.0 : 0.0;
        for (int q = 0; q < sh.n_act; ++q) {
            const int c = sh.act[q];
            const double uc = u[c];
            if (uc != 0.0) s += cache[size_t(c) * rows + lane] * uc;
        }
        res[lane] = s;
    }
    __syncwarp();
    const double last = res[p];
    if (last >= -kFeasibilityMargin) return;
    // p = p_free + R^-1 (-res[:p] / res[p]).
    double* pc = sh.vec[3];
    if (lane == 0) {
        for (int i = p - 1; i >= 0; --i) {
            double s = -res[i] / last;
            for (int j = i + 1; j < p; ++j) s -= qr[size_t(i) * p + j] * pc[j];
            pc[i] = s / qr[size_t(i) * p + i];
        }
        for (int i = 0; i < p; ++i) pc[i] = pfree[i] + pc[i];
    }
    __syncwarp();
    bool finite = true;
    for (int a = 0; a < p; ++a) finite &= bool(isfinite(pc[a]));
    if (!finite) return;
    // meets_the_constraints (:156-163).
    double vmin = INFINITY, size = 0.0;
    for (int c = lane; c < m; c += 32) {
        const double* gr = d.g + size_t(c) * p;
        double val = 0.0, sz = 0.0;
        for (int a = 0; a < p; ++a) {
            val += gr[a] * pc[a];
            sz += fabs(gr[a]) * (fabs(pc[a]) + fabs(pfree[a]));
        }
        vmin = fmin(vmin, val);
        size = fmax(size, sz);
    }
    vmin = -wmax(-vmin);
    size = wmax(size);
    if (!(vmin >= -kConstraintTolerance * size)) return;
    if (lane < p) out[lane] = pc[lane] / d.scales64[lane];
    __syncwarp();
}

// ---- the fast re-fit of DKI's constraints ----------------------------------------------------
//
// DKI's 768 constraint rows are D, V and bound D - V on 256 directions: 21 numbers per direction
// instead of 66, so a CTA keeps them all in shared memory (43 KB) and a gradient or a check
// computes D t and V t once per direction. A warp's own state is 12 KB (twelve warps per SM):
//
// - R of the weighted design W^(1/2) X by two rounds of Cholesky on its Gram matrix (CholeskyQR2:
//   the second round orthogonalises the first's Q to rounding, Yamamoto et al., ETNA 44 (2015)
//   306-326), both Gram matrices on the FP64 tensor cores (mma.sync m8n8k4) straight from the
//   design and the weights, eight rows at a time: the 134 x 22 factor is never stored. The second
//   round's rows carry the weighted signals in a spare column, which gives Q^T y.
// - S = R^-1 next to -p_free as a 23rd column: t = S r and a column R^-T g are one product each.
// - the least-distance NNLS on orthonormal rows Q of the active columns with M = L^-1 of their
//   triangle, updated in place: a column joins by two passes of orthogonalisation (its fit is an
//   update of z), leaves by rotations whose angles come from one prefix sum (as in lsi.cu).
//
// The old kernels below built a Householder QR with a warp reduction per column, read the 768 x 22
// constraints from L2 in every gradient and refactored the active columns from scratch in every
// fit: 1.7 M cycles per violator, 180 ms for the 179,846 violators of a 199,768-voxel volume of 134
// measurements (3.9 ms for 2,832 of 95); this kernel takes 15.6 ms (0.24 ms). It is bound by the
// latency of a warp's chain of steps at twelve warps per SM. What a step here cannot take (a Cholesky pivot or an active
// column that rounding makes dependent, a table past kFastMaxRows) they fit from the start.

constexpr int kFastWarps = 12;
constexpr int kFastMaxRows = 302;  // up to here a table's weights and signals take no more of a warp's state than the NNLS
constexpr int kP = kDkiP, kR = kP + 1;           // parameters; rows of the NNLS problem
constexpr int kTile = 25;                        // row stride of an 8-row tile of Q
constexpr int kNnlsDoubles = kR * kR + kR * (kR + 1) / 2;
constexpr int kFastVectors = 8 * 24;
constexpr double kMinRatio = 1e-6;       // smallest to largest diagonal entry of R
constexpr double kMinIndependent = 1e-26;  // squared share of a column outside the active span

// The design as a violator's re-fit reads it: X (n, 22) and the D and V parts of the constraints,
// transposed with row stride ldd (in shared or global memory: the arithmetic is the same).
struct FastDesign {
    const double *x, *gd, *gv, *scales;
    int n, ldd;
    double bound;
};

__host__ __device__ inline int fast_rows(int n) { return (n + 7) / 8 * 8; }
__host__ __device__ inline size_t fast_warp_doubles(int n) {
    const size_t qr = 2 * size_t(fast_rows(n)) + 8 * kTile;
    return size_t(kP) * kR + (qr > size_t(kNnlsDoubles) ? qr : size_t(kNnlsDoubles)) + kFastVectors;
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// The lower tiles of a Gram matrix of 24 columns from four rows: v[b] = column 8 b + lane / 4 of row
// lane % 4.
__device__ __forceinline__ void gram_step(double (&acc)[6][2], const double (&v)[3]) {
    int t = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) mma_f64(acc[t++], v[i], v[j]);
}

// The accumulated lower triangle into a (stride kR), rows i < rows.
__device__ __forceinline__ void store_gram(const double (&acc)[6][2], double* a, int rows, int lane) {
    int t = 0;
#pragma unroll
    for (int bi = 0; bi < 3; ++bi)
#pragma unroll
        for (int bj = 0; bj <= bi; ++bj, ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 8 * bi + (lane >> 2), j = 8 * bj + 2 * (lane & 3) + h;
                if (i < rows && j <= i && j < kP) a[i * kR + j] = acc[t][h];
            }
}

// a (kP rows, stride kR, its lower triangle G = L L^T) <- L^-T. A lane holds a row of G, then a column
// of L^-1, in registers; each finished column of L goes round through buf (two 24-entry halves in
// turn: a shuffle would move one value at a time). False when a pivot is not positive.
__device__ __noinline__ bool cholesky_inverse(double* a, double* buf, int lane) {
    const int row = lane < kP ? lane : kP - 1;
    double g[kP];
#pragma unroll
    for (int k = 0; k < kP; ++k) g[k] = a[row * kR + k];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kP; ++k) {
        const double d = __shfl_sync(0xffffffffu, g[k], k);
        ok &= d > 0.0;
        const double inv = rsqrt(d);
        // Column k of L; its diagonal entry keeps the reciprocal.
        const double l = g[k] * inv;
        g[k] = lane == k ? inv : l;
        double* column = buf + (k & 1) * 24;
        if (lane < kP) column[lane] = l;
        __syncwarp();
#pragma unroll
        for (int j = k + 1; j < kP; ++j) g[j] = fma(-l, column[j], g[j]);
    }
    if (!ok) return false;
    __syncwarp();
    if (lane < kP) {
#pragma unroll
        for (int k = 0; k < kP; ++k)
            if (k <= lane) a[lane * kR + k] = g[k];
    }
    __syncwarp();
    // Column `lane` of L^-1: forward substitution of a unit vector.
#pragma unroll
    for (int k = 0; k < kP; ++k) g[k] = k == lane ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < kP; ++k) {
        g[k] *= a[k * kR + k];
#pragma unroll
        for (int i = k + 1; i < kP; ++i) g[i] = fma(-a[i * kR + k], g[k], g[i]);
    }
    __syncwarp();
    if (lane < kP) {
#pragma unroll
        for (int k = 0; k < kP; ++k) a[lane * kR + k] = g[k];
    }
    __syncwarp();
    return true;
}

__device__ __forceinline__ int tri(int r) { return r * (r + 1) / 2; }

// The re-fit of one violator on a warp, as refit_violator: false when it needs the other kernels.
template <class Src>
__device__ __forceinline__ bool fast_refit(const FastDesign d, const Src& src, int weighted, int64_t voxel,
                                           const double* pin, double* mem, double* out, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    const int n = d.n, rows8 = fast_rows(n);
    double* const S = mem;               // (22, 23)
    double* const B = S + kP * kR;       // rw, ys, tile; then Q and M
    double* const vec = mem + fast_warp_doubles(n) - kFastVectors;
    double *const ysm = vec, *const wv = vec + 24, *const cv = vec + 48, *const gv = vec + 72, *const rv = vec + 96,
                  *const tv = vec + 120, *const cs = vec + 144, *const sn = vec + 168;
    double *const rw = B, *const ys = B + rows8, *const tile = B + 2 * rows8;
    double *const Q = B, *const M = B + kR * kR;
    const int quad = lane >> 2, part = lane & 3;

    // Root weights exp(pred - max pred) of the unconstrained solution (:259-263) and the weighted
    // signals; rows past n weigh nothing.
    if (lane < kP) gv[lane] = pin[lane];
    src.template warp_stage<double>(voxel, ys, lane);
    __syncwarp();
    double mx = -INFINITY;
    for (int j = lane; j < n; j += 32) {
        double pred = 0.0;
#pragma unroll
        for (int a = 0; a < kP; ++a) pred = fma(d.x[j * kP + a], gv[a], pred);
        rw[j] = pred;
        mx = fmax(mx, pred);
    }
    mx = wmax(mx);
    for (int j = lane; j < rows8; j += 32) {
        const double w = j >= n ? 0.0 : weighted ? exp(rw[j] - mx) : 1.0;
        rw[j] = w;
        ys[j] = j < n ? w * ys[j] : 0.0;
    }
    __syncwarp();
    // First round: the Gram matrix of W^(1/2) X.
    {
        double acc[6][2];
#pragma unroll
        for (int t = 0; t < 6; ++t) acc[t][0] = acc[t][1] = 0.0;
        for (int r0 = 0; r0 < rows8; r0 += 4) {
            const int r = r0 + part;
            const double w = rw[r];
            const double* xr = d.x + size_t(min(r, n - 1)) * kP;
            double v[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) v[b] = 8 * b + quad < kP ? w * xr[8 * b + quad] : 0.0;
            gram_step(acc, v);
        }
        store_gram(acc, S, kP, lane);
    }
    __syncwarp();
    if (!cholesky_inverse(S, cs, lane)) return false;
    // Second round: the Gram matrix of Q = W^(1/2) X S with the weighted signals as column 22.
    {
        double acc[6][2], bs[12];
#pragma unroll
        for (int t = 0; t < 6; ++t) acc[t][0] = acc[t][1] = 0.0;
        int q = 0;
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int s = 0; s < 2 * b + 2; ++s, ++q) {
                const int a = 4 * s + part, c = 8 * b + quad;
                bs[q] = a < kP && c < kP ? S[a * kR + c] : 0.0;
            }
        for (int r0 = 0; r0 < rows8; r0 += 8) {
            const int r = r0 + quad;
            const double w = rw[r];
            const double* xr = d.x + size_t(min(r, n - 1)) * kP;
            double av[6], qt[3][2];
#pragma unroll
            for (int s = 0; s < 6; ++s) av[s] = 4 * s + part < kP ? w * xr[4 * s + part] : 0.0;
            q = 0;
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                qt[b][0] = qt[b][1] = 0.0;
#pragma unroll
                for (int s = 0; s < 2 * b + 2; ++s, ++q) mma_f64(qt[b], av[s], bs[q]);
            }
            if (part == 3) qt[2][0] = ys[r];
#pragma unroll
            for (int b = 0; b < 3; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) tile[quad * kTile + 8 * b + 2 * part + h] = qt[b][h];
            __syncwarp();
#pragma unroll
            for (int s = 0; s < 8; s += 4) {
                double v[3];
#pragma unroll
                for (int b = 0; b < 3; ++b) v[b] = tile[(s + part) * kTile + 8 * b + quad];
                gram_step(acc, v);
            }
            __syncwarp();
        }
        store_gram(acc, Q, kR, lane);
    }
    __syncwarp();
    const double qty = lane < kP ? Q[kP * kR + lane] : 0.0;
    if (!cholesky_inverse(Q, cs, lane)) return false;
    // S <- S S2 (both upper triangular), p_free = S (S2^T Q^T y).
    if (lane < kP) gv[lane] = qty;
    __syncwarp();
    {
        double v = 0.0;
        if (lane < kP)
            for (int a = 0; a < kP; ++a) v = fma(Q[a * kR + lane], gv[a], v);
        if (lane < kP) wv[lane] = v;
        double acc[6][2];
        int t = 0;
#pragma unroll
        for (int bm = 0; bm < 3; ++bm)
#pragma unroll
            for (int bn = bm; bn < 3; ++bn, ++t) {
                acc[t][0] = acc[t][1] = 0.0;
#pragma unroll
                for (int s = 2 * bm; s < 2 * bn + 2; ++s) {
                    const int a = 4 * s + part, i = 8 * bm + quad, c = 8 * bn + quad;
                    mma_f64(acc[t], a < kP && i < kP ? S[i * kR + a] : 0.0, a < kP && c < kP ? Q[a * kR + c] : 0.0);
                }
            }
        __syncwarp();
        t = 0;
#pragma unroll
        for (int bm = 0; bm < 3; ++bm)
#pragma unroll
            for (int bn = bm; bn < 3; ++bn, ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = 8 * bm + quad, c = 8 * bn + 2 * part + h;
                    if (i < kP && c < kP) S[i * kR + c] = acc[t][h];
                }
    }
    __syncwarp();
    // The diagonal of R (the rank check of :183-188 is far inside kMinRatio).
    {
        const double r = lane < kP ? fabs(1.0 / S[lane * kR + lane]) : 0.0;
        const double dmax = wmax(r), dmin = -wmax(lane < kP ? -r : -INFINITY);
        if (!(dmin > kMinRatio * dmax)) return false;
    }
    double pf = 0.0;
    if (lane < kP)
        for (int i = 0; i < kP; ++i) pf = fma(S[lane * kR + i], wv[i], pf);
    if (lane < kP) S[lane * kR + kP] = -pf;
    __syncwarp();
    // The NNLS tolerance 10 eps norm1(C) max(p + 1, m): every column's absolute sum, two directions
    // at a time (entry i of a column is the sum over k <= i; rows 1..6 have no V part).
    double norm1 = 0.0;
    for (int dir = lane; dir < kDkiDirs; dir += 64) {
        double dk[2][kDkiD], vk[2][kDkiV], sd[2] = {0.0, 0.0}, sv[2] = {0.0, 0.0}, sc[2] = {0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int k = 0; k < kDkiD; ++k) dk[q][k] = d.gd[k * d.ldd + dir + 32 * q];
#pragma unroll
            for (int k = 0; k < kDkiV; ++k) vk[q][k] = d.gv[k * d.ldd + dir + 32 * q];
        }
        for (int i = 1; i < kR; ++i) {
            double cd[2] = {0.0, 0.0}, cv2[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < kDkiD; ++k) {
                const double s = S[(1 + k) * kR + i];
#pragma unroll
                for (int q = 0; q < 2; ++q) cd[q] = fma(s, dk[q][k], cd[q]);
            }
            if (i > kDkiD) {
#pragma unroll
                for (int k = 0; k < kDkiV; ++k) {
                    const double s = S[(1 + kDkiD + k) * kR + i];
#pragma unroll
                    for (int q = 0; q < 2; ++q) cv2[q] = fma(s, vk[q][k], cv2[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                sd[q] += fabs(cd[q]);
                sv[q] += fabs(cv2[q]);
                sc[q] += fabs(fma(d.bound, cd[q], -cv2[q]));
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) norm1 = fmax(norm1, fmax(sd[q], fmax(sv[q], sc[q])));
    }
    norm1 = wmax(norm1);
    const double tol = 10.0 * kEps * norm1 * double(3 * kDkiDirs);
    // Lawson-Hanson (cpp/src/sd/nnls.cpp:187-221) on C u ~ e_p: lane r holds the r-th active column's
    // number, u and z; bit 8 b + t of `flags` is constraint b of direction lane + 32 t.
    int na = 0, inner = 0, col = -1;
    double u = 0.0, z = 1.0, rr = 0.0;
    unsigned flags = 0u;
    for (;;) {
        // The residual e_p - Q y, then t = R^-1 r[:p] - r_p p_free.
        rr = lane == kP ? 1.0 : 0.0;
        if (lane < kR)
            for (int r = 0; r < na; ++r) rr = fma(-Q[r * kR + lane], ysm[r], rr);
        if (lane < kR) rv[lane] = rr;
        __syncwarp();
        if (lane < kP) {
            double a = 0.0, b = 0.0;
            for (int i = 0; i + 1 < kR; i += 2) {
                a = fma(S[lane * kR + i], rv[i], a);
                b = fma(S[lane * kR + i + 1], rv[i + 1], b);
            }
            tv[lane] = a + fma(S[lane * kR + kP], rv[kP], b);
        }
        __syncwarp();
        double dt[8], vt[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) dt[t] = vt[t] = 0.0;
#pragma unroll
        for (int k = 0; k < kDkiD; ++k) {
            const double s = tv[1 + k];
#pragma unroll
            for (int t = 0; t < 8; ++t) dt[t] = fma(d.gd[k * d.ldd + lane + 32 * t], s, dt[t]);
        }
#pragma unroll 5
        for (int k = 0; k < kDkiV; ++k) {
            const double s = tv[1 + kDkiD + k];
#pragma unroll
            for (int t = 0; t < 8; ++t) vt[t] = fma(d.gv[k * d.ldd + lane + 32 * t], s, vt[t]);
        }
        // The steepest inactive entry, the first on a tie.
        double bv = 0.0;
        int bi = -1;
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const double w = b == 0 ? dt[t] : b == 1 ? vt[t] : fma(d.bound, dt[t], -vt[t]);
                if (!((flags >> (8 * b + t)) & 1u) && (bi < 0 || w > bv)) {
                    bv = w;
                    bi = b * kDkiDirs + lane + 32 * t;
                }
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(kAll, bv, o);
            const int oi = __shfl_xor_sync(kAll, bi, o);
            const bool take = oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi));
            bv = take ? ov : bv;
            bi = take ? oi : bi;
        }
        if (bi < 0 || bv <= tol) break;
        if (na >= kR) return false;
        // The column [R^-T g; -g p_free] of constraint bi joins.
        const int blk = bi >> 8, dir = bi & 255;
        if (lane < kP) {
            double g = 0.0;
            if (lane >= 1 && lane <= kDkiD && blk != 1) {
                g = d.gd[(lane - 1) * d.ldd + dir];
                if (blk == 2) g *= d.bound;
            } else if (lane > kDkiD && blk != 0) {
                g = d.gv[(lane - 1 - kDkiD) * d.ldd + dir];
                if (blk == 2) g = -g;
            }
            gv[lane] = g;
        }
        __syncwarp();
        double c = 0.0;
        if (lane < kR)
            for (int k = 1; k < kP; ++k) c = fma(S[k * kR + lane], gv[k], c);
        const double size = wsum(c * c);
        double w = 0.0;
        for (int pass = 0; pass < 2; ++pass) {
            if (lane < kR) cv[lane] = c;
            __syncwarp();
            double p = 0.0;
            if (lane < na)
                for (int i = 0; i < kR; ++i) p = fma(Q[lane * kR + i], cv[i], p);
            w += p;
            if (lane < na) wv[lane] = p;
            __syncwarp();
            if (lane < kR)
                for (int r = 0; r < na; ++r) c = fma(-Q[r * kR + lane], wv[r], c);
        }
        const double d2 = wsum(c * c);
        if (!(d2 > kMinIndependent * size)) return false;
        const double inv = rsqrt(d2);
        const double ye = __shfl_sync(kAll, c, kP) * inv;
        __syncwarp();
        if (lane < na) wv[lane] = w;
        if (lane < kR) Q[na * kR + lane] = c * inv;
        __syncwarp();
        double m = 0.0;
        for (int r = 0; r < na; ++r)
            if (lane <= r) m = fma(M[tri(r) + lane], wv[r], m);
        m = lane == na ? inv : -m * inv;
        if (lane <= na) M[tri(na) + lane] = m;
        if (lane < na) z = fma(m, ye, z);
        if (lane == na) {
            z = m * ye;
            u = 0.0;
            col = bi;
            ysm[na] = ye;
        }
        if (lane == (dir & 31)) flags |= 1u << (8 * blk + (dir >> 5));
        ++na;
        __syncwarp();
        // While a candidate is not positive: the blocking step, the drops, the fit.
        for (;;) {
            const bool blocks = lane < na && !(z > 0.0);
            if (!__any_sync(kAll, blocks)) break;
            if (++inner > kInnerStepsPerConstraint * 3 * kDkiDirs) return false;
            const double dist = u - z;
            double step;
            const int b = warp_argmin_first(blocks && dist > 0.0 ? u / dist : 0.0, blocks ? col : -1, &step);
            bool drop = false;
            if (lane < na) {
                u += step * (z - u);
                drop = col == b || !(fabs(u) >= tol);
            }
            unsigned gone = __ballot_sync(kAll, drop);
            while (gone) {
                const int pos = 31 - __clz(gone);
                gone ^= 1u << pos;
                const int out_col = __shfl_sync(kAll, col, pos);
                if (lane == (out_col & 31)) flags &= ~(1u << (8 * (out_col >> 8) + ((out_col & 255) >> 5)));
                // The rotations that clear column pos of M from the top down.
                const double v = lane >= pos && lane < na ? M[tri(lane) + pos] : 0.0;
                double s = v * v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double a = __shfl_up_sync(kAll, s, o);
                    if (lane >= o) s += a;
                }
                const double rt = rsqrt(s);
                const double before = __shfl_up_sync(kAll, s * rt, 1);
                if (lane > pos && lane < na) {
                    cs[lane - 1] = v * rt;
                    sn[lane - 1] = before * rt;
                }
                // Lane j runs column j's chain and Q's column j; lane 31 y's.
                double a = lane <= pos ? M[tri(pos) + lane] : 0.0;
                if (lane == 31) a = ysm[pos];
                double qa = lane < kR ? Q[pos * kR + lane] : 0.0;
                __syncwarp();
                for (int k = pos; k < na - 1; ++k) {
                    const double ck = cs[k], sk = sn[k];
                    double x = 0.0, qx = 0.0;
                    if (lane <= k + 1) x = M[tri(k + 1) + lane];
                    if (lane == 31) x = ysm[k + 1];
                    if (lane < kR) qx = Q[(k + 1) * kR + lane];
                    __syncwarp();
                    const double row = sk * x - ck * a;
                    if (lane <= k + 1 && lane != pos) M[tri(k) + (lane < pos ? lane : lane - 1)] = row;
                    if (lane == 31) ysm[k] = row;
                    a = sk * a + ck * x;
                    if (lane < kR) Q[k * kR + lane] = sk * qx - ck * qa;
                    qa = sk * qa + ck * qx;
                }
                const double un = __shfl_down_sync(kAll, u, 1);
                const int cn = __shfl_down_sync(kAll, col, 1);
                if (lane >= pos) {
                    u = un;
                    col = cn;
                }
                --na;
                __syncwarp();
            }
            z = 0.0;
            for (int r = 0; r < na; ++r)
                if (lane <= r) z = fma(M[tri(r) + lane], ysm[r], z);
        }
        if (lane < na) u = z;
    }
    // p = p_free + R^-1 (-res[:p] / res[p]) with res = C u - e_p = -rr.
    const double last = -__shfl_sync(kAll, rr, kP);
    if (last >= -kFeasibilityMargin) return true;
    if (lane < kP) wv[lane] = rr / last;
    __syncwarp();
    double pc = pf;
    if (lane < kP)
        for (int i = 0; i < kP; ++i) pc = fma(S[lane * kR + i], wv[i], pc);
    if (!__all_sync(kAll, lane >= kP || isfinite(pc))) return true;
    // meets_the_constraints (:156-163): the values, and the sums of |g| (|p| + |p_free|).
    if (lane < kP) {
        tv[lane] = pc;
        rv[lane] = fabs(pc) + fabs(pf);
    }
    __syncwarp();
    double vmin = INFINITY, most = 0.0;
    for (int dir = lane; dir < kDkiDirs; dir += 32) {
        double dv = 0.0, ds = 0.0, vv = 0.0, vs = 0.0;
#pragma unroll
        for (int k = 0; k < kDkiD; ++k) {
            const double g = d.gd[k * d.ldd + dir];
            dv = fma(g, tv[1 + k], dv);
            ds = fma(fabs(g), rv[1 + k], ds);
        }
#pragma unroll
        for (int k = 0; k < kDkiV; ++k) {
            const double g = d.gv[k * d.ldd + dir];
            vv = fma(g, tv[1 + kDkiD + k], vv);
            vs = fma(fabs(g), rv[1 + kDkiD + k], vs);
        }
        vmin = fmin(vmin, fmin(dv, fmin(vv, fma(d.bound, dv, -vv))));
        most = fmax(most, fmax(ds, fmax(vs, fma(fabs(d.bound), ds, vs))));
    }
    vmin = -wmax(-vmin);
    most = wmax(most);
    if (!(vmin >= -kConstraintTolerance * most)) return true;
    if (lane < kP) out[lane] = pc / d.scales[lane];
    return true;
}

// Warps take the violators of the list from a device counter; an entry whose voxel is ~voxel is
// done. X comes along into shared memory where it fits beside the constraints (use_x).
template <class Src>
__global__ void __launch_bounds__(kFastWarps * 32, 1) fast_refit_kernel(
    LogDesignDevice<double> d, Src src, int weighted, ViolatorList<double> list, int* queue, int use_x,
    double* __restrict__ params) {
    extern __shared__ __align__(16) double fsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* gd = fsm;
    double* gv = gd + kDkiD * kDkiDirs;
    double* xs = gv + kDkiV * kDkiDirs;
    double* mem = xs + (use_x ? d.n * kP : 0) + warp * fast_warp_doubles(d.n);
    for (int i = threadIdx.x; i < kDkiD * kDkiDirs; i += blockDim.x)
        gd[i] = d.gt[(1 + i / kDkiDirs) * d.m + i % kDkiDirs];
    for (int i = threadIdx.x; i < kDkiV * kDkiDirs; i += blockDim.x)
        gv[i] = d.gt[(1 + kDkiD + i / kDkiDirs) * d.m + kDkiDirs + i % kDkiDirs];
    if (use_x)
        for (int i = threadIdx.x; i < d.n * kP; i += blockDim.x) xs[i] = d.x[i];
    __syncthreads();
    const FastDesign fd{use_x ? xs : d.x, gd, gv, d.scales64, d.n, kDkiDirs, d.bound};
    const int total = min(*list.count, list.capacity);
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(queue, 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= total) break;
        const int64_t voxel = list.voxel[idx];
        const bool done = fast_refit<Src>(fd, src, weighted, voxel, list.params + size_t(idx) * kP, mem,
                                          params + voxel * kP, lane);
        __syncwarp();
        if (done && lane == 0) list.voxel[idx] = ~voxel;
    }
}

// The same for the DKI family of a batch: each violator with its volume's design, read from global
// memory (the arithmetic, and so the result, is the same).
__global__ void __launch_bounds__(kFastWarps * 32, 1) batch_fast_refit_kernel(
    const DkiBatchJob* __restrict__ jobs, BatchViolators list, int weighted, int n_max, int* queue) {
    extern __shared__ __align__(16) double fsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* mem = fsm + warp * fast_warp_doubles(n_max);
    const int total = min(*list.count, list.capacity);
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(queue, 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= total) break;
        const DkiBatchJob& job = jobs[list.job[idx]];
        const LogDesignDevice<double> d = job.d;
        if (!d.dki || d.n > kFastMaxRows) continue;
        const CappedSource src{job.s, job.s0, job.floor, job.is_b0, d.n};
        const FastDesign fd{d.x, d.gt + d.m, d.gt + (1 + kDkiD) * d.m + kDkiDirs, d.scales64, d.n, d.m, d.bound};
        const int64_t voxel = list.voxel[idx];
        const bool done = fast_refit<CappedSource>(fd, src, weighted, voxel, list.params + size_t(idx) * kP, mem,
                                                   job.params + voxel * kP, lane);
        __syncwarp();
        if (done && lane == 0) list.voxel[idx] = ~voxel;
    }
}

// The next violator of a warp of the kernels below: entries in turn from the counter, `step` at a
// time, those already fitted (~voxel) skipped. -1 at the end.
struct ViolatorWalk {
    int first = 0;
    unsigned todo = 0u;
    __device__ __forceinline__ int next(const int64_t* voxel, int total, int step, int* queue, int lane) {
        while (todo == 0u) {
            if (lane == 0) first = atomicAdd(queue, step);
            first = __shfl_sync(0xffffffffu, first, 0);
            if (first >= total) return -1;
            todo = __ballot_sync(0xffffffffu, lane < step && first + lane < total && voxel[first + lane] >= 0);
        }
        const int idx = first + __ffs(todo) - 1;
        todo &= todo - 1u;
        return idx;
    }
};

template <class Src>
__global__ void __launch_bounds__(kCWarps * 32, 4) constrained_fit_kernel(
    LogDesignDevice<double> d, Src src, int weighted, ViolatorList<double> list, int step, int* queue,
    double* __restrict__ workspace, size_t slot_doubles, double* __restrict__ params) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpShared* shared = reinterpret_cast<WarpShared*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpShared& sh = shared[warp];
    const int p = d.p;
    double* slot = workspace + (size_t(blockIdx.x) * kCWarps + warp) * slot_doubles;
    const int total = min(*list.count, list.capacity);
    ViolatorWalk walk;
    for (;;) {
        const int idx = walk.next(list.voxel, total, step, queue, lane);
        if (idx < 0) break;
        const int64_t voxel = list.voxel[idx];
        RefitMem mem = slot_refit_mem(slot, d.n, p, d.m);
        mem.ysub = sh.ysub;
        refit_violator<Src>(d, src, weighted, voxel, list.params + size_t(idx) * p, mem, sh, params + voxel * p,
                            lane);
    }
}

// The same re-fit with one warp per CTA and the weighted design's QR, signals, weights and the
// QR of up to kSmemActive active NNLS columns in shared memory (refit_smem_doubles): a violator
// takes ~3x fewer warp cycles than with them in the global slot, at fewer warps per SM, which
// pays while a warp's state stays small (a modest table; see launch_constrained).
template <class Src>
__global__ void __launch_bounds__(32) constrained_fit_smem_kernel(
    LogDesignDevice<double> d, Src src, int weighted, ViolatorList<double> list, int step, int* queue,
    double* __restrict__ workspace, size_t slot_doubles, double* __restrict__ params) {
    __shared__ WarpState sh;
    extern __shared__ __align__(16) double wsm[];
    const int lane = threadIdx.x & 31;
    const int n = d.n, p = d.p, rows = p + 1;
    double* slot = workspace + size_t(blockIdx.x) * slot_doubles;
    RefitMem mem = slot_refit_mem(slot, n, p, d.m);
    mem.qr = wsm;
    mem.ys = mem.qr + size_t(n) * p;
    mem.rw = mem.ys + n;
    mem.ssub = mem.rw + n;
    mem.ysub = refit_ysub_aliased(n, p) ? mem.qr + size_t(p) * p : mem.ssub + size_t(rows) * kSmemActive;
    const int total = min(*list.count, list.capacity);
    ViolatorWalk walk;
    for (;;) {
        const int idx = walk.next(list.voxel, total, step, queue, lane);
        if (idx < 0) break;
        const int64_t voxel = list.voxel[idx];
        refit_violator<Src>(d, src, weighted, voxel, list.params + size_t(idx) * p, mem, sh, params + voxel * p,
                            lane);
    }
}

// The DKI family of a batch (batch.cuh): warps take the violators of every DKI volume from one
// list, each with its volume's design, signals and outputs.
__global__ void __launch_bounds__(kCWarps * 32, 4) batch_refit_kernel(
    const DkiBatchJob* __restrict__ jobs, BatchViolators list, int weighted, int step, int* queue,
    double* __restrict__ workspace, size_t slot_doubles) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpShared* shared = reinterpret_cast<WarpShared*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpShared& sh = shared[warp];
    double* slot = workspace + (size_t(blockIdx.x) * kCWarps + warp) * slot_doubles;
    const int total = min(*list.count, list.capacity);
    ViolatorWalk walk;
    for (;;) {
        const int idx = walk.next(list.voxel, total, step, queue, lane);
        if (idx < 0) break;
        const DkiBatchJob& job = jobs[list.job[idx]];
        const LogDesignDevice<double> d = job.d;
        const CappedSource src{job.s, job.s0, job.floor, job.is_b0, d.n};
        const int64_t voxel = list.voxel[idx];
        RefitMem mem = slot_refit_mem(slot, d.n, d.p, d.m);
        mem.ysub = sh.ysub;
        refit_violator<CappedSource>(d, src, weighted, voxel, list.params + size_t(idx) * d.p, mem, sh,
                                     job.params + voxel * d.p, lane);
    }
}

}  // namespace

constexpr size_t kCSmem = kCWarps * sizeof(WarpShared);

template <class Src>
void allow_smem() {
    static_assert(kCSmem <= 200 * 1024, "the re-fit's shared state outgrows an SM");
    allow_smem(constrained_fit_kernel<Src>, kCSmem);
}

// The shared-memory re-fit is used while a warp's state stays within this many bytes (at least
// five warps per SM): on the 134-measurement DKI table (35 KB, six warps per SM) it took 187 ms
// against 213 ms with the state in the global slot at sixteen warps per SM, on the 288-measurement
// tables (65 KB, three warps per SM) it lost.
constexpr size_t kSmemRefitMaxBytes = 40 * 1024;

bool use_smem_refit(int n, int p) {
    return refit_smem_doubles(n, p) * sizeof(double) + sizeof(WarpState) <= kSmemRefitMaxBytes;
}

int global_resident_warps() {
    int per_sm = 0;
    allow_smem<CappedSource>();
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, constrained_fit_kernel<CappedSource>,
                                                             kCWarps * 32, kCSmem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    return sm_count() * ctas_per_sm(per_sm, "dki.refit.ctas_per_sm") * kCWarps;
}

template <class Kernel>
void allow_refit_smem(Kernel kernel, size_t bytes) {
    allow_smem(kernel, bytes);
}

// Where the fast re-fit runs: DKI's constraints and a table whose rows fit a warp's state.
bool use_fast_refit(int n, bool dki) { return dki && n <= kFastMaxRows; }

int constrained_resident_warps(int n, int p, bool dki) {
    // What the fast re-fit hands on is rare: about one warp per SM.
    if (use_fast_refit(n, dki)) return sm_count() / 4 * 4;
    if (!use_smem_refit(n, p)) return global_resident_warps();
    const size_t bytes = refit_smem_doubles(n, p) * sizeof(double);
    allow_refit_smem(constrained_fit_smem_kernel<CappedSource>, bytes);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, constrained_fit_smem_kernel<CappedSource>, 32,
                                                             bytes),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    return sm_count() * ctas_per_sm(per_sm, "dki.refit.ctas_per_sm") / 4 * 4;
}

size_t batch_refit_slot_doubles(int n_max, int p, int m_max) { return constrained_slot_doubles(n_max, p, m_max); }

// Batches keep the global slot: their shared memory would be sized for the largest table.
int batch_refit_slots() { return global_resident_warps(); }

bool batch_fast_refit(const LogDesignDevice<double>& d) { return use_fast_refit(d.n, d.dki); }

void launch_batch_refit(const DkiBatchJob* jobs, int n_jobs, int fast_jobs, int n_max, const BatchViolators& violators,
                        int weighted, int* queue, double* workspace, int slots, size_t slot_doubles,
                        cudaStream_t stream) {
    const int blocks = std::max(1, slots / kCWarps);
    allow_smem(batch_refit_kernel, kCSmem);
    cuda_check(cudaMemsetAsync(queue, 0, 2 * sizeof(int), stream), "cudaMemsetAsync");
    if (fast_jobs > 0) {
        const int n = std::min(n_max, kFastMaxRows);
        const size_t bytes = kFastWarps * fast_warp_doubles(n) * sizeof(double);
        allow_refit_smem(batch_fast_refit_kernel, bytes);
        LaunchScope scope("batch_fast_refit_kernel", stream);
        batch_fast_refit_kernel<<<unsigned(sm_count()), kFastWarps * 32, bytes, stream>>>(jobs, violators, weighted, n,
                                                                                          queue + 1);
        cuda_check(cudaGetLastError(), "batch_fast_refit_kernel launch");
    }
    // The other volumes' violators one by one; where every volume took the fast kernel, the few left.
    const int step = fast_jobs == n_jobs ? 32 : 1;
    LaunchScope scope("batch_refit_kernel", stream);
    batch_refit_kernel<<<blocks, kCWarps * 32, kCSmem, stream>>>(jobs, violators, weighted, step, queue, workspace,
                                                                 slot_doubles);
    cuda_check(cudaGetLastError(), "batch_refit_kernel launch");
}

template <class Src>
void launch_constrained(const LogDesignDevice<double>& d, const Src& src, int weighted,
                        const ViolatorList<double>& list, int /*list_count_host_bound*/, int* queue,
                        double* workspace, int slots, double* params, cudaStream_t stream) {
    require(d.p + 1 <= 32, "the constrained fit takes at most 31 parameters");
    const bool fast = use_fast_refit(d.n, d.dki);
    const int step = fast ? 32 : 1;
    if (fast) {
        size_t bytes = ((kDkiD + kDkiV) * kDkiDirs + kFastWarps * fast_warp_doubles(d.n)) * sizeof(double);
        const size_t x_bytes = size_t(d.n) * kP * sizeof(double);
        const bool use_x = bytes + x_bytes <= 227 * 1024;
        if (use_x) bytes += x_bytes;
        allow_refit_smem(fast_refit_kernel<Src>, bytes);
        LaunchScope scope("fast_refit_kernel", stream);
        fast_refit_kernel<Src><<<unsigned(sm_count()), kFastWarps * 32, bytes, stream>>>(d, src, weighted, list,
                                                                                       queue + 1, use_x, params);
        cuda_check(cudaGetLastError(), "fast_refit_kernel launch");
    }
    if (use_smem_refit(d.n, d.p)) {
        const size_t bytes = refit_smem_doubles(d.n, d.p) * sizeof(double);
        allow_refit_smem(constrained_fit_smem_kernel<Src>, bytes);
        LaunchScope scope("constrained_fit_kernel", stream);
        constrained_fit_smem_kernel<Src><<<std::max(1, slots), 32, bytes, stream>>>(
            d, src, weighted, list, step, queue, workspace, constrained_slot_doubles(d.n, d.p, d.m), params);
        cuda_check(cudaGetLastError(), "constrained_fit_smem_kernel launch");
        return;
    }
    const int blocks = std::max(1, slots / kCWarps);
    allow_smem<Src>();
    LaunchScope scope("constrained_fit_kernel", stream);
    constrained_fit_kernel<Src><<<blocks, kCWarps * 32, kCSmem, stream>>>(
        d, src, weighted, list, step, queue, workspace, constrained_slot_doubles(d.n, d.p, d.m), params);
    cuda_check(cudaGetLastError(), "constrained_fit_kernel launch");
}

template void launch_constrained<LogSource>(const LogDesignDevice<double>&, const LogSource&, int,
                                            const ViolatorList<double>&, int, int*, double*, int, double*,
                                            cudaStream_t);
template void launch_constrained<CappedSource>(const LogDesignDevice<double>&, const CappedSource&, int,
                                               const ViolatorList<double>&, int, int*, double*, int, double*,
                                               cudaStream_t);

}  // namespace lar
