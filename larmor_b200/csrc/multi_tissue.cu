// Multi-tissue spherical deconvolution (SDModel's mFOD method) on the GPU.
//
// Follows cpp/src/sd/multi_tissue.cpp:76-148 per voxel (a voxel's rounds do not depend on the
// other voxels of its block, cpp/tests/sd/test_multi_tissue.cpp:56): up to max_rounds rounds of
//   the anisotropic signal max(s_w - W_iso f_iso, 0) (:68-72),
//   its low-resolution FOD by non-negative least squares (solve_ridge_nnls, cpp/src/sd/nnls.cpp
//   :362-418, with the normal equations and an active-set Cholesky factor, :237-301, falling
//   back to QR on the stacked matrix from the first pivot that fails),
//   the fractions: FOD values below their median set to zero, all anisotropic tissues as one
//   column scaled to a maximum of 1, next to the isotropic columns, fitted by NNLS with QR fits
//   (compute_fractions, cpp/src/sd/fractions.cpp:70-101),
// until no fraction changes by fraction_tol; then the high-resolution FOD (ridge NNLS) and the
// per-block fractions with the final tolerance, normalised to sum to 1 (+1e-16).
//
// Work distribution: the voxels go through the rounds together, each round as three kernels
// over the list of voxels still iterating:
//   correlate_kernel  K^T max(s_w - W_iso f_iso, 0) for 32 voxels x 16 RC columns per CTA, the
//                     signals built while the tile is staged in shared memory (a tiled FP64
//                     product, each entry summed over the measurements in increasing order);
//   ridge_nnls_low_kernel the active-set NNLS on the Gram matrix and those correlations, one warp per
//                     voxel (lean_nnls.cuh; ridge_nnls_high_kernel at high resolution); the few
//                     voxels it hands back, and other sizes, take ridge_nnls_kernel (no work of the
//                     measurements' length unless its QR fallback runs);
//   lr_fractions_kernel  the fractions, the convergence test and the next round's voxel list.
// The high-resolution FOD then runs the first two for all voxels, and hr_fractions_kernel the
// final fractions. Each kernel's code is small (the warps of an SM share their instruction
// cache), and the per-voxel state between kernels lives in HBM.

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "batch.cuh"
#include "common.cuh"
#include "host_la.hpp"
#include "drl.cuh"
#include "lean_nnls.cuh"
#include "plain_fp32.cuh"
#include "warp_chol.cuh"
#include "warp_nnls.cuh"

namespace lar {

namespace {

constexpr int kMtWarps = 4;
constexpr int kCholCap = 256;   // active columns the Cholesky factor holds
constexpr int kQrCap = 64;      // active columns of the ridge QR fallback
constexpr int kMaxGroups = 16;  // fraction columns (anisotropic groups + isotropic tissues)
constexpr double kMinPivot = 1e-12;
constexpr int kMaxColumns = 640;  // kernel columns (directions) a solver may have
constexpr double kMedianTie = 1e-9;
constexpr double kFractionSumOffset = 1e-16;

struct RidgeDev {
    int m, c;
    double ridge, tol;
    int normal_equations;
    const double* k;     // (m, c) row-major
    const double* gram;  // (c, c)
};

struct TissueDev {
    int m, ca, ci, nb;
    const double* kt;    // (ca, m): the unweighted anisotropic kernel, transposed
    const double* iso;   // (m, ci)
    const double* wiso;  // (m, ci)
    const int* blocks;   // (nb, 2)
    // The constants of the lane-per-voxel fractions (FracConstants), or null where they do not apply.
    const double* fx;
    int fx_rows;
};

// The signal a ridge NNLS fits, entry i of voxel v: s(v, i) itself (single tissue), or
// max(s(v, i) w_i - sum_t W_iso(i, t) f_iso(v, t), 0) (cpp/src/sd/multi_tissue.cpp:68-72).
struct SignalDev {
    const double* s;     // (v, m)
    const double* w;     // (m,) or null: the plain signal
    const double* wiso;  // (m, ci)
    const double* fiso;  // (v, ci)
    int m, ci;
    __device__ __forceinline__ double operator()(int64_t voxel, int i) const {
        const double si = s[voxel * m + i];
        if (w == nullptr) return si;
        const double ws = __dmul_rn(si, w[i]);
        double r = 0.0;
        for (int t = 0; t < ci; ++t) r = fma(wiso[size_t(i) * ci + t], fiso[voxel * ci + t], r);
        return fmax(ws - r, 0.0);
    }
};

// The voxel at position p of a round's list (the identity when there is no list).
__device__ __forceinline__ int64_t listed(const int* list, int64_t p) { return list ? int64_t(list[p]) : p; }

// ---- correlations ----------------------------------------------------------------------
//
// The product of the signals and K on the FP64 tensor cores (mma.sync m8n8k4): a CTA keeps 48 columns
// of K for every measurement in shared memory (127 KB at 280), and a warp takes eight voxels, whose
// signals go straight from global memory into its A fragments (four consecutive samples of a voxel
// per step, a sector each; 32 samples ahead in registers) with the weights and the isotropic part
// applied on the way. What bounds it: the tensor cores (13.4 kFMA per voxel and 44 columns). The
// CUDA-core tiles below re-staged 16 measurements at a time behind two barriers and their loads'
// latency: 16.9 ms for the ten rounds and the high-resolution pass of 250,000 voxels, now 5.6 ms (3.9
// and 1.2 ms for 8,191 voxels). They take what does not fit here (corr_tc_fits).

constexpr int kCorrTcCols = 48, kCorrTcWarps = 16, kCorrTcLd = 52;  // 4 mod 16 doubles
constexpr int kCorrTcMaxIso = 3, kCorrTcUnit = 8;
constexpr int kCorrTcTicket = kCorrTcUnit * kCorrTcWarps;  // voxels of a batch's ticket
__host__ __device__ inline int corr_tc_rows(int m) { return (m + 31) / 32 * 32; }
__host__ __device__ inline size_t corr_tc_smem(int m, int ci) {
    return size_t(corr_tc_rows(m)) * (kCorrTcLd + 1 + ci) * sizeof(double);
}
__host__ __device__ inline bool corr_tc_fits(int m, int ci) {
    return ci <= kCorrTcMaxIso && corr_tc_smem(m, ci) <= 227 * 1024;
}

__device__ __forceinline__ void corr_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Columns col0.. of K, the weights and W_iso into shared memory, zero past the last measurement and
// column (the CTA; the caller synchronises).
__device__ __forceinline__ void corr_tc_stage(double* sm, const SignalDev& S, const double* __restrict__ k, int c,
                                              int col0) {
    const int m = S.m, rows = corr_tc_rows(m);
    for (int e = threadIdx.x; e < rows * kCorrTcCols; e += blockDim.x) {
        const int i = e / kCorrTcCols, j = e % kCorrTcCols;
        sm[i * kCorrTcLd + j] = i < m && col0 + j < c ? k[size_t(i) * c + col0 + j] : 0.0;
    }
    double* ws = sm + size_t(rows) * kCorrTcLd;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) ws[i] = i < m && S.w ? S.w[i] : 1.0;
    for (int i = threadIdx.x; i < rows * S.ci; i += blockDim.x) ws[rows + i] = i < m * S.ci ? S.wiso[i] : 0.0;
}

// A warp's eight voxels (voxel: the lane's, lane / 4 of the eight; -1: none) against the staged columns.
// CI isotropic tissues; CI < 0: the plain signal.
template <int CI>
__device__ __forceinline__ void corr_tc_unit(const double* sm, const SignalDev& S, int64_t voxel, int c, int col0,
                                             double* __restrict__ corr, int ldc, int lane) {
    const int m = S.m, rows = corr_tc_rows(m), l = lane & 3, v = lane >> 2;
    const double* ws = sm + size_t(rows) * kCorrTcLd;
    const double* wi = ws + rows;
    const double* s = S.s + (voxel < 0 ? 0 : voxel) * m;
    double f[CI > 0 ? CI : 1];
#pragma unroll
    for (int t = 0; t < CI; ++t) f[t] = voxel < 0 ? 0.0 : S.fiso[voxel * CI + t];
    double acc[6][2];
#pragma unroll
    for (int t = 0; t < 6; ++t) acc[t][0] = acc[t][1] = 0.0;
    double ahead[8];
    auto load = [&](int i0) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int i = i0 + 4 * q + l;
            ahead[q] = voxel >= 0 && i < m ? s[i] : 0.0;
        }
    };
    load(0);
    for (int i0 = 0; i0 < m; i0 += 32) {
        double raw[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) raw[q] = ahead[q];
        if (i0 + 32 < m) load(i0 + 32);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int i = i0 + 4 * q + l;
            double a = raw[q];
            if constexpr (CI >= 0) {
                // max(s w - W_iso f_iso, 0) (SignalDev); rows past m have no columns.
                const double weighted = __dmul_rn(a, ws[i]);
                double r = 0.0;
#pragma unroll
                for (int t = 0; t < CI; ++t) r = fma(wi[i * CI + t], f[t], r);
                a = fmax(weighted - r, 0.0);
            }
            const double* kr = sm + i * kCorrTcLd + v;
#pragma unroll
            for (int t = 0; t < 6; ++t) corr_mma(acc[t], a, kr[8 * t]);
        }
    }
    if (voxel < 0) return;
    double* out = corr + voxel * ldc + col0;
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 8 * t + 2 * l + h;
            if (col0 + j < c) out[j] = acc[t][h];
        }
}

// corr(v, j) of the listed voxels, columns 48 blockIdx.y on: the units of eight voxels dealt to the CTAs
// first, so that a short list spreads over the SMs.
template <int CI>
__global__ void __launch_bounds__(kCorrTcWarps * 32, 1) correlate_tc_kernel(
    SignalDev S, const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev,
    const double* __restrict__ k, int c, double* __restrict__ corr, int ldc) {
    if (count_dev) count = min(count, int64_t(*count_dev));
    if (count <= int64_t(blockIdx.x) * kCorrTcUnit) return;
    extern __shared__ __align__(16) double csm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col0 = blockIdx.y * kCorrTcCols;
    corr_tc_stage(csm, S, k, c, col0);
    __syncthreads();
    for (int64_t p0 = (blockIdx.x + int64_t(gridDim.x) * warp) * kCorrTcUnit; p0 < count;
         p0 += int64_t(gridDim.x) * kCorrTcWarps * kCorrTcUnit) {
        const int64_t p = p0 + (lane >> 2);
        corr_tc_unit<CI>(csm, S, p < count ? listed(list, p) : -1, c, col0, corr, ldc, lane);
    }
}

constexpr int kCorrVoxels = 32;  // voxels per CTA tile
constexpr int kCorrResidentCtas = 8;  // CTAs per SM of a correlation grid whose count is on the device
constexpr int kCorrDepth = 16;   // measurements per shared-memory stage

// corr(v, j) = sum_i K(i, j) signal(v, i), i increasing, for the listed voxels: 128 threads as
// 8 voxel lanes x 16 column lanes, each with 4 voxels x RC columns of the tile.
// corr(v, j) for the kCorrVoxels voxels vox[] (shared; -1: none) and the columns col0 .. col0 +
// 16 RC - 1 of the tile: 128 threads as 8 voxel lanes x 16 column lanes, each with 4 voxels x RC
// columns; each entry summed in increasing measurement order.
template <int RC>
__device__ __forceinline__ void correlate_tile(const SignalDev& S, const int64_t* vox, const double* __restrict__ k,
                                               int c, int col0, double* __restrict__ corr, int ldc) {
    constexpr int TC = 16 * RC;
    __shared__ double sig_t[kCorrDepth][kCorrVoxels + 1];
    __shared__ double k_t[kCorrDepth][TC];
    const int tid = threadIdx.x, tv = tid & 7, tc = tid >> 3;
    const int m = S.m;
    double acc[4][RC];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < RC; ++b) acc[a][b] = 0.0;
    for (int i0 = 0; i0 < m; i0 += kCorrDepth) {
        const int depth = min(kCorrDepth, m - i0);
        for (int e = tid; e < kCorrVoxels * kCorrDepth; e += 128) {
            const int vv = e / kCorrDepth, ii = e % kCorrDepth;
            const int64_t voxel = vox[vv];
            sig_t[ii][vv] = (voxel >= 0 && ii < depth) ? S(voxel, i0 + ii) : 0.0;
        }
        for (int e = tid; e < kCorrDepth * TC; e += 128) {
            const int ii = e / TC, cc = e % TC;
            const int col = col0 + cc;
            k_t[ii][cc] = (ii < depth && col < c) ? k[size_t(i0 + ii) * c + col] : 0.0;
        }
        __syncthreads();
        for (int ii = 0; ii < depth; ++ii) {
            double sv[4], kv[RC];
#pragma unroll
            for (int a = 0; a < 4; ++a) sv[a] = sig_t[ii][tv + 8 * a];
#pragma unroll
            for (int b = 0; b < RC; ++b) kv[b] = k_t[ii][tc + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < RC; ++b) acc[a][b] = fma(kv[b], sv[a], acc[a][b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int64_t voxel = vox[tv + 8 * a];
        if (voxel < 0) continue;
#pragma unroll
        for (int b = 0; b < RC; ++b) {
            const int col = col0 + tc + 16 * b;
            if (col < c) corr[voxel * ldc + col] = acc[a][b];
        }
    }
}

// corr(v, j) = sum_i K(i, j) signal(v, i) for the listed voxels: tiles of kCorrVoxels voxels x
// 16 RC columns, a CTA's tiles strided by the grid (a round whose count lives on the device is
// launched with a resident-sized grid, so an empty round costs little).
template <int RC>
__global__ void __launch_bounds__(128) correlate_kernel(SignalDev S, const int* __restrict__ list, int64_t count,
                                                        const int* __restrict__ count_dev,
                                                        const double* __restrict__ k, int c,
                                                        double* __restrict__ corr, int ldc) {
    __shared__ int64_t vox[kCorrVoxels];
    const int tid = threadIdx.x;
    if (count_dev) count = min(count, int64_t(*count_dev));
    for (int64_t p0 = int64_t(blockIdx.x) * kCorrVoxels; p0 < count; p0 += int64_t(gridDim.x) * kCorrVoxels) {
        __syncthreads();  // the previous tile's voxels are read
        if (tid < kCorrVoxels) vox[tid] = p0 + tid < count ? listed(list, p0 + tid) : -1;
        __syncthreads();
        correlate_tile<RC>(S, vox, k, c, blockIdx.y * 16 * RC, corr, ldc);
    }
}

// ---- ridge NNLS ------------------------------------------------------------------------

// A warp's NNLS workspace. Shared memory: the solution x, its candidate z, the factor's vectors
// h, w and y (InvFactor), the active and in-factor flags. Global slot: the packed factor and
// its inverse, the signal (for the QR fallback) and the QR workspace.
struct NnlsSlot {
    double *x, *z, *h, *w, *y, *L, *M, *sig, *qsub, *qd, *qrv;
    uint8_t *flag, *inf;
};

inline size_t nnls_slot_doubles(int m, int cap) {
    return 2 * size_t(packed_size(cap)) + size_t(m) + size_t(m + kQrCap) * kQrCap + 2 * size_t(m + kQrCap) + 8;
}

__host__ __device__ inline size_t nnls_smem_bytes(int c, int cap) {
    return ((2 * size_t(c) + 3 * size_t(cap)) * sizeof(double) + 2 * size_t(c) + 15) / 16 * 16;
}

__device__ NnlsSlot carve_nnls(double* base, unsigned char* smem, int m, int c, int cap) {
    NnlsSlot s;
    double* p = base;
    s.L = p; p += packed_size(cap);
    s.M = p; p += packed_size(cap);
    s.sig = p; p += m;
    s.qsub = p; p += size_t(m + kQrCap) * kQrCap;
    s.qd = p; p += m + kQrCap;
    s.qrv = p;
    double* q = reinterpret_cast<double*>(smem);
    s.x = q; q += c;
    s.z = q; q += c;
    s.h = q; q += cap;
    s.w = q; q += cap;
    s.y = q; q += cap;
    s.flag = reinterpret_cast<uint8_t*>(q);
    s.inf = s.flag + c;
    return s;
}

template <int CAP, int CMAX>
struct NnlsState {
    int cols[CAP];     // factor columns, joining order
    int sorted[CMAX];  // columns with x != 0, increasing; the columns to append again in a fit
    int qact[kQrCap];  // QR fallback active columns, increasing
    double qtau[kQrCap], qnu[kQrCap], qnd[kQrCap];
    int qperm[kQrCap];
};

// The stacked columns [K_A; ridge I] of the ridge QR fallback.
struct StackedColumns {
    const double* k;
    int m, c;
    double ridge;
    __device__ __forceinline__ double operator()(int r, int col, int q) const {
        return r < m ? k[size_t(r) * c + col] : (r - m == q ? ridge : 0.0);
    }
};

// Least squares on the active columns by QR (fit_by_qr, cpp/src/sd/nnls.cpp:385-401); false
// when more columns are active than the QR workspace holds.
template <class State>
__device__ __noinline__ bool ridge_qr_fit(const RidgeDev R, const double* sig, const NnlsSlot sl, State& st, int lane) {
    int k = 0;
    if (lane == 0) {
        for (int j = 0; j < R.c; ++j)
            if (sl.flag[j]) {
                if (k < kQrCap) st.qact[k] = j;
                ++k;
            }
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    for (int j = lane; j < R.c; j += 32) sl.z[j] = 0.0;
    __syncwarp();
    if (k > kQrCap) return false;
    const bool has_ridge = R.ridge > 0.0;
    const int rows = R.m + (has_ridge ? k : 0);
    for (int r = lane; r < rows; r += 32) sl.qd[r] = r < R.m ? sig[r] : 0.0;
    __syncwarp();
    QrScratch qs{sl.qsub, st.qtau, st.qnu, st.qnd, st.qperm, sl.qrv};
    warp_qr_least_squares_cols(StackedColumns{R.k, R.m, R.c, R.ridge}, rows, st.qact, k, sl.qd, qs, sl.z, lane);
    return true;
}

// min ||K x - sig||^2 + ridge^2 ||x||^2 over x >= 0 (solve_ridge_nnls with l1 = 0,
// cpp/src/sd/nnls.cpp:362-418) from corr = K^T sig, the result in sl.x. The signal itself is
// built only when a QR fit needs it. Returns false only when the QR fallback's workspace
// overflowed (x is then the last fit). VPL * 32 is the factor's capacity, CPL * 32 >= c.
//
// Inlined into its kernel with every argument by value, so that its state (the active count,
// the flags, the workspace pointers) stays in registers; the outer (entering column) and inner
// (blocking step) iterations of Lawson-Hanson share one loop with one fit, so the factor code
// is emitted once.
template <int VPL, int CPL, class State>
__device__ __forceinline__ bool ridge_nnls(const RidgeDev R, const SignalDev S, int64_t voxel,
                                           const double* __restrict__ corr, const NnlsSlot sl, State& st,
                                           int lane) {
    const int c = R.c;
    const InvFactor fac{sl.L, sl.M, sl.h, sl.w, sl.y, st.cols, VPL * 32};
    for (int j = lane; j < c; j += 32) {
        sl.x[j] = 0.0;
        sl.z[j] = 0.0;
        sl.flag[j] = 0;
        sl.inf[j] = 0;
    }
    __syncwarp();
    const bool use_qr_only = !R.normal_equations;
    bool failed = false, overflow = false, have_sig = false;
    int na = 0, inner = 0;
    const int max_inner = 3 * c;
    bool blocked = false;  // the last fit left an active column at or below zero: an inner step
    for (;;) {
        int entering = -1;
        if (!blocked) {
            // Outer step: the gradient corr - G x over the non-zero x, columns in increasing
            // order; the steepest inactive entry, the first on a tie.
            int n_sorted = 0;
            for (int base = 0; base < c; base += 32) {
                const int j = base + lane;
                const bool nz = j < c && sl.x[j] != 0.0;
                const unsigned ballot = __ballot_sync(0xffffffffu, nz);
                if (nz) st.sorted[n_sorted + __popc(ballot & ((1u << lane) - 1u))] = j;
                n_sorted += __popc(ballot);
            }
            __syncwarp();
            double g[CPL];
#pragma unroll
            for (int t = 0; t < CPL; ++t) {
                const int j = lane + 32 * t;
                g[t] = j < c ? corr[j] : 0.0;
            }
            for (int q = 0; q < n_sorted; ++q) {
                const int col = st.sorted[q];
                const double xc = sl.x[col];
                const double* row = R.gram + size_t(col) * c;
#pragma unroll
                for (int t = 0; t < CPL; ++t) {
                    const int j = lane + 32 * t;
                    if (j < c) g[t] -= xc * row[j];
                }
            }
            double bv = 0.0;
            int bi = -1;
#pragma unroll
            for (int t = 0; t < CPL; ++t) {
                const int j = lane + 32 * t;
                if (j < c && !sl.flag[j] && (bi < 0 || g[t] > bv)) { bv = g[t]; bi = j; }
            }
            const int e = warp_argmax_first(bv, bi);
            const double ge = e >= 0 ? __shfl_sync(0xffffffffu, bv, e & 31) : 0.0;
            if (e < 0 || ge <= R.tol) break;
            if (lane == 0) sl.flag[e] = 1;
            __syncwarp();
            entering = e;
        } else {
            // Inner step: move towards the fit until the first active column reaches zero,
            // drop it and every active column below the tolerance.
            if (++inner > max_inner) {
                // The last least-squares fit is the answer (cpp/src/sd/nnls.cpp:204-207).
                for (int j = lane; j < c; j += 32) sl.x[j] = sl.z[j];
                __syncwarp();
                return !overflow;
            }
            double sv = 0.0;
            int si = -1;
            for (int j = lane; j < c; j += 32) {
                if (!sl.flag[j] || sl.z[j] > 0.0) continue;
                const double dist = sl.x[j] - sl.z[j];
                const double stp = dist > 0.0 ? sl.x[j] / dist : 0.0;
                if (si < 0 || stp < sv) { sv = stp; si = j; }
            }
            double step;
            const int b = warp_argmin_first(sv, si, &step);
            for (int j = lane; j < c; j += 32) sl.x[j] += step * (sl.z[j] - sl.x[j]);
            __syncwarp();
            if (lane == 0) {
                sl.x[b] = 0.0;
                sl.flag[b] = 0;
            }
            __syncwarp();
            for (int j = lane; j < c; j += 32)
                if (sl.flag[j] && !(fabs(sl.x[j]) >= R.tol)) sl.flag[j] = 0;
            __syncwarp();
        }
        // The fit on the active set (ActiveCholesky::update, :246-262), or QR from the first
        // failing pivot on: the columns that left the active set leave the factor (from the
        // last position down), then the entering column joins (every other active column is
        // in the factor already, so update()'s scan appends only it).
        if (!use_qr_only && !failed) {
            for (int pos = na - 1; pos >= 0; --pos) {
                const int col = st.cols[pos];
                if (sl.flag[col]) continue;
                if (VPL == 1 || na <= 32) inv_remove<1>(fac, na, pos, lane);
                else inv_remove<VPL>(fac, na, pos, lane);
                if (lane == 0) sl.inf[col] = 0;
                --na;
                __syncwarp();
            }
            if (entering >= 0) {
                for (int r = lane; r < na; r += 32) sl.h[r] = R.gram[size_t(st.cols[r]) * c + entering];
                __syncwarp();
                // Below 32 active columns one row slice per lane holds the factor's rows: the
                // one-slice code skips the unrolled empty slices of the larger capacity.
                const double gee = R.gram[size_t(entering) * c + entering];
                const bool appended =
                    (VPL == 1 || na < 32)
                        ? inv_append<1>(fac, na, gee, corr[entering], entering, kMinPivot, lane)
                        : inv_append<VPL>(fac, na, gee, corr[entering], entering, kMinPivot, lane);
                if (!appended) {
                    failed = true;
                } else {
                    if (lane == 0) sl.inf[entering] = 1;
                    __syncwarp();
                }
            }
        }
        if (use_qr_only || failed) {
            if (!have_sig) {
                for (int i = lane; i < R.m; i += 32) sl.sig[i] = S(voxel, i);
                __syncwarp();
                have_sig = true;
            }
            overflow |= !ridge_qr_fit(R, sl.sig, sl, st, lane);
        } else if (VPL == 1 || na <= 32) {
            inv_solve<1>(fac, na, sl.z, c, lane);
        } else {
            inv_solve<VPL>(fac, na, sl.z, c, lane);
        }
        bool any = false;
        for (int j = lane; j < c; j += 32) any |= sl.flag[j] && sl.z[j] <= 0.0;
        blocked = __any_sync(0xffffffffu, any);
        if (!blocked) {
            for (int j = lane; j < c; j += 32) sl.x[j] = sl.z[j];
            __syncwarp();
        }
    }
    return !overflow;
}

// One warp per listed voxel, pulled from a device counter: x(v) <- the ridge NNLS of corr(v);
// bad(v) <- 1 when the QR fallback overflowed.
template <int VPL, int CPL>
__global__ void __launch_bounds__(kMtWarps * 32, (CPL <= 2 ? 6 : 4)) ridge_nnls_kernel(
    RidgeDev R, SignalDev S, const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev,
    const double* __restrict__ corr, int ldc, double* __restrict__ x_out, int ldx, uint8_t* __restrict__ bad,
    int* queue, double* __restrict__ workspace, size_t slot_size) {
    using State = NnlsState<VPL * 32, CPL * 32>;
    if (count_dev) count = min(count, int64_t(*count_dev));
    __shared__ State states[kMtWarps];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    State& st = states[warp];
    NnlsSlot sl = carve_nnls(workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size,
                             smem_raw + warp * nnls_smem_bytes(R.c, VPL * 32), R.m, R.c, VPL * 32);
    for (;;) {
        int64_t p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= count) break;
        const int64_t voxel = listed(list, p);
        const bool ok = ridge_nnls<VPL, CPL>(R, S, voxel, corr + voxel * ldc, sl, st, lane);
        for (int j = lane; j < R.c; j += 32) x_out[voxel * ldx + j] = sl.x[j];
        if (lane == 0 && !ok && bad) bad[voxel] = 1;
        __syncwarp();
    }
}

// ---- ridge NNLS of small active sets (lean_nnls.cuh) ---------------------------------------------

// Low-resolution kernels (at most kLowCols columns): the Gram matrix in the CTA's shared memory.
constexpr int kLowCols = 48, kLowWarps = 16;
inline size_t low_smem_bytes(int c) {
    return (size_t(kLowWarps) * kLeanWarpDoubles + size_t(c) * c) * sizeof(double);
}
// High-resolution kernels: its rows come from L2.
constexpr int kHighWarps = 4, kHighCtas = 5;
inline size_t high_smem_bytes() { return size_t(kHighWarps) * kLeanWarpDoubles * sizeof(double); }

__device__ __forceinline__ void stage_gram(double* gs, const RidgeDev& R) {
    for (int i = threadIdx.x; i < R.c * R.c; i += blockDim.x) gs[i] = R.gram[i];
}

// One warp per listed voxel, pulled from a device counter: x(v) <- the ridge NNLS of corr(v), or v
// appended to `redo` when it needs the full-factor kernel.
__global__ void __launch_bounds__(kLowWarps * 32, 2) ridge_nnls_low_kernel(
    RidgeDev R, const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev,
    const double* __restrict__ corr, int ldc, double* __restrict__ x_out, int ldx, int* __restrict__ redo,
    int* redo_count, int* queue) {
    if (count_dev) count = min(count, int64_t(*count_dev));
    if (count == 0) return;
    extern __shared__ __align__(16) double lsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LeanWarp q(lsm + warp * kLeanWarpDoubles);
    double* const gs = lsm + kLowWarps * kLeanWarpDoubles;
    stage_gram(gs, R);
    __syncthreads();
    for (;;) {
        int p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= count) break;
        const int64_t voxel = listed(list, p);
        if (!lean_nnls<2>(gs, R.c, R.c, R.tol, kMinPivot, corr + voxel * ldc, q, x_out + voxel * ldx, lane) && lane == 0)
            redo[atomicAdd(redo_count, 1)] = int(voxel);
        __syncwarp();
    }
}

// The first pass of the high-resolution NNLS (65 to 320 columns): the active sets of the 300-direction
// FODs rarely pass 32 columns, and the voxels that do go on `redo`.
__global__ void __launch_bounds__(kHighWarps * 32, kHighCtas) ridge_nnls_high_kernel(
    RidgeDev R, int64_t count, const double* __restrict__ corr, int ldc, double* __restrict__ x_out, int ldx,
    int* __restrict__ redo, int* redo_count, int* queue) {
    extern __shared__ __align__(16) double lsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LeanWarp q(lsm + warp * kLeanWarpDoubles);
    for (;;) {
        int voxel = 0;
        if (lane == 0) voxel = atomicAdd(queue, 1);
        voxel = __shfl_sync(0xffffffffu, voxel, 0);
        if (voxel >= count) break;
        if (!lean_nnls<10>(R.gram, R.c, R.c, R.tol, kMinPivot, corr + int64_t(voxel) * ldc, q,
                           x_out + int64_t(voxel) * ldx, lane) &&
            lane == 0)
            redo[atomicAdd(redo_count, 1)] = voxel;
        __syncwarp();
    }
}

// ---- fractions -------------------------------------------------------------------------

// A warp's fraction workspace in its global slot: the thresholded FOD, the fraction columns
// (row-major) and the NNLS / QR workspace.
struct FracSlot {
    double *th, *cols, *fu, *fz, *fsub, *frv, *res;
    uint8_t* fflag;
};

inline size_t frac_slot_doubles(int m, int ca, int ng) {
    return size_t(ca) + size_t(m) * ng + 2 * size_t(ng) + size_t(ng) * m + 2 * size_t(m) + (size_t(ng) + 7) / 8 + 8;
}

__device__ FracSlot carve_frac(double* base, int m, int ca, int ng) {
    FracSlot s;
    double* p = base;
    s.th = p; p += ca;
    s.cols = p; p += size_t(m) * ng;
    s.fu = p; p += ng;
    s.fz = p; p += ng;
    s.fsub = p; p += size_t(ng) * m;
    s.frv = p; p += m;
    s.res = p; p += m;
    s.fflag = reinterpret_cast<uint8_t*>(p);
    return s;
}

struct FracState {
    int fact[kMaxGroups], fn_act;
    double ftau[kMaxGroups], fnu[kMaxGroups], fnd[kMaxGroups];
    int fperm[kMaxGroups];
    double fr[kMaxGroups];
    double med[2];
    uint16_t idx[kMaxColumns];  // the columns above the threshold, increasing
};

// Median of v[0..n), the mean of the two middle values for even n (cpp/src/sd/fractions.cpp:56-68). A
// non-negative vector with more zeros than half, as an NNLS solution is, has median 0; else by
// ranks: the element of stable rank r is the r-th smallest (300 x 300 comparisons at high
// resolution).
__device__ __forceinline__ double warp_median(const double* v, int n, FracState& st, int lane) {
    const int hi = n / 2, lo = n % 2 ? n / 2 : n / 2 - 1;
    int zeros = 0;
    bool odd = false;
    for (int i = lane; i < n; i += 32) {
        zeros += v[i] == 0.0;
        odd |= !(v[i] >= 0.0);
    }
    zeros = __reduce_add_sync(0xffffffffu, zeros);
    if (!__any_sync(0xffffffffu, odd) && zeros > hi) return 0.0;
    for (int i = lane; i < n; i += 32) {
        const double vi = v[i];
        int rank = 0;
        for (int j = 0; j < n; ++j) {
            const double vj = v[j];
            rank += (vj < vi) || (vj == vi && j < i);
        }
        if (rank == hi) st.med[0] = vi;
        if (rank == lo) st.med[1] = vi;
    }
    __syncwarp();
    return n % 2 ? st.med[0] : (st.med[1] + st.med[0]) / 2.0;
}

constexpr int kFastRowsPerLane = 10;  // measurements per lane of the register fraction fit (m <= 320)

// Lawson-Hanson (cpp/src/sd/nnls.cpp:187-221) on the normal equations G u = b of at most four
// columns, every lane running the same scalar steps: the gradient b - G u over the active
// columns, the steepest inactive column (the first on a tie), the least-squares fit of the
// active block by Cholesky, the blocking step and the drops below tol, at most max_inner inner
// steps. Inactive rows of the active block's system are the identity, so each solve runs on
// compile-time indices. False when a pivot is not positive (the caller then fits by QR).
__device__ __forceinline__ bool small_nnls(const double (&G)[4][4], const double (&b)[4], int n, double tol,
                                           int max_inner, double (&u)[4]) {
    bool flag[4];
    double z[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        flag[j] = false;
        u[j] = 0.0;
        z[j] = 0.0;
    }
    auto solve = [&]() -> bool {
        double L[4][4], y[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int c = 0; c <= a; ++c) {
                double sum = flag[a] && flag[c] ? G[a][c] : (a == c ? 1.0 : 0.0);
#pragma unroll
                for (int k = 0; k < c; ++k) sum -= L[a][k] * L[c][k];
                if (a == c) {
                    if (!(sum > 0.0)) return false;
                    L[a][a] = sqrt(sum);
                } else {
                    L[a][c] = sum / L[c][c];
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double sum = flag[a] ? b[a] : 0.0;
#pragma unroll
            for (int k = 0; k < a; ++k) sum -= L[a][k] * y[k];
            y[a] = sum / L[a][a];
        }
#pragma unroll
        for (int a = 3; a >= 0; --a) {
            double sum = y[a];
#pragma unroll
            for (int k = a + 1; k < 4; ++k) sum -= L[k][a] * z[k];
            z[a] = flag[a] ? sum / L[a][a] : 0.0;
        }
        return true;
    };
    int inner = 0;
    for (;;) {
        int e = -1;
        double best = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j >= n) continue;
            double w = b[j];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (flag[q]) w -= G[j][q] * u[q];
            if (!flag[j] && (e < 0 || w > best)) {
                best = w;
                e = j;
            }
        }
        if (e < 0 || best <= tol) return true;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j == e) flag[j] = true;
        if (!solve()) return false;
        for (;;) {
            bool any = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) any |= flag[j] && z[j] <= 0.0;
            if (!any) break;
            if (++inner > max_inner) {
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = flag[j] ? z[j] : 0.0;
                return true;
            }
            double sv = 0.0;
            int si = -1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (!flag[j] || z[j] > 0.0) continue;
                const double dist = u[j] - z[j];
                const double stp = dist > 0.0 ? u[j] / dist : 0.0;
                if (si < 0 || stp < sv) {
                    sv = stp;
                    si = j;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double zj = flag[j] ? z[j] : 0.0;
                u[j] += sv * (zj - u[j]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j == si) u[j] = 0.0;
                if (flag[j] && (j == si || !(fabs(u[j]) >= tol))) flag[j] = false;
            }
            if (!solve()) return false;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = flag[j] ? z[j] : 0.0;
    }
}

// compute_fractions for one anisotropic column next to at most three isotropic ones and at most
// 320 measurements: the column K th scaled to a maximum of 1 in registers (over the columns listed
// first, above the threshold), then C^T C, C^T s and the columns' norm1 in one reduction, and the NNLS
// on those (small_nnls). False when that needs the QR fit.
__device__ __forceinline__ bool fractions_small(const TissueDev T, const double* fod, const double* sig, int gb, int ge,
                                                double threshold, double tol, FracState& st, int lane) {
    const int m = T.m, ci = T.ci, n = 1 + ci;
    int kept = 0;
    for (int j0 = gb; j0 < ge; j0 += 32) {
        const int j = j0 + lane;
        const double f = j < ge ? fod[j] : 0.0;
        const bool in = j < ge && !(f < threshold) && f != 0.0;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) st.idx[kept + __popc(b & ((1u << lane) - 1u))] = uint16_t(j);
        kept += __popc(b);
    }
    __syncwarp();
    double col[kFastRowsPerLane];
#pragma unroll
    for (int t = 0; t < kFastRowsPerLane; ++t) col[t] = 0.0;
    for (int q = 0; q < kept; ++q) {
        const int j = st.idx[q];
        const double tj = fod[j];
        const double* kr = T.kt + size_t(j) * m;
#pragma unroll
        for (int t = 0; t < kFastRowsPerLane; ++t) {
            const int i = lane + 32 * t;
            if (i < m) col[t] += kr[i] * tj;
        }
    }
    double largest = -INFINITY;
    bool any = false;
#pragma unroll
    for (int t = 0; t < kFastRowsPerLane; ++t) {
        const int i = lane + 32 * t;
        if (i < m && !isnan(col[t])) {
            largest = any ? fmax(largest, col[t]) : col[t];
            any = true;
        }
    }
    // The largest non-NaN value over the lanes (Eigen's maxCoeff<PropagateNumbers>).
    largest = warp_max(any ? largest : -INFINITY);
    const bool all_nan = !__any_sync(0xffffffffu, any);
    if (!all_nan && largest > 0.0) {
#pragma unroll
        for (int t = 0; t < kFastRowsPerLane; ++t) col[t] /= largest;
    }
    // Partial sums: G (upper triangle, 10), C^T s (4), norm1 (4).
    double part[18];
#pragma unroll
    for (int k = 0; k < 18; ++k) part[k] = 0.0;
#pragma unroll
    for (int t = 0; t < kFastRowsPerLane; ++t) {
        const int i = lane + 32 * t;
        if (i >= m) continue;
        double v[4];
        v[0] = col[t];
#pragma unroll
        for (int q = 1; q < 4; ++q) v[q] = q <= ci ? T.iso[size_t(i) * ci + q - 1] : 0.0;
        const double si = sig[i];
        int k = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int c = a; c < 4; ++c) part[k++] += v[a] * v[c];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            part[10 + a] += v[a] * si;
            part[14 + a] += fabs(v[a]);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < 18; ++k) part[k] += __shfl_xor_sync(0xffffffffu, part[k], off);
    double G[4][4], b[4], u[4];
    {
        int k = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int c = a; c < 4; ++c) {
                G[a][c] = part[k];
                G[c][a] = part[k];
                ++k;
            }
    }
    double colmax = 0.0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        b[a] = part[10 + a];
        if (a < n) colmax = fmax(colmax, part[14 + a]);
    }
    if (tol < 0.0) tol = 10.0 * kEps64 * colmax * double(max(m, n));
    if (!small_nnls(G, b, n, tol, 3 * n, u)) return false;
    if (lane < n) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q == lane) st.fr[q] = u[q];
    }
    __syncwarp();
    return true;
}

// compute_fractions (cpp/src/sd/fractions.cpp:70-101): tol < 0 uses the default tolerance of the
// fraction columns. Writes the fractions (groups, then isotropic tissues) to st.fr. One
// anisotropic group, at most three isotropic tissues and at most 320 measurements take the
// register fit (fractions_small); otherwise, or when its normal equations are not positive
// definite, the columns are built in the warp's slot and fitted by QR.
__device__ __forceinline__ void fractions(const TissueDev T, const double* fod, const double* sig, bool per_block,
                                          double tol, const FracSlot sl, FracState& st, int lane) {
    const int m = T.m, ca = T.ca, ci = T.ci;
    const double threshold = warp_median(fod, ca, st, lane) * (1.0 - kMedianTie);
    const int ng = per_block ? T.nb : 1;
    const int ncol = ng + ci;
    if (ng == 1 && ci <= 3 && m <= 32 * kFastRowsPerLane) {
        const int gb = per_block ? T.blocks[0] : 0, ge = per_block ? T.blocks[1] : ca;
        if (fractions_small(T, fod, sig, gb, ge, threshold, tol, st, lane)) return;
    }
    for (int j = lane; j < ca; j += 32) sl.th[j] = fod[j] < threshold ? 0.0 : fod[j];
    __syncwarp();
    double colmax = 0.0;
    for (int g = 0; g < ng; ++g) {
        const int b = per_block ? T.blocks[2 * g] : 0, e = per_block ? T.blocks[2 * g + 1] : ca;
        double largest = -INFINITY;
        bool any = false;
        for (int i = lane; i < m; i += 32) {
            double acc = 0.0;
            for (int j = b; j < e; ++j) {
                const double t = sl.th[j];
                if (t != 0.0) acc += T.kt[size_t(j) * m + i] * t;
            }
            sl.cols[size_t(i) * ncol + g] = acc;
            if (!isnan(acc)) {
                largest = any ? fmax(largest, acc) : acc;
                any = true;
            }
        }
        // The largest non-NaN value over the lanes (Eigen's maxCoeff<PropagateNumbers>).
        const bool lane_any = any;
        largest = lane_any ? largest : -INFINITY;
        largest = warp_max(largest);
        const bool all_nan = !__any_sync(0xffffffffu, lane_any);
        __syncwarp();
        if (!all_nan && largest > 0.0)
            for (int i = lane; i < m; i += 32) sl.cols[size_t(i) * ncol + g] /= largest;
        __syncwarp();
    }
    for (int i = lane; i < m; i += 32)
        for (int j = 0; j < ci; ++j) sl.cols[size_t(i) * ncol + ng + j] = T.iso[size_t(i) * ci + j];
    __syncwarp();
    if (tol < 0.0) {
        // 10 eps norm1(C) max(rows, columns) (cpp/src/sd/nnls.cpp:177-181).
        for (int g = 0; g < ncol; ++g) {
            double sum = 0.0;
            for (int i = lane; i < m; i += 32) sum += fabs(sl.cols[size_t(i) * ncol + g]);
            colmax = fmax(colmax, warp_sum(sum));
        }
        tol = 10.0 * kEps64 * colmax * double(max(m, ncol));
    }
    NnlsScratch ns{sl.fu, sl.fz, sl.fflag, st.fact, &st.fn_act, sl.res,
                   QrScratch{sl.fsub, st.ftau, st.fnu, st.fnd, st.fperm, sl.frv}, kMaxGroups};
    warp_nnls_explicit(sl.cols, m, ncol, sig, tol, 3 * ncol, ns, lane);
    for (int g = lane; g < ncol; g += 32) st.fr[g] = sl.fu[g];
    __syncwarp();
}

// ---- fractions, a lane per voxel (low-resolution NNLS solutions) ----------------------------------
//
// A round's fractions need of the column K th only its maximum, its sum and its products with itself,
// the isotropic columns and the signal. A non-negative K gives all but the first from small
// constants, (th, K^T K th), (K^T iso)^T th and (K^T s)^T th, sums of non-negative terms; K^T s and
// iso^T s do not change over the rounds and are taken once per fit. The maximum needs only the rows of K
// that no other row bounds entry by entry (with a b0 among the measurements, that one row), and is
// the same number, as the order of a row's sum is. Solutions have ~8 of 44 entries, so their median is 0 (else,
// or for values that are not finite and non-negative, the warp takes the voxel by the general way).
// So a voxel is ~200 FMAs on one lane, where a warp ranked 44 entries, built 280 rows and reduced
// 18 sums: 28.1 ms for ten
// rounds of 250,000 voxels, 2.0 ms for 8,191; now 3.4 and 1.9 ms (the latency of a lane's chain)

constexpr int kFracCols = 48, kFracRows = 16, kFracList = 24, kFracWarps = 4;
static_assert(kFracList >= kFracCols - kFracCols / 2 - 1, "the list holds every solution with median 0");

// The constants of one kernel, packed: K^T K (c, c), K^T iso (c, ci), the column sums (c), the rows
// that can hold the maximum (rows, c), iso^T iso (ci, ci), the isotropic columns' absolute sums (ci).
struct FracConstants {
    const double *gram, *ki, *ksum, *top, *ii, *isum;
    __host__ __device__ FracConstants(const double* p, int c, int ci, int rows) {
        gram = p;
        ki = gram + c * c;
        ksum = ki + c * ci;
        top = ksum + c;
        ii = top + rows * c;
        isum = ii + ci * ci;
    }
    __host__ __device__ static int doubles(int c, int ci, int rows) {
        return c * c + c * ci + c + rows * c + ci * ci + ci;
    }
};

inline size_t frac_lane_smem(int doubles) {
    return size_t(doubles) * sizeof(double) + size_t(kFracWarps) * 32 * kFracList * (sizeof(double) + 1);
}

// The fractions u of the solution x (c) with ks = [K^T s, iso^T s]; false when the general way is needed.
__device__ __forceinline__ bool lane_fractions(const FracConstants& F, int m, int c, int ci, int rows,
                                               const double* __restrict__ x, const double* __restrict__ ks,
                                               double* vals, uint8_t* cols, double (&u)[4]) {
    // The lane's list: entry q at [32 q].
    int n = 0;
    bool odd = false;
    for (int j0 = 0; j0 < c; j0 += 8) {
        double some[8];  // loaded together: each is its own trip to L2
#pragma unroll
        for (int q = 0; q < 8; ++q) some[q] = j0 + q < c ? x[j0 + q] : 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double v = some[q];
            if (v == 0.0) continue;
            odd |= !(v > 0.0 && v < INFINITY);
            if (n < kFracList) {
                vals[32 * n] = v;
                cols[32 * n] = uint8_t(j0 + q);
            }
            ++n;
        }
    }
    if (odd || c - n <= c / 2) return false;
    double largest = -INFINITY;
    for (int r = 0; r < rows; ++r) {
        double s = 0.0;
        for (int q = 0; q < n; ++q) s = fma(F.top[r * c + cols[32 * q]], vals[32 * q], s);
        largest = fmax(largest, s);
    }
    double cc = 0.0, cs = 0.0, sum = 0.0, ct[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
    for (int q = 0; q < n; ++q) cs = fma(vals[32 * q], ks[cols[32 * q]], cs);
    for (int q = 0; q < n; ++q) {
        const double v = vals[32 * q];
        const int j = cols[32 * q];
        const double* row = F.gram + j * c;
        double s = 0.0;
        for (int p = 0; p < q; ++p) s = fma(row[cols[32 * p]], vals[32 * p], s);
        cc = fma(v, fma(2.0, s, row[j] * v), cc);
        sum = fma(v, F.ksum[j], sum);
#pragma unroll
        for (int t = 0; t < 3; ++t)
            if (t < ci) ct[t] = fma(v, F.ki[j * ci + t], ct[t]);
    }
    if (largest > 0.0) {
        cc = cc / largest / largest;
        cs /= largest;
        sum /= largest;
#pragma unroll
        for (int t = 0; t < 3; ++t) ct[t] /= largest;
    }
    double G[4][4], b[4], norm1 = sum;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        b[a] = a == 0 ? cs : a <= ci ? ks[c + a - 1] : 0.0;
        if (a > 0 && a <= ci) norm1 = fmax(norm1, F.isum[a - 1]);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            if (a == 0 || d == 0)
                G[a][d] = a + d == 0 ? cc : ct[a + d > 3 ? 2 : a + d - 1];
            else
                G[a][d] = a <= ci && d <= ci ? F.ii[(a - 1) * ci + d - 1] : 0.0;
        }
    }
    return small_nnls(G, b, 1 + ci, 10.0 * kEps64 * norm1 * double(max(m, 1 + ci)), 3 * (1 + ci), u);
}

// A round's state of one volume, as the fraction kernels update it.
struct FracRound {
    const double* s;       // (v, m) signals
    const double* x;       // (v, ldx) low-resolution solutions
    const double* ks;      // (v, c + ci)
    double *fiso, *prev;   // (v, ci), (v, ci + 1)
    int32_t* rounds;
    int* next;             // the next round's list and its count
    int* next_count;
    int ldx, round, max_rounds;
    double tol;
};

// The general way, out of line: its registers stay out of the lane-per-voxel kernels.
__device__ __noinline__ void fractions_by_warp(const TissueDev& T, const double* fod, const double* sig,
                                               const FracSlot& sl, FracState& st, int lane) {
    fractions(T, fod, sig, false, -1.0, sl, st, lane);
}

// One warp's voxels, one per lane (-1: none): fractions, the convergence test and the next list
// (lr_fractions_kernel).
__device__ __forceinline__ void lane_fractions_unit(const TissueDev& T, const FracConstants& F, const FracRound& R,
                                                    int64_t voxel, double* vals, uint8_t* cols, const FracSlot& sl,
                                                    FracState& st, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    const int c = T.ca, ci = T.ci;
    double u[4] = {0.0, 0.0, 0.0, 0.0};
    bool ok = true;
    if (voxel >= 0)
        ok = lane_fractions(F, T.m, c, ci, T.fx_rows, R.x + voxel * R.ldx, R.ks + voxel * (c + ci), vals, cols, u);
    __syncwarp();
    for (unsigned left = __ballot_sync(kAll, !ok); left; left &= left - 1u) {
        const int who = __ffs(left) - 1;
        const int64_t w = __shfl_sync(kAll, voxel, who);
        fractions_by_warp(T, R.x + w * R.ldx, R.s + w * T.m, sl, st, lane);
        if (lane == who) {
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = j <= ci ? st.fr[j] : 0.0;
        }
        __syncwarp();
    }
    bool goes_on = false;
    if (voxel >= 0) {
        // The first round has nothing to compare with (its previous fractions are infinite).
        bool converged = R.round > 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j > ci) continue;
            double& before = R.prev[voxel * (ci + 1) + j];
            if (R.round > 0) converged &= fabs(u[j] - before) < R.tol;
            before = u[j];
            if (j > 0) R.fiso[voxel * ci + j - 1] = u[j];
        }
        goes_on = !converged && R.round + 1 < R.max_rounds;
        if (!goes_on) R.rounds[voxel] = R.round + 1;
    }
    const unsigned on = __ballot_sync(kAll, goes_on);
    if (on) {
        int base = 0;
        if (lane == 0) base = atomicAdd(R.next_count, __popc(on));
        base = __shfl_sync(kAll, base, 0);
        if (goes_on) R.next[base + __popc(on & ((1u << lane) - 1u))] = int(voxel);
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kFracWarps * 32) lane_fractions_kernel(
    TissueDev T, FracRound R, const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev,
    double* __restrict__ workspace, size_t slot_size) {
    if (count_dev) count = min(count, int64_t(*count_dev));
    if (count <= int64_t(blockIdx.x) * 32) return;
    extern __shared__ __align__(16) double fsm[];
    __shared__ FracState states[kFracWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = FracConstants::doubles(T.ca, T.ci, T.fx_rows);
    for (int i = threadIdx.x; i < n; i += blockDim.x) fsm[i] = T.fx[i];
    __syncthreads();
    const FracConstants F(fsm, T.ca, T.ci, T.fx_rows);
    double* vals = fsm + n + warp * 32 * kFracList + lane;
    uint8_t* cols = reinterpret_cast<uint8_t*>(fsm + n + kFracWarps * 32 * kFracList) + warp * 32 * kFracList + lane;
    const FracSlot sl =
        carve_frac(workspace + (size_t(blockIdx.x) * kFracWarps + warp) * slot_size, T.m, T.ca, 1 + T.ci);
    // Units of 32 voxels dealt to the CTAs first (a grid of a CTA per four units of the whole call: a later round's
    // shorter list has a CTA for each of its own).
    for (int64_t p0 = (blockIdx.x + int64_t(gridDim.x) * warp) * 32; p0 < count;
         p0 += int64_t(gridDim.x) * kFracWarps * 32)
        lane_fractions_unit(T, F, R, p0 + lane < count ? listed(list, p0 + lane) : -1, vals, cols, sl, states[warp],
                            lane);
}

// One round's fractions of the listed voxels (cpp/src/sd/multi_tissue.cpp:100-125): f_iso(v)
// takes the isotropic fractions; a voxel whose fractions all moved by less than fraction_tol, or
// that used its last round, records its round count, the others join the next round's list
// with their fractions kept for the next comparison.
__global__ void __launch_bounds__(kMtWarps * 32, 5) lr_fractions_kernel(
    TissueDev T, const double* __restrict__ signals, const double* __restrict__ fods, int ldf,
    const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev, int round, int max_rounds,
    double fraction_tol, double* __restrict__ fiso, double* __restrict__ prev, int32_t* __restrict__ rounds,
    int* __restrict__ next, int* next_count, int* queue, double* __restrict__ workspace, size_t slot_size) {
    if (count_dev) count = min(count, int64_t(*count_dev));
    __shared__ FracState states[kMtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FracState& st = states[warp];
    FracSlot sl = carve_frac(workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size, T.m, T.ca, 1 + T.ci);
    const int ci = T.ci;
    for (;;) {
        int64_t p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= count) break;
        const int64_t voxel = listed(list, p);
        fractions(T, fods + voxel * ldf, signals + voxel * T.m, false, -1.0, sl, st, lane);
        // The first round has nothing to compare with (its previous fractions are infinite).
        bool converged = round > 0;
        for (int j = 0; j <= ci; ++j) converged &= fabs(st.fr[j] - prev[voxel * (ci + 1) + j]) < fraction_tol;
        __syncwarp();
        if (lane < ci) fiso[voxel * ci + lane] = st.fr[1 + lane];
        if (converged || round + 1 >= max_rounds) {
            if (lane == 0) rounds[voxel] = round + 1;
        } else {
            if (lane <= ci) prev[voxel * (ci + 1) + lane] = st.fr[lane];
            if (lane == 0) next[atomicAdd(next_count, 1)] = int(voxel);
        }
        __syncwarp();
    }
}

// The final per-block fractions of every voxel, normalised to sum to 1 (+1e-16), with the round
// counts and statuses (cpp/src/sd/multi_tissue.cpp:127-148).
__global__ void __launch_bounds__(kMtWarps * 32, 5) hr_fractions_kernel(
    TissueDev T, const double* __restrict__ signals, const double* __restrict__ fods, int64_t count,
    double final_tol, const int32_t* __restrict__ rounds_in, const uint8_t* __restrict__ bad,
    double* __restrict__ fractions_out, int32_t* __restrict__ rounds_out, uint8_t* __restrict__ status, int* queue,
    double* __restrict__ workspace, size_t slot_size) {
    __shared__ FracState states[kMtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FracState& st = states[warp];
    FracSlot sl = carve_frac(workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size, T.m, T.ca,
                             T.nb + T.ci);
    const int nf = T.nb + T.ci;
    for (;;) {
        int64_t voxel = 0;
        if (lane == 0) voxel = atomicAdd(queue, 1);
        voxel = __shfl_sync(0xffffffffu, voxel, 0);
        if (voxel >= count) break;
        fractions(T, fods + voxel * T.ca, signals + voxel * T.m, true, final_tol, sl, st, lane);
        double total = kFractionSumOffset;
        for (int g = 0; g < nf; ++g) total += st.fr[g];
        for (int g = lane; g < nf; g += 32) fractions_out[voxel * nf + g] = st.fr[g] / total;
        if (lane == 0) {
            if (rounds_out) rounds_out[voxel] = rounds_in[voxel];
            if (status) status[voxel] = bad[voxel];
        }
        __syncwarp();
    }
}

// ---- batches (batch.cuh): every mFOD volume of a batch through one queue per stage ------------

constexpr int kLowTicket = 256;  // voxels of a ticket of the low-resolution NNLS

// A volume of a batch: its solvers and kernels, signals, shell weights and outputs.
struct MfodBatchJob {
    int64_t v, off;  // voxels; the row of its first voxel in the batch's per-voxel state
    RidgeDev lr, hr;
    TissueDev lrt, hrt;
    const double* s;   // (v, m) S0-normalised signals
    const double* w;   // (m,) shell weights
    const double* kx;  // [K, iso] of the low-resolution kernel, unweighted (m, ca + ci), where lrt.fx is set
    int64_t ks_off;    // its first double in the batch's ks
    double* fods;      // (v, hr.c)
    double* fractions; // (v, hrt.nb + hrt.ci)
    int32_t* rounds;   // (v,) or null
    uint8_t* status;   // (v,) or null
};

// The per-voxel state of a batch (volume j's voxel v at row off_j + v) and the stage's tickets.
struct MfodBatchState {
    const MfodBatchJob* jobs;
    int n_jobs, ci, ldc, ldx;  // isotropic tissues; row strides of corr and of the low-resolution FODs
    double *fiso, *prev, *corr, *xlr, *ks;
    int32_t* rounds;
    uint8_t* bad;
    int64_t* vfirst;   // (n_jobs + 1) this stage's first voxel ticket per volume
    int64_t* tfirst;   // (n_jobs + 1) its first correlation tile per volume
    int64_t* qfirst;   // (n_jobs + 1) its first ticket of kLowTicket voxels per volume
    int64_t* cfirst;   // (n_jobs + 1) its first ticket of kCorrTcTicket voxels per volume
    int64_t* redo;     // volume << 32 | voxel, for the one-warp NNLS
    int* redo_count;
};

// A round's lists are per-volume segments of one array (volume j's at row off_j), null for
// every voxel of every volume.
struct BatchItem {
    int job;
    int64_t voxel;
};

__device__ __forceinline__ BatchItem batch_item(const MfodBatchState& B, const int* list, int64_t p) {
    const int j = ticket_job(B.vfirst, B.n_jobs, p);
    const int64_t q = p - B.vfirst[j];
    return BatchItem{j, list ? int64_t(list[B.jobs[j].off + q]) : q};
}

__device__ __forceinline__ SignalDev batch_signal(const MfodBatchState& B, const MfodBatchJob& J, const TissueDev& T) {
    return SignalDev{J.s, J.w, T.wiso, B.fiso + J.off * B.ci, T.m, B.ci};
}

// The tickets of a stage from each volume's count (null: every voxel).
__global__ void batch_plan_kernel(MfodBatchState B, const int* __restrict__ counts) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int64_t a = 0, b = 0, q = 0, e = 0;
    for (int j = 0; j < B.n_jobs; ++j) {
        B.vfirst[j] = a;
        B.tfirst[j] = b;
        B.qfirst[j] = q;
        B.cfirst[j] = e;
        const int64_t c = counts ? int64_t(counts[j]) : B.jobs[j].v;
        a += c;
        b += (c + kCorrVoxels - 1) / kCorrVoxels;
        q += (c + kLowTicket - 1) / kLowTicket;
        e += (c + kCorrTcTicket - 1) / kCorrTcTicket;
    }
    B.vfirst[B.n_jobs] = a;
    B.tfirst[B.n_jobs] = b;
    B.qfirst[B.n_jobs] = q;
    B.cfirst[B.n_jobs] = e;
}

// correlate_kernel over the volumes that do not fit correlate_tc_kernel: a CTA per (volume, tile of
// kCorrVoxels listed voxels).
template <int RC, bool HR>
__global__ void __launch_bounds__(128) batch_correlate_kernel(MfodBatchState B, const int* __restrict__ list) {
    __shared__ int64_t vox[kCorrVoxels];
    const int tid = threadIdx.x;
    const int64_t total = B.tfirst[B.n_jobs];
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = ticket_job(B.tfirst, B.n_jobs, t);
        const MfodBatchJob& J = B.jobs[j];
        const RidgeDev R = HR ? J.hr : J.lr;
        if (corr_tc_fits(R.m, B.ci)) continue;
        const int64_t count = B.vfirst[j + 1] - B.vfirst[j];
        const int64_t p0 = (t - B.tfirst[j]) * kCorrVoxels;
        __syncthreads();  // the previous tile's voxels are read
        if (tid < kCorrVoxels) {
            const int64_t q = p0 + tid;
            vox[tid] = q < count ? (list ? int64_t(list[J.off + q]) : q) : -1;
        }
        __syncthreads();
        const TissueDev T = HR ? J.hrt : J.lrt;
        correlate_tile<RC>(batch_signal(B, J, T), vox, R.k, R.c, blockIdx.y * 16 * RC, B.corr + J.off * B.ldc,
                           B.ldc);
    }
}

// correlate_tc_kernel over every volume: a CTA takes a ticket of kCorrTcTicket listed voxels, eight to
// a warp, and restages when its ticket moves to another volume.
template <int CI, bool HR>
__global__ void __launch_bounds__(kCorrTcWarps * 32, 1) batch_correlate_tc_kernel(MfodBatchState B,
                                                                                 const int* __restrict__ list) {
    extern __shared__ __align__(16) double csm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col0 = blockIdx.y * kCorrTcCols;
    const int64_t total = B.cfirst[B.n_jobs];
    int cur = -1;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = ticket_job(B.cfirst, B.n_jobs, t);
        const MfodBatchJob& J = B.jobs[j];
        const RidgeDev R = HR ? J.hr : J.lr;
        if (!corr_tc_fits(R.m, CI) || col0 >= R.c) continue;
        const SignalDev S = batch_signal(B, J, HR ? J.hrt : J.lrt);
        if (j != cur) {
            __syncthreads();
            corr_tc_stage(csm, S, R.k, R.c, col0);
            cur = j;
            __syncthreads();
        }
        const int64_t p = (t - B.cfirst[j]) * kCorrTcTicket + warp * kCorrTcUnit + (lane >> 2);
        const int64_t count = B.vfirst[j + 1] - B.vfirst[j];
        const int64_t voxel = p < count ? (list ? int64_t(list[J.off + p]) : p) : -1;
        corr_tc_unit<CI>(csm, S, voxel, R.c, col0, B.corr + J.off * B.ldc, B.ldc, lane);
    }
}

// ridge_nnls_low_kernel over every volume's list: a CTA takes a ticket of kLowTicket listed voxels of
// one volume, whose Gram matrix it keeps until its ticket moves to another.
__global__ void __launch_bounds__(kLowWarps * 32, 2) batch_low_kernel(MfodBatchState B, const int* __restrict__ list,
                                                                     int* queue) {
    extern __shared__ __align__(16) double lsm[];
    __shared__ int ticket, taken;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LeanWarp q(lsm + warp * kLeanWarpDoubles);
    double* const gs = lsm + kLowWarps * kLeanWarpDoubles;
    const int64_t total = B.qfirst[B.n_jobs];
    int cur = -1;
    for (;;) {
        __syncthreads();  // every warp is done with the last ticket
        if (threadIdx.x == 0) {
            ticket = atomicAdd(queue, 1);
            taken = 0;
        }
        __syncthreads();
        const int64_t t = ticket;
        if (t >= total) break;
        const int j = ticket_job(B.qfirst, B.n_jobs, t);
        const MfodBatchJob& J = B.jobs[j];
        const RidgeDev R = J.lr;
        if (j != cur) {
            stage_gram(gs, R);
            cur = j;
            __syncthreads();
        }
        const int64_t p0 = (t - B.qfirst[j]) * kLowTicket;
        const int64_t count = min(int64_t(kLowTicket), B.vfirst[j + 1] - B.vfirst[j] - p0);
        for (;;) {
            int p = 0;
            if (lane == 0) p = atomicAdd(&taken, 1);
            p = __shfl_sync(0xffffffffu, p, 0);
            if (p >= count) break;
            const int64_t voxel = list ? int64_t(list[J.off + p0 + p]) : p0 + p, row = J.off + voxel;
            if (!lean_nnls<2>(gs, R.c, R.c, R.tol, kMinPivot, B.corr + row * B.ldc, q, B.xlr + row * B.ldx, lane) &&
                lane == 0)
                B.redo[atomicAdd(B.redo_count, 1)] = (int64_t(j) << 32) | voxel;
            __syncwarp();
        }
    }
}

// ridge_nnls_kernel over the voxels the first passes handed back, from every volume.
template <int VPL, int CPL, bool HR>
__global__ void __launch_bounds__(kMtWarps * 32, (CPL <= 2 ? 6 : 4)) batch_redo_kernel(
    MfodBatchState B, int c_max, int* queue, double* __restrict__ workspace, size_t slot_size) {
    using State = NnlsState<VPL * 32, CPL * 32>;
    __shared__ State states[kMtWarps];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    State& st = states[warp];
    double* slot = workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size;
    unsigned char* wsm = smem_raw + warp * nnls_smem_bytes(c_max, VPL * 32);
    const int total = *B.redo_count;
    for (;;) {
        int p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= total) break;
        const int64_t e = B.redo[p];
        const MfodBatchJob& J = B.jobs[int(e >> 32)];
        const int64_t voxel = e & 0xffffffffll;
        const RidgeDev R = HR ? J.hr : J.lr;
        const TissueDev T = HR ? J.hrt : J.lrt;
        NnlsSlot sl = carve_nnls(slot, wsm, R.m, R.c, VPL * 32);
        const int64_t row = J.off + voxel;
        const bool ok = ridge_nnls<VPL, CPL>(R, batch_signal(B, J, T), voxel, B.corr + row * B.ldc, sl, st, lane);
        double* x = HR ? J.fods + voxel * R.c : B.xlr + row * B.ldx;
        for (int j = lane; j < R.c; j += 32) x[j] = sl.x[j];
        if (lane == 0 && !ok) B.bad[row] = 1;
        __syncwarp();
    }
}

// ridge_nnls_high_kernel over every voxel of every volume.
__global__ void __launch_bounds__(kHighWarps * 32, kHighCtas) batch_high_kernel(MfodBatchState B, int* queue) {
    extern __shared__ __align__(16) double lsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LeanWarp q(lsm + warp * kLeanWarpDoubles);
    const int64_t total = B.vfirst[B.n_jobs];
    for (;;) {
        long long p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= total) break;
        const BatchItem it = batch_item(B, nullptr, p);
        const MfodBatchJob& J = B.jobs[it.job];
        const RidgeDev R = J.hr;
        if (!lean_nnls<10>(R.gram, R.c, R.c, R.tol, kMinPivot, B.corr + (J.off + it.voxel) * B.ldc, q,
                           J.fods + it.voxel * R.c, lane) &&
            lane == 0)
            B.redo[atomicAdd(B.redo_count, 1)] = (int64_t(it.job) << 32) | it.voxel;
        __syncwarp();
    }
}

// [K^T s, iso^T s] of every voxel of the volumes whose fractions take a lane per voxel, once per fit.
__global__ void __launch_bounds__(kCorrTcWarps * 32, 1) batch_ks_kernel(MfodBatchState B) {
    extern __shared__ __align__(16) double csm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col0 = blockIdx.y * kCorrTcCols;
    const int64_t total = B.cfirst[B.n_jobs];
    int cur = -1;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = ticket_job(B.cfirst, B.n_jobs, t);
        const MfodBatchJob& J = B.jobs[j];
        const int c = J.lrt.ca + J.lrt.ci;
        if (J.lrt.fx == nullptr || col0 >= c) continue;
        const SignalDev S{J.s, nullptr, nullptr, nullptr, J.lrt.m, 0};
        if (j != cur) {
            __syncthreads();
            corr_tc_stage(csm, S, J.kx, c, col0);
            cur = j;
            __syncthreads();
        }
        const int64_t p = (t - B.cfirst[j]) * kCorrTcTicket + warp * kCorrTcUnit + (lane >> 2);
        corr_tc_unit<-1>(csm, S, p < J.v ? p : -1, c, col0, B.ks + J.ks_off, c, lane);
    }
}

// lane_fractions_kernel over those volumes' lists: a CTA takes a ticket of kLowTicket listed voxels.
__global__ void __launch_bounds__(kFracWarps * 32) batch_lane_fractions_kernel(
    MfodBatchState B, int doubles, const int* __restrict__ list, int round, int max_rounds, double fraction_tol,
    int* __restrict__ next, int* next_counts, double* __restrict__ workspace, size_t slot_size) {
    extern __shared__ __align__(16) double fsm[];
    __shared__ FracState states[kFracWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ci = B.ci;
    double* vals = fsm + doubles + warp * 32 * kFracList + lane;
    uint8_t* cols =
        reinterpret_cast<uint8_t*>(fsm + doubles + kFracWarps * 32 * kFracList) + warp * 32 * kFracList + lane;
    double* slot = workspace + (size_t(blockIdx.x) * kFracWarps + warp) * slot_size;
    const int64_t total = B.qfirst[B.n_jobs];
    int cur = -1;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int j = ticket_job(B.qfirst, B.n_jobs, t);
        const MfodBatchJob& J = B.jobs[j];
        const TissueDev T = J.lrt;
        if (T.fx == nullptr) continue;
        if (j != cur) {
            __syncthreads();
            const int n = FracConstants::doubles(T.ca, T.ci, T.fx_rows);
            for (int i = threadIdx.x; i < n; i += blockDim.x) fsm[i] = T.fx[i];
            cur = j;
            __syncthreads();
        }
        const FracConstants F(fsm, T.ca, T.ci, T.fx_rows);
        const FracSlot sl = carve_frac(slot, T.m, T.ca, 1 + ci);
        const FracRound R{J.s, B.xlr + J.off * B.ldx, B.ks + J.ks_off, B.fiso + J.off * ci,
                          B.prev + J.off * (ci + 1), B.rounds + J.off, next + J.off, next_counts + j, B.ldx, round,
                          max_rounds, fraction_tol};
        const int64_t p0 = (t - B.qfirst[j]) * kLowTicket;
        const int64_t count = min(int64_t(kLowTicket), B.vfirst[j + 1] - B.vfirst[j] - p0);
        for (int64_t q = warp * 32; q < count; q += kFracWarps * 32) {
            const int64_t p = p0 + q + lane;
            const int64_t voxel = q + lane < count ? (list ? int64_t(list[J.off + p]) : p) : -1;
            lane_fractions_unit(T, F, R, voxel, vals, cols, sl, states[warp], lane);
        }
    }
}

// lr_fractions_kernel over every volume's list; the next round's list goes to each volume's
// segment.
__global__ void __launch_bounds__(kMtWarps * 32, 4) batch_lr_fractions_kernel(
    MfodBatchState B, const int* __restrict__ list, int round, int max_rounds, double fraction_tol,
    int* __restrict__ next, int* next_counts, int* queue, double* __restrict__ workspace, size_t slot_size) {
    __shared__ FracState states[kMtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FracState& st = states[warp];
    double* slot = workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size;
    const int ci = B.ci;
    const int64_t total = B.vfirst[B.n_jobs];
    for (;;) {
        long long p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= total) break;
        const BatchItem it = batch_item(B, list, p);
        const MfodBatchJob& J = B.jobs[it.job];
        const TissueDev T = J.lrt;
        if (T.fx != nullptr) continue;  // batch_lane_fractions_kernel's
        const FracSlot sl = carve_frac(slot, T.m, T.ca, 1 + T.ci);
        const int64_t row = J.off + it.voxel;
        fractions(T, B.xlr + row * B.ldx, J.s + it.voxel * T.m, false, -1.0, sl, st, lane);
        bool converged = round > 0;
        for (int j = 0; j <= ci; ++j) converged &= fabs(st.fr[j] - B.prev[row * (ci + 1) + j]) < fraction_tol;
        __syncwarp();
        if (lane < ci) B.fiso[row * ci + lane] = st.fr[1 + lane];
        if (converged || round + 1 >= max_rounds) {
            if (lane == 0) B.rounds[row] = round + 1;
        } else {
            if (lane <= ci) B.prev[row * (ci + 1) + lane] = st.fr[lane];
            if (lane == 0) next[J.off + atomicAdd(next_counts + it.job, 1)] = int(it.voxel);
        }
        __syncwarp();
    }
}

// hr_fractions_kernel over every voxel of every volume.
__global__ void __launch_bounds__(kMtWarps * 32, 4) batch_hr_fractions_kernel(MfodBatchState B, double final_tol,
                                                                             int* queue,
                                                                             double* __restrict__ workspace,
                                                                             size_t slot_size) {
    __shared__ FracState states[kMtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FracState& st = states[warp];
    double* slot = workspace + (size_t(blockIdx.x) * kMtWarps + warp) * slot_size;
    const int64_t total = B.vfirst[B.n_jobs];
    for (;;) {
        long long p = 0;
        if (lane == 0) p = atomicAdd(queue, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= total) break;
        const BatchItem it = batch_item(B, nullptr, p);
        const MfodBatchJob& J = B.jobs[it.job];
        const TissueDev T = J.hrt;
        const int nf = T.nb + T.ci;
        const FracSlot sl = carve_frac(slot, T.m, T.ca, nf);
        const int64_t row = J.off + it.voxel;
        fractions(T, J.fods + it.voxel * T.ca, J.s + it.voxel * T.m, true, final_tol, sl, st, lane);
        double sum = kFractionSumOffset;
        for (int g = 0; g < nf; ++g) sum += st.fr[g];
        for (int g = lane; g < nf; g += 32) J.fractions[it.voxel * nf + g] = st.fr[g] / sum;
        if (lane == 0) {
            if (J.rounds) J.rounds[it.voxel] = B.rounds[row];
            if (J.status) J.status[it.voxel] = B.bad[row];
        }
        __syncwarp();
    }
}

// ---- host side -------------------------------------------------------------------------

// The warps of a persistent grid: as many as the SMs hold at once (or one per item), in whole
// CTAs of `warps`.
template <class Kernel>
int64_t resident_slots(Kernel kernel, size_t smem, int64_t items, const char* setting, int warps = kMtWarps) {
    require(smem <= 200 * 1024, "the kernel has too many columns for the shared-memory solver");
    allow_smem(kernel, smem);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((items + warps - 1) / warps,
                                                                  int64_t(sm_count()) * ctas_per_sm(per_sm, setting)));
    return blocks * warps;
}

// A bump allocator over one device buffer, 256-byte aligned pieces.
struct Carver {
    char* base;
    size_t used = 0;
    template <class T>
    T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base ? base + used : nullptr);
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
};

// Launches the ridge NNLS of `count` listed voxels on the instantiation that fits the solver.
struct NnlsLaunch {
    void (*kernel)(RidgeDev, SignalDev, const int*, int64_t, const int*, const double*, int, double*, int, uint8_t*,
                   int*, double*, size_t);
    int cap;
    const char* name;
};

inline NnlsLaunch nnls_variant(int c) {
    // Up to 64 directions (the low-resolution kernels): a 32-column factor, the active sets
    // being far smaller (past 32 active columns the fit continues by QR).
    if (c <= 64) return {ridge_nnls_kernel<1, 2>, 32, "ridge_nnls_kernel<1,2>"};
    if (c <= 320) return {ridge_nnls_kernel<kCholCap / 32, 10>, kCholCap, "ridge_nnls_kernel<8,10>"};
    return {ridge_nnls_kernel<kCholCap / 32, kMaxColumns / 32>, kCholCap, "ridge_nnls_kernel<8,20>"};
}

inline void launch_correlate(const SignalDev& S, const int* list, int64_t count, const int* count_dev,
                             const RidgeDev& R, double* corr, int ldc, cudaStream_t st) {
    if (count == 0) return;
    if (corr_tc_fits(R.m, S.w ? S.ci : 0)) {
        const unsigned gy = unsigned((R.c + kCorrTcCols - 1) / kCorrTcCols);
        const int64_t units = (count + kCorrTcUnit - 1) / kCorrTcUnit;
        const unsigned gx = unsigned(std::max<int64_t>(1, std::min<int64_t>(units, sm_count() / gy)));
        const size_t smem = corr_tc_smem(R.m, S.w ? S.ci : 0);
        auto run = [&](auto kernel) {
            allow_smem(kernel, smem);
            LaunchScope scope("correlate_kernel", st);
            kernel<<<dim3(gx, gy), kCorrTcWarps * 32, smem, st>>>(S, list, count, count_dev, R.k, R.c, corr, ldc);
            cuda_check(cudaGetLastError(), "correlate_tc_kernel launch");
        };
        if (S.w == nullptr) run(correlate_tc_kernel<-1>);
        else if (S.ci == 0) run(correlate_tc_kernel<0>);
        else if (S.ci == 1) run(correlate_tc_kernel<1>);
        else if (S.ci == 2) run(correlate_tc_kernel<2>);
        else run(correlate_tc_kernel<3>);
        return;
    }
    // count is exact unless the round's count lives on the device (count_dev): then it is an
    // upper bound and the grid stays resident-sized, the CTAs striding over the live tiles.
    int64_t tiles = (count + kCorrVoxels - 1) / kCorrVoxels;
    if (count_dev) tiles = std::min<int64_t>(tiles, int64_t(sm_count()) * kCorrResidentCtas);
    const unsigned gx = unsigned(tiles);
    LaunchScope scope("correlate_kernel", st);
    if (R.c <= 48) {
        correlate_kernel<3><<<dim3(gx, 1), 128, 0, st>>>(S, list, count, count_dev, R.k, R.c, corr, ldc);
    } else {
        correlate_kernel<4><<<dim3(gx, unsigned((R.c + 63) / 64)), 128, 0, st>>>(S, list, count, count_dev, R.k, R.c,
                                                                                 corr, ldc);
    }
    cuda_check(cudaGetLastError(), "correlate_kernel launch");
}

// lsqnonneg (cpp/src/python/sd.cpp:208-228): one warp solves min ||c x - d|| over x >= 0 for c
// (m, n) row-major by the fraction fits' Lawson-Hanson with QR fits (cpp/src/sd/nnls.cpp:187-258),
// at most 3 n inner steps. default_tol: tol = 10 eps norm1(c) max(m, n) (nnls.cpp:177-181).
__global__ void __launch_bounds__(32) lsqnonneg_kernel(const double* __restrict__ c, int m, int n,
                                                       const double* __restrict__ d, bool default_tol, double tol,
                                                       double* __restrict__ x, double* __restrict__ workspace) {
    __shared__ FracState st;
    const int lane = threadIdx.x;
    const FracSlot sl = carve_frac(workspace, m, 0, n);
    if (default_tol) {
        double colmax = 0.0;
        for (int g = 0; g < n; ++g) {
            double sum = 0.0;
            for (int i = lane; i < m; i += 32) sum += fabs(c[size_t(i) * n + g]);
            colmax = fmax(colmax, warp_sum(sum));
        }
        tol = 10.0 * kEps64 * colmax * double(max(m, n));
    }
    NnlsScratch ns{sl.fu, sl.fz, sl.fflag, st.fact, &st.fn_act, sl.res,
                   QrScratch{sl.fsub, st.ftau, st.fnu, st.fnd, st.fperm, sl.frv}, kMaxGroups};
    warp_nnls_explicit(c, m, n, d, tol, 3 * n, ns, lane);
    for (int g = lane; g < n; g += 32) x[g] = sl.fu[g];
}

}  // namespace

}  // namespace lar

namespace lar {
// A device FP32 copy of an FP64 host array (rounded to nearest).
inline void upload_fp32(DeviceArray<float>& dst, const std::vector<double>& src) {
    std::vector<float> f(src.begin(), src.end());
    dst.upload(f.data(), f.size());
}
}  // namespace lar

// FodSolver.l2nnls (cpp/src/python/sd.cpp:89-102, cpp/src/sd/solver.cpp:464-467).
struct lar_fod_solver_s {
    // 0: the ridge NNLS (L2NNLS) with its design below; 1: damped Richardson-Lucy (dRL).
    int kind = 0;
    lar::DeviceArray<double> drl_kt, drl_gram;
    lar::DeviceArray<float> drl_gtc;  // K^T K for the tensor-core dRL (precision LAR_TF32X3)
    lar::DeviceArray<int> drl_err;    // where the tensor-core dRL records a wait that ran out
    lar::DrlDev drl{};
    lar::host::RidgeDesignHost host;
    double tol = 0.0;
    lar::DeviceArray<double> k, gram;
    lar::DeviceArray<float> k32, gram32;  // FP32 copies for the plain single-precision fit
    void* scratch = nullptr;
    size_t scratch_bytes = 0;
    int* pinned = nullptr;  // one host int the round loop reads the next round's count into
    ~lar_fod_solver_s() {
        if (scratch) cudaFree(scratch);
        if (pinned) cudaFreeHost(pinned);
    }
    int* count_buffer() {
        if (!pinned) lar::cuda_check(cudaMallocHost(&pinned, sizeof(int)), "cudaMallocHost");
        return pinned;
    }
    // The shell weights on the device, uploaded when they differ from the last call's. Under
    // stream capture nothing may be uploaded, so they must match an earlier uncaptured call.
    std::vector<double> weights_host;
    lar::DeviceArray<double> weights_dev;
    const double* device_weights(const double* w, int64_t m, bool capturing) {
        if (weights_host.size() != size_t(m) || !std::equal(w, w + m, weights_host.begin())) {
            lar::require(!capturing, "under stream capture the weights must be those of an earlier uncaptured "
                                     "call with this solver");
            weights_host.assign(w, w + m);
            weights_dev.upload(weights_host.data(), weights_host.size());
        }
        return weights_dev.ptr;
    }
    lar::RidgeDev view() const {
        return lar::RidgeDev{int(host.m), int(host.c), host.ridge, tol, host.normal_equations ? 1 : 0, k.ptr, gram.ptr};
    }
    void* reserve(size_t need) {
        if (need > scratch_bytes) {
            if (scratch) lar::cuda_check(cudaFree(scratch), "cudaFree");
            scratch = nullptr;
            scratch_bytes = 0;
            lar::cuda_check(cudaMalloc(&scratch, need), "cudaMalloc (SD scratch)");
            scratch_bytes = need;
        }
        return scratch;
    }
};

// DeconvKernel (cpp/src/python/sd.cpp:260-292): one resolution of a multi-tissue kernel.
struct lar_deconv_kernel_s {
    int64_t m = 0, ca = 0, ci = 0, nb = 0;
    lar::DeviceArray<double> kt, iso, wiso;
    lar::DeviceArray<float> kt32, iso32, wiso32;  // FP32 copies for the plain single-precision fit
    lar::DeviceArray<int> blocks;
    // The lane-per-voxel fractions' constants and [K, iso] (m, ca + ci), where they apply.
    lar::DeviceArray<double> fx, kx;
    int fx_rows = 0;
    lar::TissueDev view() const {
        return lar::TissueDev{int(m), int(ca), int(ci), int(nb), kt.ptr, iso.ptr, wiso.ptr, blocks.ptr, fx.ptr, fx_rows};
    }
};

using namespace lar;

// The constants of a kernel's lane-per-voxel fractions (FracConstants) and its columns side by side;
// left out for a kernel that is too wide, not finite and non-negative, or has many candidate rows.
static void prepare_frac_constants(lar_deconv_kernel_s* h, const double* k, const double* iso) {
    const int m = int(h->m), c = int(h->ca), ci = int(h->ci);
    if (c > kFracCols || ci > 3 || !corr_tc_fits(m, 0)) return;
    for (int64_t i = 0; i < int64_t(m) * c; ++i)
        if (!(k[i] >= 0.0 && std::isfinite(k[i]))) return;
    // The rows that no other row bounds.
    std::vector<int> top;
    for (int i = 0; i < m; ++i) {
        auto bounds = [&](int a, int b) {  // row a >= row b everywhere
            for (int j = 0; j < c; ++j)
                if (k[size_t(a) * c + j] < k[size_t(b) * c + j]) return false;
            return true;
        };
        bool out = false;
        for (int t : top) out |= bounds(t, i);
        if (out) continue;
        top.erase(std::remove_if(top.begin(), top.end(), [&](int t) { return bounds(i, t); }), top.end());
        top.push_back(i);
        if (int(top.size()) > 4 * kFracRows) return;
    }
    if (int(top.size()) > kFracRows) return;
    const int rows = int(top.size());
    std::vector<double> p(size_t(FracConstants::doubles(c, ci, rows)), 0.0);
    const FracConstants f(p.data(), c, ci, rows);
    auto at = [&](const double* q, int i) -> double& { return p[size_t(q - p.data()) + size_t(i)]; };
    for (int i = 0; i < m; ++i) {
        const double* ki = k + size_t(i) * c;
        for (int a = 0; a < c; ++a) {
            for (int b = 0; b < c; ++b) at(f.gram, a * c + b) += ki[a] * ki[b];
            for (int t = 0; t < ci; ++t) at(f.ki, a * ci + t) += ki[a] * iso[size_t(i) * ci + t];
            at(f.ksum, a) += ki[a];
        }
        for (int t = 0; t < ci; ++t) {
            for (int q = 0; q < ci; ++q) at(f.ii, t * ci + q) += iso[size_t(i) * ci + t] * iso[size_t(i) * ci + q];
            at(f.isum, t) += std::fabs(iso[size_t(i) * ci + t]);
        }
    }
    for (int r = 0; r < rows; ++r)
        for (int j = 0; j < c; ++j) at(f.top, r * c + j) = k[size_t(top[size_t(r)]) * c + j];
    h->fx.upload(p.data(), p.size());
    h->fx_rows = rows;
    std::vector<double> kx(size_t(m) * (c + ci));
    for (int i = 0; i < m; ++i) {
        for (int j = 0; j < c; ++j) kx[size_t(i) * (c + ci) + j] = k[size_t(i) * c + j];
        for (int t = 0; t < ci; ++t) kx[size_t(i) * (c + ci) + c + t] = iso[size_t(i) * ci + t];
    }
    h->kx.upload(kx.data(), kx.size());
}

// The multi-tissue fit behind both entry points. device_rounds: enqueue every round with its
// voxel count read on the device (as under stream capture) instead of reading each count back.
static int fit_multi_tissue(const double* signals, int64_t v, const double* weights, lar_deconv_kernel lr,
                            lar_fod_solver lr_solver, lar_deconv_kernel hr, lar_fod_solver hr_solver,
                            int64_t max_outer, double fraction_tol, double final_tol_x, double* fods,
                            double* fractions, int32_t* rounds, uint8_t* status, void* stream,
                            bool device_rounds) {
    return guarded([&] {
        require(lr && hr && lr_solver && hr_solver, "kernels and solvers must not be NULL");
        require(weights != nullptr, "weights must not be NULL");
        const int64_t m = hr->m;
        require(lr->m == m, "signals, weights and the kernels' measurements do not match");
        require(lr->ci == hr->ci, "the two kernels have different numbers of isotropic tissues");
        // require_matching_solver (cpp/src/python/sd.cpp:294-307), with its message.
        auto matching = [m](const char* name, const lar_deconv_kernel_s& k, const lar_fod_solver_s& sv) {
            require(sv.host.c == k.ca && sv.host.m == m,
                    std::string("the ") + name + " solver (" + std::to_string(sv.host.c) + " directions, " +
                        std::to_string(sv.host.m) + " measurements) does not match its kernel (" +
                        std::to_string(k.ca) + " directions, " + std::to_string(m) + " measurements)");
        };
        matching("low-resolution", *lr, *lr_solver);
        matching("high-resolution", *hr, *hr_solver);
        require(max_outer >= 0, "max_outer must be at least 0");
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(signals && fods && fractions, "signals, fods and fractions must not be NULL");
        const int mi = int(m), ci = int(lr->ci), c_lr = int(lr->ca), c_hr = int(hr->ca);
        const int nf = int(hr->nb + hr->ci);
        const int max_rounds = int(std::min<int64_t>(max_outer, 1 << 20));
        const RidgeDev lrs = lr_solver->view(), hrs = hr_solver->view();
        const TissueDev lrt = lr->view(), hrt = hr->view();
        // A dRL solver (GRL) replaces the correlations and the NNLS of its stage by drl_kernel on
        // the stage's anisotropic signals; the fractions are the same.
        const bool lr_drl = lr_solver->kind == 1, hr_drl = hr_solver->kind == 1;
        const NnlsLaunch lr_nnls = nnls_variant(c_lr), hr_nnls = nnls_variant(c_hr);
        const size_t lr_smem = nnls_smem_bytes(c_lr, lr_nnls.cap) * kMtWarps;
        const size_t hr_smem = nnls_smem_bytes(c_hr, hr_nnls.cap) * kMtWarps;
        // Voxels per pass: the per-voxel state of a pass (correlations, the low-resolution FOD,
        // f_iso and the previous fractions, two list entries, the round count and status) within
        // 4 GiB.
        // (a lane per voxel for the fractions: K^T s and iso^T s too)
        const bool lane_frac = !lr_drl && lrt.fx != nullptr;
        const size_t per_voxel = (size_t(std::max(c_lr, c_hr)) + size_t(c_lr) + 2 * size_t(ci) + 1 +
                                  (lane_frac ? size_t(c_lr + ci) : 0)) *
                                     sizeof(double) +
                                 3 * sizeof(int) + 1;
        const int64_t n_max = std::min<int64_t>(v, std::max<int64_t>(4096, int64_t((size_t(4) << 30) / per_voxel)));
        const int64_t lr_slots = lr_drl ? 0 : resident_slots(lr_nnls.kernel, lr_smem, n_max, "sd.nnls.ctas_per_sm");
        // Low-resolution kernels of at most 48 directions with normal equations: the lean NNLS with the
        // Gram matrix in shared memory, the voxels that need the QR fallback or a larger factor then
        // refitted by the full-factor kernel.
        const bool low = !lr_drl && lrs.normal_equations && c_lr <= kLowCols;
        const size_t low_smem = low_smem_bytes(c_lr);
        const int64_t low_slots =
            low ? resident_slots(ridge_nnls_low_kernel, low_smem, n_max, "sd.nnls.ctas_per_sm", kLowWarps) : 0;
        const int64_t hr_slots = hr_drl ? 0 : resident_slots(hr_nnls.kernel, hr_smem, n_max, "sd.nnls.ctas_per_sm");
        // High-resolution kernels of 65 to 320 directions with normal equations: the same, with the
        // Gram matrix in L2.
        const bool high = !hr_drl && hrs.normal_equations && c_hr > 64 && c_hr <= 320;
        const int64_t high_slots =
            high ? resident_slots(ridge_nnls_high_kernel, high_smem_bytes(), n_max, "sd.nnls.ctas_per_sm", kHighWarps) : 0;
        const size_t lane_smem = lane_frac ? frac_lane_smem(FracConstants::doubles(c_lr, ci, lrt.fx_rows)) : 0;
        const int64_t lf_slots =
            lane_frac ? resident_slots(lane_fractions_kernel, lane_smem, (n_max + 31) / 32, "sd.fractions.ctas_per_sm")
                      : resident_slots(lr_fractions_kernel, 0, n_max, "sd.fractions.ctas_per_sm");
        const int64_t hf_slots = resident_slots(hr_fractions_kernel, 0, n_max, "sd.fractions.ctas_per_sm");
        const size_t lr_slot = nnls_slot_doubles(mi, lr_nnls.cap), hr_slot = nnls_slot_doubles(mi, hr_nnls.cap);
        const size_t lf_slot = frac_slot_doubles(mi, c_lr, 1 + ci), hf_slot = frac_slot_doubles(mi, c_hr, nf);
        const size_t slot_doubles =
            std::max(std::max(size_t(lr_slots) * lr_slot, size_t(hr_slots) * hr_slot),
                     std::max(size_t(lf_slots) * lf_slot, size_t(hf_slots) * hf_slot));
        struct Pieces {
            int* counters;  // [0] the persistent kernels' work counter, [2], [3] the two lists' counts,
                            // [4] the voxels to refit by the one-warp NNLS
            int* list[2];
            int* redo;
            double *fiso, *prev, *corr, *xlr, *ks, *slots;
            int32_t* rounds;
            uint8_t* bad;
        };
        auto carve_all = [&](Carver& cv) {
            Pieces p;
            p.counters = cv.take<int>(8);
            p.list[0] = cv.take<int>(size_t(n_max));
            p.list[1] = cv.take<int>(size_t(n_max));
            p.redo = cv.take<int>(size_t(n_max));
            p.fiso = cv.take<double>(size_t(n_max) * std::max(ci, 1));
            p.prev = cv.take<double>(size_t(n_max) * (ci + 1));
            p.corr = cv.take<double>(size_t(n_max) * std::max(c_lr, c_hr));
            p.xlr = cv.take<double>(size_t(n_max) * c_lr);
            p.ks = cv.take<double>(lane_frac ? size_t(n_max) * (c_lr + ci) : 0);
            p.rounds = cv.take<int32_t>(size_t(n_max));
            p.bad = cv.take<uint8_t>(size_t(n_max));
            p.slots = cv.take<double>(slot_doubles);
            return p;
        };
        Carver sizing{nullptr};
        carve_all(sizing);
        Carver cv{static_cast<char*>(hr_solver->reserve(sizing.used))};
        const Pieces P = carve_all(cv);
        auto st = static_cast<cudaStream_t>(stream);
        // Under stream capture (a CUDA graph) nothing may wait on the host: every round is
        // enqueued and reads its voxel count on the device, exiting at once when it is 0.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        cuda_check(cudaStreamIsCapturing(st, &capture), "cudaStreamIsCapturing");
        const bool capturing = capture != cudaStreamCaptureStatusNone;
        const bool graph = capturing || device_rounds;
        const double* dweights = hr_solver->device_weights(weights, m, capturing);
        int* host_count = graph ? nullptr : hr_solver->count_buffer();
        auto blocks = [](int64_t slots, int64_t count, int warps = kMtWarps) {
            return unsigned(std::max<int64_t>(1, std::min<int64_t>(slots / warps, (count + warps - 1) / warps)));
        };
        // The low-resolution kernel's wide CTAs: a short list still takes a CTA per SM, so that its voxels
        // do not queue on a few SMs.
        auto low_blocks = [&](int64_t slots, int64_t count) {
            return unsigned(std::min<int64_t>(slots / kLowWarps,
                                              std::max<int64_t>((count + kLowWarps - 1) / kLowWarps,
                                                                std::min<int64_t>(count, sm_count()))));
        };
        auto reset_queue = [&] { cuda_check(cudaMemsetAsync(P.counters, 0, sizeof(int), st), "cudaMemsetAsync"); };
        for (int64_t v0 = 0; v0 < v; v0 += n_max) {
            const int64_t n = std::min(n_max, v - v0);
            const double* sig = signals + v0 * m;
            if (ci > 0) cuda_check(cudaMemsetAsync(P.fiso, 0, size_t(n) * ci * sizeof(double), st), "cudaMemsetAsync");
            cuda_check(cudaMemsetAsync(P.rounds, 0, size_t(n) * sizeof(int32_t), st), "cudaMemsetAsync");
            cuda_check(cudaMemsetAsync(P.bad, 0, size_t(n), st), "cudaMemsetAsync");
            const SignalDev lr_sig{sig, dweights, lrt.wiso, P.fiso, mi, ci};
            if (lane_frac && max_rounds > 0) {
                const RidgeDev kx{mi, c_lr + ci, 0.0, 0.0, 0, lr->kx.ptr, nullptr};
                launch_correlate(SignalDev{sig, nullptr, nullptr, nullptr, mi, 0}, nullptr, n, nullptr, kx, P.ks,
                                 c_lr + ci, st);
            }
            // The first round takes every voxel; later rounds the list the previous one wrote,
            // with its count read back on the host (or, under capture, on the device).
            const int* cur = nullptr;
            const int* cur_count = nullptr;
            int side = 0;
            int64_t count = n;
            for (int round = 0; round < max_rounds && count > 0; ++round) {
                int* nxt = P.list[side];
                int* nxt_count = P.counters + 2 + side;
                if (!lr_drl) launch_correlate(lr_sig, cur, count, cur_count, lrs, P.corr, c_lr, st);
                reset_queue();
                cuda_check(cudaMemsetAsync(nxt_count, 0, sizeof(int), st), "cudaMemsetAsync");
                if (lr_drl) {
                    const DrlSignal lr_as{sig, dweights, lrt.wiso, P.fiso, mi, ci};
                    launch_drl_listed(lr_solver->drl, lr_as, cur, count, cur_count, P.xlr, c_lr, st);
                } else if (low) {
                    cuda_check(cudaMemsetAsync(P.counters + 4, 0, sizeof(int), st), "cudaMemsetAsync");
                    {
                        LaunchScope scope("ridge_nnls_low_kernel", st);
                        ridge_nnls_low_kernel<<<low_blocks(low_slots, count), kLowWarps * 32, low_smem, st>>>(
                            lrs, cur, count, cur_count, P.corr, c_lr, P.xlr, c_lr, P.redo, P.counters + 4, P.counters);
                        cuda_check(cudaGetLastError(), "ridge_nnls_low_kernel launch");
                    }
                    reset_queue();
                    // The voxels it handed back are rare: a persistent grid of one CTA per SM takes them.
                    LaunchScope scope(lr_nnls.name, st);
                    const unsigned redo_blocks = std::min<unsigned>(blocks(lr_slots, count), unsigned(sm_count()));
                    lr_nnls.kernel<<<redo_blocks, kMtWarps * 32, lr_smem, st>>>(
                        lrs, lr_sig, P.redo, count, P.counters + 4, P.corr, c_lr, P.xlr, c_lr, P.bad, P.counters,
                        P.slots, lr_slot);
                    cuda_check(cudaGetLastError(), "ridge_nnls_kernel launch");
                } else {
                    LaunchScope scope(lr_nnls.name, st);
                    lr_nnls.kernel<<<blocks(lr_slots, count), kMtWarps * 32, lr_smem, st>>>(
                        lrs, lr_sig, cur, count, cur_count, P.corr, c_lr, P.xlr, c_lr, P.bad, P.counters, P.slots,
                        lr_slot);
                    cuda_check(cudaGetLastError(), "ridge_nnls_kernel launch");
                }
                if (lane_frac) {
                    LaunchScope scope("lane_fractions_kernel", st);
                    const FracRound fr{sig, P.xlr, P.ks, P.fiso, P.prev, P.rounds, nxt, nxt_count, c_lr, round,
                                       max_rounds, fraction_tol};
                    const unsigned grid = unsigned(std::min<int64_t>((count + 31) / 32, lf_slots / kFracWarps));
                    lane_fractions_kernel<<<grid, kFracWarps * 32, lane_smem, st>>>(lrt, fr, cur, count, cur_count,
                                                                                   P.slots, lf_slot);
                    cuda_check(cudaGetLastError(), "lane_fractions_kernel launch");
                } else {
                    reset_queue();
                    LaunchScope scope("lr_fractions_kernel", st);
                    lr_fractions_kernel<<<blocks(lf_slots, count), kMtWarps * 32, 0, st>>>(
                        lrt, sig, P.xlr, c_lr, cur, count, cur_count, round, max_rounds, fraction_tol, P.fiso, P.prev,
                        P.rounds, nxt, nxt_count, P.counters, P.slots, lf_slot);
                    cuda_check(cudaGetLastError(), "lr_fractions_kernel launch");
                }
                if (!graph) {
                    cuda_check(cudaMemcpyAsync(host_count, nxt_count, sizeof(int), cudaMemcpyDeviceToHost, st),
                               "cudaMemcpyAsync (round count)");
                    cuda_check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
                    count = *host_count;
                } else {
                    cur_count = nxt_count;
                }
                cur = nxt;
                side ^= 1;
            }
            const SignalDev hr_sig{sig, dweights, hrt.wiso, P.fiso, mi, ci};
            if (hr_drl) {
                const DrlSignal hr_as{sig, dweights, hrt.wiso, P.fiso, mi, ci};
                launch_drl_listed(hr_solver->drl, hr_as, nullptr, n, nullptr, fods + v0 * c_hr, c_hr, st);
            } else {
                launch_correlate(hr_sig, nullptr, n, nullptr, hrs, P.corr, c_hr, st);
                reset_queue();
                if (high) {
                    cuda_check(cudaMemsetAsync(P.counters + 4, 0, sizeof(int), st), "cudaMemsetAsync");
                    {
                        LaunchScope scope("ridge_nnls_high_kernel", st);
                        ridge_nnls_high_kernel<<<blocks(high_slots, n, kHighWarps), kHighWarps * 32, high_smem_bytes(),
                                                 st>>>(hrs, n, P.corr, c_hr, fods + v0 * c_hr, c_hr, P.redo,
                                                       P.counters + 4, P.counters);
                        cuda_check(cudaGetLastError(), "ridge_nnls_high_kernel launch");
                    }
                    reset_queue();
                    // The voxels the first pass handed back (rare): a grid of one CTA per SM.
                    LaunchScope scope(hr_nnls.name, st);
                    const unsigned redo_blocks = std::min<unsigned>(blocks(hr_slots, n), unsigned(sm_count()));
                    hr_nnls.kernel<<<redo_blocks, kMtWarps * 32, hr_smem, st>>>(
                        hrs, hr_sig, P.redo, n, P.counters + 4, P.corr, c_hr, fods + v0 * c_hr, c_hr, P.bad,
                        P.counters, P.slots, hr_slot);
                    cuda_check(cudaGetLastError(), "ridge_nnls_kernel launch");
                } else {
                    LaunchScope scope(hr_nnls.name, st);
                    hr_nnls.kernel<<<blocks(hr_slots, n), kMtWarps * 32, hr_smem, st>>>(
                        hrs, hr_sig, nullptr, n, nullptr, P.corr, c_hr, fods + v0 * c_hr, c_hr, P.bad, P.counters,
                        P.slots, hr_slot);
                    cuda_check(cudaGetLastError(), "ridge_nnls_kernel launch");
                }
            }
            reset_queue();
            LaunchScope scope("hr_fractions_kernel", st);
            hr_fractions_kernel<<<blocks(hf_slots, n), kMtWarps * 32, 0, st>>>(
                hrt, sig, fods + v0 * c_hr, n, final_tol_x, P.rounds, P.bad, fractions + v0 * nf,
                rounds ? rounds + v0 : nullptr, status ? status + v0 : nullptr, P.counters, P.slots, hf_slot);
            cuda_check(cudaGetLastError(), "hr_fractions_kernel launch");
        }
    });
}

// ---- batches (batch.cuh): the mFOD family --------------------------------------------------

namespace lar {

struct MfodBatch {
    std::vector<MfodBatchJob> jobs;
    std::vector<std::vector<double>> weights;
    std::vector<std::unique_ptr<DeviceArray<double>>> weights_dev;
    int max_rounds = -1;
    double fraction_tol = 0.0, final_tol = 0.0;
    int ci = -1, m_max = 0, c_lr_max = 0, c_hr_max = 0, nf_max = 0;
    int64_t voxels = 0, tiles = 0;
    // Finalized: the device job table, the per-voxel state and the launch shapes.
    DeviceArray<MfodBatchJob> d_jobs;
    void* scratch = nullptr;
    MfodBatchState B{};
    int *list[2] = {nullptr, nullptr}, *counts[2] = {nullptr, nullptr}, *queue = nullptr;
    double* slots = nullptr;
    int64_t low_slots = 0, high_slots = 0, lr_slots = 0, hr_slots = 0, lf_slots = 0, hf_slots = 0;
    size_t low_smem = 0, lr_smem = 0, hr_smem = 0;
    size_t lr_slot = 0, hr_slot = 0, lf_slot = 0, hf_slot = 0;
    ~MfodBatch() {
        if (scratch) cudaFree(scratch);
    }
    int64_t ks_doubles = 0;  // of the volumes whose fractions take a lane per voxel
    int ks_m = 0, fx_doubles = 0;  // their most measurements and constants
    bool lane_all = true;          // they are all of them
    int64_t lane_slots = 0;
    int tc_m = 0;         // the most measurements of the volumes the tensor-core correlations take
    bool tc_all = true;   // they take every volume
    // A stage's correlations: the tensor-core kernel's volumes, then the others.
    template <bool HR>
    void correlate(const int* list, unsigned grid, cudaStream_t st) {
        const int c_max = HR ? c_hr_max : c_lr_max;
        if (tc_m > 0) {
            const size_t smem = corr_tc_smem(tc_m, ci);
            const unsigned gy = unsigned((c_max + kCorrTcCols - 1) / kCorrTcCols);
            const unsigned gx = std::max(1u, unsigned(sm_count()) / gy);
            auto run = [&](auto kernel) {
                allow_smem(kernel, smem);
                LaunchScope scope("batch_correlate_kernel", st);
                kernel<<<dim3(gx, gy), kCorrTcWarps * 32, smem, st>>>(B, list);
                cuda_check(cudaGetLastError(), "batch_correlate_tc_kernel launch");
            };
            if (ci == 0) run(batch_correlate_tc_kernel<0, HR>);
            else if (ci == 1) run(batch_correlate_tc_kernel<1, HR>);
            else if (ci == 2) run(batch_correlate_tc_kernel<2, HR>);
            else run(batch_correlate_tc_kernel<3, HR>);
        }
        if (tc_all) return;
        LaunchScope scope("batch_correlate_kernel", st);
        if constexpr (HR)
            batch_correlate_kernel<4, true><<<dim3(grid, unsigned((c_max + 63) / 64)), 128, 0, st>>>(B, list);
        else
            batch_correlate_kernel<3, false><<<grid, 128, 0, st>>>(B, list);
        cuda_check(cudaGetLastError(), "batch_correlate_kernel launch");
    }
};

MfodBatch* mfod_batch_create() { return new MfodBatch(); }

void mfod_batch_destroy(MfodBatch* b) { delete b; }

void mfod_batch_add(MfodBatch* b, const double* signals, int64_t v, const double* weights, lar_deconv_kernel lr,
                    lar_fod_solver lr_solver, lar_deconv_kernel hr, lar_fod_solver hr_solver, int64_t max_outer,
                    double fraction_tol, double final_tol_x, double* fods, double* fractions, int32_t* rounds,
                    uint8_t* status) {
    require(lr && hr && lr_solver && hr_solver, "kernels and solvers must not be NULL");
    require(weights != nullptr, "weights must not be NULL");
    const int64_t m = hr->m;
    require(lr->m == m, "signals, weights and the kernels' measurements do not match");
    require(lr->ci == hr->ci, "the two kernels have different numbers of isotropic tissues");
    require(lr_solver->host.c == lr->ca && lr_solver->host.m == m && hr_solver->host.c == hr->ca &&
                hr_solver->host.m == m,
            "a solver does not match its kernel");
    require(lr_solver->kind == 0 && hr_solver->kind == 0 && lr_solver->host.normal_equations &&
                hr_solver->host.normal_equations,
            "a batch takes ridge NNLS (L2NNLS) solvers with normal equations");
    require(lr->ca <= 48 && hr->ca > 64 && hr->ca <= 320,
            "a batch takes low-resolution kernels of at most 48 directions and high-resolution ones of 65 to 320");
    require(max_outer >= 0 && v >= 0, "max_outer and v must be at least 0");
    require(v == 0 || (signals && fods && fractions), "signals, fods and fractions must not be NULL");
    const int rounds_cap = int(std::min<int64_t>(max_outer, 1 << 20));
    if (b->max_rounds < 0) {
        b->max_rounds = rounds_cap;
        b->fraction_tol = fraction_tol;
        b->final_tol = final_tol_x;
        b->ci = int(lr->ci);
    }
    require(rounds_cap == b->max_rounds && fraction_tol == b->fraction_tol && final_tol_x == b->final_tol,
            "every mFOD job of a batch takes the same max_outer, fraction_tol and final_tol_x");
    require(int(lr->ci) == b->ci, "every mFOD job of a batch has the same isotropic tissues");
    MfodBatchJob j{};
    j.v = v;
    j.off = b->voxels;
    j.lr = lr_solver->view();
    j.hr = hr_solver->view();
    j.lrt = lr->view();
    j.hrt = hr->view();
    j.s = signals;
    j.fods = fods;
    j.fractions = fractions;
    j.rounds = rounds;
    j.status = status;
    j.kx = lr->kx.ptr;
    j.ks_off = b->ks_doubles;
    if (j.lrt.fx != nullptr) {
        b->ks_doubles += v * (lr->ca + lr->ci);
        b->ks_m = std::max(b->ks_m, int(m));
        b->fx_doubles = std::max(b->fx_doubles, FracConstants::doubles(int(lr->ca), int(lr->ci), lr->fx_rows));
    } else {
        b->lane_all = false;
    }
    b->jobs.push_back(j);
    b->weights.emplace_back(weights, weights + m);
    b->voxels += v;
    b->tiles += (v + kCorrVoxels - 1) / kCorrVoxels;
    b->m_max = std::max(b->m_max, int(m));
    if (corr_tc_fits(int(m), int(lr->ci))) b->tc_m = std::max(b->tc_m, int(m));
    else b->tc_all = false;
    b->c_lr_max = std::max(b->c_lr_max, int(lr->ca));
    b->c_hr_max = std::max(b->c_hr_max, int(hr->ca));
    b->nf_max = std::max(b->nf_max, int(hr->nb + hr->ci));
}

void mfod_batch_finalize(MfodBatch* b) {
    if (b->jobs.empty()) return;
    require(b->voxels < (int64_t(1) << 31), "at most 2^31 - 1 mFOD voxels per batch");
    for (size_t k = 0; k < b->jobs.size(); ++k) {
        b->weights_dev.push_back(std::make_unique<DeviceArray<double>>());
        b->weights_dev.back()->upload(b->weights[k].data(), b->weights[k].size());
        b->jobs[k].w = b->weights_dev.back()->ptr;
    }
    b->d_jobs.upload(b->jobs.data(), b->jobs.size());
    const int64_t V = b->voxels, nj = int64_t(b->jobs.size());
    const int ci = b->ci, mi = b->m_max, ldc = std::max(b->c_lr_max, b->c_hr_max), ldx = b->c_lr_max;
    // Launch shapes: the single-volume fit's persistent grids, sized for the whole batch.
    b->low_smem = low_smem_bytes(b->c_lr_max);
    b->low_slots = resident_slots(batch_low_kernel, b->low_smem, V, "sd.nnls.ctas_per_sm", kLowWarps);
    b->high_slots = resident_slots(batch_high_kernel, high_smem_bytes(), V, "sd.nnls.ctas_per_sm", kHighWarps);
    b->lr_smem = nnls_smem_bytes(b->c_lr_max, 32) * kMtWarps;
    b->lr_slots = resident_slots(batch_redo_kernel<1, 2, false>, b->lr_smem, V, "sd.nnls.ctas_per_sm");
    b->hr_smem = nnls_smem_bytes(b->c_hr_max, kCholCap) * kMtWarps;
    b->hr_slots = resident_slots(batch_redo_kernel<kCholCap / 32, 10, true>, b->hr_smem, V, "sd.nnls.ctas_per_sm");
    b->lf_slots = b->lane_all ? 0 : resident_slots(batch_lr_fractions_kernel, 0, V, "sd.fractions.ctas_per_sm");
    b->lane_slots = b->fx_doubles ? resident_slots(batch_lane_fractions_kernel, frac_lane_smem(b->fx_doubles),
                                                   (V + 31) / 32, "sd.fractions.ctas_per_sm")
                                  : 0;
    b->hf_slots = resident_slots(batch_hr_fractions_kernel, 0, V, "sd.fractions.ctas_per_sm");
    b->lr_slot = nnls_slot_doubles(mi, 32);
    b->hr_slot = nnls_slot_doubles(mi, kCholCap);
    b->lf_slot = frac_slot_doubles(mi, b->c_lr_max, 1 + ci);
    b->hf_slot = frac_slot_doubles(mi, b->c_hr_max, b->nf_max);
    const size_t slot_doubles =
        std::max({size_t(b->lr_slots) * b->lr_slot, size_t(b->hr_slots) * b->hr_slot,
                  size_t(std::max(b->lf_slots, b->lane_slots)) * b->lf_slot, size_t(b->hf_slots) * b->hf_slot});
    auto carve_all = [&](Carver& cv) {
        MfodBatchState s{};
        s.jobs = b->d_jobs.ptr;
        s.n_jobs = int(nj);
        s.ci = ci;
        s.ldc = ldc;
        s.ldx = ldx;
        s.fiso = cv.take<double>(size_t(V) * std::max(ci, 1));
        s.prev = cv.take<double>(size_t(V) * (ci + 1));
        s.corr = cv.take<double>(size_t(V) * ldc);
        s.xlr = cv.take<double>(size_t(V) * ldx);
        s.ks = cv.take<double>(size_t(b->ks_doubles));
        s.rounds = cv.take<int32_t>(size_t(V));
        s.bad = cv.take<uint8_t>(size_t(V));
        s.vfirst = cv.take<int64_t>(size_t(nj) + 1);
        s.tfirst = cv.take<int64_t>(size_t(nj) + 1);
        s.qfirst = cv.take<int64_t>(size_t(nj) + 1);
        s.cfirst = cv.take<int64_t>(size_t(nj) + 1);
        s.redo = cv.take<int64_t>(size_t(V));
        s.redo_count = cv.take<int>(1);
        b->list[0] = cv.take<int>(size_t(V));
        b->list[1] = cv.take<int>(size_t(V));
        b->counts[0] = cv.take<int>(size_t(nj));
        b->counts[1] = cv.take<int>(size_t(nj));
        b->queue = cv.take<int>(1);
        b->slots = cv.take<double>(slot_doubles);
        return s;
    };
    Carver sizing{nullptr};
    carve_all(sizing);
    cuda_check(cudaMalloc(&b->scratch, sizing.used), "cudaMalloc (mFOD batch state)");
    Carver cv{static_cast<char*>(b->scratch)};
    b->B = carve_all(cv);
}

void mfod_batch_run(MfodBatch* b, cudaStream_t st) {
    if (b->jobs.empty() || b->voxels == 0) return;
    const MfodBatchState& B = b->B;
    const int64_t V = b->voxels, nj = int64_t(b->jobs.size());
    const int ci = b->ci;
    auto blocks = [](int64_t slots, int64_t count, int warps = kMtWarps) {
        return unsigned(std::max<int64_t>(1, std::min<int64_t>(slots / warps, (count + warps - 1) / warps)));
    };
    auto zero = [&](void* p, size_t bytes) { cuda_check(cudaMemsetAsync(p, 0, bytes, st), "cudaMemsetAsync"); };
    auto launched = [](const char* what) { cuda_check(cudaGetLastError(), what); };
    if (ci > 0) zero(B.fiso, size_t(V) * ci * sizeof(double));
    zero(B.rounds, size_t(V) * sizeof(int32_t));
    zero(B.bad, size_t(V));
    // The correlation grids stay resident-sized: a round's tiles are only known on the device.
    const unsigned corr_grid = unsigned(std::min<int64_t>(b->tiles, int64_t(sm_count()) * kCorrResidentCtas));
    const unsigned lr_redo_blocks = std::min<unsigned>(blocks(b->lr_slots, V), unsigned(sm_count()));
    const unsigned hr_redo_blocks = std::min<unsigned>(blocks(b->hr_slots, V), unsigned(sm_count()));
    // Every round is enqueued: each stage reads its tickets on the device, so a round whose
    // lists are all empty costs only its launches.
    const int* cur = nullptr;
    const int* cur_counts = nullptr;
    int side = 0;
    for (int round = 0; round < b->max_rounds; ++round) {
        int* nxt = b->list[side];
        int* nxt_counts = b->counts[side];
        {
            LaunchScope scope("batch_plan_kernel", st);
            batch_plan_kernel<<<1, 32, 0, st>>>(B, cur_counts);
            launched("batch_plan_kernel launch");
        }
        if (round == 0 && b->fx_doubles > 0) {
            const size_t smem = corr_tc_smem(b->ks_m, 0);
            allow_smem(batch_ks_kernel, smem);
            LaunchScope scope("batch_ks_kernel", st);
            const unsigned gy = unsigned((b->c_lr_max + ci + kCorrTcCols - 1) / kCorrTcCols);
            batch_ks_kernel<<<dim3(unsigned(sm_count()) / gy, gy), kCorrTcWarps * 32, smem, st>>>(B);
            launched("batch_ks_kernel launch");
        }
        b->correlate<false>(cur, corr_grid, st);
        zero(b->queue, sizeof(int));
        zero(nxt_counts, size_t(nj) * sizeof(int));
        zero(B.redo_count, sizeof(int));
        {
            LaunchScope scope("batch_low_kernel", st);
            batch_low_kernel<<<blocks(b->low_slots, V, kLowWarps), kLowWarps * 32, b->low_smem, st>>>(B, cur, b->queue);
            launched("batch_low_kernel launch");
        }
        zero(b->queue, sizeof(int));
        {
            LaunchScope scope("batch_redo_kernel<1,2>", st);
            batch_redo_kernel<1, 2, false><<<lr_redo_blocks, kMtWarps * 32, b->lr_smem, st>>>(
                B, b->c_lr_max, b->queue, b->slots, b->lr_slot);
            launched("batch_redo_kernel launch");
        }
        if (b->fx_doubles > 0) {
            LaunchScope scope("batch_lane_fractions_kernel", st);
            batch_lane_fractions_kernel<<<unsigned(b->lane_slots / kFracWarps), kFracWarps * 32,
                                          frac_lane_smem(b->fx_doubles), st>>>(
                B, b->fx_doubles, cur, round, b->max_rounds, b->fraction_tol, nxt, nxt_counts, b->slots, b->lf_slot);
            launched("batch_lane_fractions_kernel launch");
        }
        if (!b->lane_all) {
            zero(b->queue, sizeof(int));
            LaunchScope scope("batch_lr_fractions_kernel", st);
            batch_lr_fractions_kernel<<<blocks(b->lf_slots, V), kMtWarps * 32, 0, st>>>(
                B, cur, round, b->max_rounds, b->fraction_tol, nxt, nxt_counts, b->queue, b->slots, b->lf_slot);
            launched("batch_lr_fractions_kernel launch");
        }
        cur = nxt;
        cur_counts = nxt_counts;
        side ^= 1;
    }
    {
        LaunchScope scope("batch_plan_kernel", st);
        batch_plan_kernel<<<1, 32, 0, st>>>(B, nullptr);
        launched("batch_plan_kernel launch");
    }
    b->correlate<true>(nullptr, corr_grid, st);
    zero(b->queue, sizeof(int));
    zero(B.redo_count, sizeof(int));
    {
        LaunchScope scope("batch_high_kernel", st);
        batch_high_kernel<<<blocks(b->high_slots, V, kHighWarps), kHighWarps * 32, high_smem_bytes(), st>>>(B, b->queue);
        launched("batch_high_kernel launch");
    }
    zero(b->queue, sizeof(int));
    {
        LaunchScope scope("batch_redo_kernel<8,10>", st);
        batch_redo_kernel<kCholCap / 32, 10, true><<<hr_redo_blocks, kMtWarps * 32, b->hr_smem, st>>>(
            B, b->c_hr_max, b->queue, b->slots, b->hr_slot);
        launched("batch_redo_kernel launch");
    }
    zero(b->queue, sizeof(int));
    LaunchScope scope("batch_hr_fractions_kernel", st);
    batch_hr_fractions_kernel<<<blocks(b->hf_slots, V), kMtWarps * 32, 0, st>>>(B, b->final_tol, b->queue, b->slots,
                                                                              b->hf_slot);
    launched("batch_hr_fractions_kernel launch");
}

}  // namespace lar

extern "C" {

int lar_fit_multi_tissue(const double* signals, int64_t v, const double* weights, lar_deconv_kernel lr,
                         lar_fod_solver lr_solver, lar_deconv_kernel hr, lar_fod_solver hr_solver,
                         int64_t max_outer, double fraction_tol, double final_tol_x, double* fods,
                         double* fractions, int32_t* rounds, uint8_t* status, void* stream) {
    return fit_multi_tissue(signals, v, weights, lr, lr_solver, hr, hr_solver, max_outer, fraction_tol, final_tol_x,
                            fods, fractions, rounds, status, stream, false);
}

int lar_fit_multi_tissue_async(const double* signals, int64_t v, const double* weights, lar_deconv_kernel lr,
                               lar_fod_solver lr_solver, lar_deconv_kernel hr, lar_fod_solver hr_solver,
                               int64_t max_outer, double fraction_tol, double final_tol_x, double* fods,
                               double* fractions, int32_t* rounds, uint8_t* status, void* stream) {
    return fit_multi_tissue(signals, v, weights, lr, lr_solver, hr, hr_solver, max_outer, fraction_tol, final_tol_x,
                            fods, fractions, rounds, status, stream, true);
}

int lar_fit_multi_tissue_plain_fp32(const float* signals, int64_t v, const double* weights, lar_deconv_kernel lr,
                                    lar_fod_solver lr_solver, lar_deconv_kernel hr, lar_fod_solver hr_solver,
                                    int64_t max_outer, double fraction_tol, double final_tol_x, float* fods,
                                    float* fractions, int32_t* rounds, uint8_t* status, void* stream) {
    return guarded([&] {
        require(lr && hr && lr_solver && hr_solver, "kernels and solvers must not be NULL");
        require(weights != nullptr, "weights must not be NULL");
        require(lr_solver->kind == 0 && hr_solver->kind == 0, "the plain FP32 fit takes L2NNLS solvers");
        const int64_t m = hr->m;
        require(lr->m == m && lr_solver->host.m == m && hr_solver->host.m == m,
                "signals, weights and the kernels' measurements do not match");
        require(lr_solver->host.c == lr->ca && hr_solver->host.c == hr->ca, "a solver does not match its kernel");
        require(lr->ci == hr->ci && lr->nb == 1, "the low-resolution kernel must have one anisotropic block and the "
                                                 "isotropic tissues of the high-resolution one");
        require(m <= kPlainMaxMeasurements && std::max(lr->ca, hr->ca) <= kPlainMaxColumns &&
                    hr->nb + hr->ci <= kPlainMaxGroups && 1 + lr->ci <= kPlainMaxGroups,
                "the plain FP32 fit takes at most 512 measurements, 320 directions and 4 fraction columns");
        require(max_outer >= 0 && v >= 0, "max_outer and v must be at least 0");
        if (v == 0) return;
        require(signals && fods && fractions, "signals, fods and fractions must not be NULL");
        auto st = static_cast<cudaStream_t>(stream);
        auto stage = [](const lar_deconv_kernel_s& k, const lar_fod_solver_s& sv) {
            return PlainStage{int(k.m), int(k.ca), int(k.ci), int(k.nb), float(sv.tol), sv.k32.ptr, sv.gram32.ptr,
                              k.kt32.ptr, k.iso32.ptr, k.wiso32.ptr, k.blocks.ptr};
        };
        std::vector<float> w32(weights, weights + m);
        float* dw = nullptr;
        cuda_check(cudaMallocAsync(reinterpret_cast<void**>(&dw), size_t(m) * sizeof(float), st), "cudaMallocAsync");
        cuda_check(cudaMemcpyAsync(dw, w32.data(), size_t(m) * sizeof(float), cudaMemcpyHostToDevice, st),
                   "cudaMemcpyAsync");
        launch_plain_fp32(stage(*lr, *lr_solver), stage(*hr, *hr_solver), signals, v, dw,
                          int(std::min<int64_t>(max_outer, 1 << 20)), float(fraction_tol), float(final_tol_x), fods,
                          fractions, rounds, status, st);
        // The weights' host copy must outlive the copy above.
        cuda_check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
        cuda_check(cudaFreeAsync(dw, st), "cudaFreeAsync");
    });
}

int lar_lsqnonneg(const double* c, int64_t m, int64_t n, const double* d, int default_tol, double tol_x, double* x,
                  void* stream) {
    return guarded([&] {
        require(m >= 1 && n >= 1 && n <= kMaxGroups, "lsqnonneg takes c of (m, n), m >= 1, 1 <= n <= 16");
        require(c && d && x, "c, d and x must not be NULL");
        auto st = static_cast<cudaStream_t>(stream);
        double* ws = nullptr;
        const size_t bytes = frac_slot_doubles(int(m), 0, int(n)) * sizeof(double);
        cuda_check(cudaMallocAsync(reinterpret_cast<void**>(&ws), bytes, st), "cudaMallocAsync");
        {
            LaunchScope scope("lsqnonneg_kernel", st);
            lsqnonneg_kernel<<<1, 32, 0, st>>>(c, int(m), int(n), d, default_tol != 0, tol_x, x, ws);
            cuda_check(cudaGetLastError(), "lsqnonneg_kernel launch");
        }
        cuda_check(cudaFreeAsync(ws, st), "cudaFreeAsync");
    });
}


int lar_drl_create(const double* k_t, const double* k_t_k, int64_t c, int64_t m, double nu, int64_t n_iter,
                   double init, lar_fod_solver* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(k_t != nullptr && k_t_k != nullptr && c > 0 && m > 1, "k_t must be a non-empty (c, m) array, m > 1");
        require(drl_fits(int(c)), "dRL takes at most 640 directions");
        require(n_iter >= 0, "n_iter must be at least 0");
        auto h = std::make_unique<lar_fod_solver_s>();
        h->kind = 1;
        h->host.m = m;
        h->host.c = c;
        h->drl_kt.upload(k_t, size_t(c * m));
        h->drl_gram.upload(k_t_k, size_t(c * c));
        h->drl = DrlDev{h->drl_kt.ptr, h->drl_gram.ptr, int(c), int(m), int(n_iter), nu, init};
        *out = h.release();
    });
}

int lar_l2nnls_create(const double* k, int64_t m, int64_t c, double reg, double tol_x, lar_fod_solver* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(reg >= 0.0, "reg must be at least 0");
        require(tol_x > 0.0, "tol_x must be positive");
        require(k != nullptr && m > 0 && c > 0, "k must be a non-empty (m, c) array");
        require(c <= 640 && m <= 4096, "the kernel has more than 640 directions or 4096 measurements");
        auto h = std::make_unique<lar_fod_solver_s>();
        h->host = host::prepare_ridge_design(k, m, c, reg);
        h->tol = tol_x;
        h->k.upload(h->host.kernel.data(), h->host.kernel.size());
        h->gram.upload(h->host.gram.data(), h->host.gram.size());
        upload_fp32(h->k32, h->host.kernel);
        upload_fp32(h->gram32, h->host.gram);
        *out = h.release();
    });
}

int lar_drl_set_precision(lar_fod_solver solver, int precision) {
    return guarded([&] {
        require(solver != nullptr && solver->kind == 1, "solver must be a dRL solver");
        require(precision == LAR_FP64 || precision == LAR_TF32X3, "precision must be LAR_FP64 or LAR_TF32X3");
        if (precision == LAR_FP64) {
            solver->drl.gtc = nullptr;
            solver->drl.err = nullptr;
            return;
        }
        const int c = int(solver->host.c);
        require(drl_tc_fits(c) && drl_tc_fits_measurements(c, int(solver->host.m)),
                "the tensor-core dRL takes 65 to 320 directions and at most " +
                    std::to_string(drl_tc_smem_bytes(c) / (48 * 8)) + " measurements");
        std::vector<double> gram(size_t(c) * c);
        cuda_check(cudaMemcpy(gram.data(), solver->drl_gram.ptr, gram.size() * sizeof(double), cudaMemcpyDeviceToHost),
                   "cudaMemcpy");
        const std::vector<float> layout = drl_tc_layout(gram.data(), c);
        solver->drl_gtc.upload(layout.data(), layout.size());
        const int zero = 0;
        solver->drl_err.upload(&zero, 1);
        solver->drl.gtc = solver->drl_gtc.ptr;
        solver->drl.err = solver->drl_err.ptr;
    });
}

int lar_drl_errors(lar_fod_solver solver, int* out) {
    return guarded([&] {
        require(solver != nullptr && out != nullptr, "solver and out must not be NULL");
        *out = 0;
        if (solver->drl.err == nullptr) return;
        cuda_check(cudaMemcpy(out, solver->drl.err, sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy");
    });
}

void lar_fod_solver_destroy(lar_fod_solver solver) { delete solver; }

int lar_deconv_kernel_create(const double* k_aniso, int64_t m, int64_t ca, const double* k_iso,
                             const double* w_k_iso, int64_t ci, const int64_t* blocks, int64_t nb,
                             lar_deconv_kernel* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(k_aniso != nullptr && m > 0 && ca > 0, "k_aniso must be a non-empty (m, ca) array");
        require(ci >= 0 && (ci == 0 || (k_iso && w_k_iso)), "k_iso and w_k_iso must be (m, ci) arrays");
        require(nb >= 1 && blocks != nullptr, "aniso_blocks must hold at least one block");
        require(nb + ci <= kMaxGroups, "at most 16 tissues");
        std::string text;
        for (int64_t b = 0; b < nb; ++b) {
            const int64_t s = blocks[2 * b], e = blocks[2 * b + 1];
            require(s >= 0 && s < e && e <= ca, "aniso_blocks must be non-empty ranges within 0.." +
                                                    std::to_string(ca));
        }
        auto h = std::make_unique<lar_deconv_kernel_s>();
        h->m = m; h->ca = ca; h->ci = ci; h->nb = nb;
        std::vector<double> kt(size_t(ca * m));
        for (int64_t i = 0; i < m; ++i)
            for (int64_t j = 0; j < ca; ++j) kt[size_t(j * m + i)] = k_aniso[i * ca + j];
        h->kt.upload(kt.data(), kt.size());
        upload_fp32(h->kt32, kt);
        std::vector<double> iso(size_t(std::max<int64_t>(1, m * ci)), 0.0), wiso(iso.size(), 0.0);
        if (ci > 0) {
            std::copy(k_iso, k_iso + m * ci, iso.begin());
            std::copy(w_k_iso, w_k_iso + m * ci, wiso.begin());
        }
        h->iso.upload(iso.data(), iso.size());
        h->wiso.upload(wiso.data(), wiso.size());
        upload_fp32(h->iso32, iso);
        upload_fp32(h->wiso32, wiso);
        std::vector<int> bl(size_t(2 * nb));
        for (int64_t b = 0; b < 2 * nb; ++b) bl[size_t(b)] = int(blocks[b]);
        h->blocks.upload(bl.data(), bl.size());
        prepare_frac_constants(h.get(), k_aniso, iso.data());
        *out = h.release();
    });
}

void lar_deconv_kernel_destroy(lar_deconv_kernel kernel) { delete kernel; }

int lar_fit_single_tissue(const double* signals, int64_t v, lar_fod_solver solver, double* fods, uint8_t* status,
                          void* stream) {
    return guarded([&] {
        require(solver != nullptr, "solver must not be NULL");
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(signals && fods, "signals and fods must not be NULL");
        if (solver->kind == 1) {
            if (status) cuda_check(cudaMemsetAsync(status, 0, size_t(v), static_cast<cudaStream_t>(stream)),
                                   "cudaMemsetAsync");
            launch_drl(solver->drl, signals, v, fods, static_cast<cudaStream_t>(stream));
            return;
        }
        const int m = int(solver->host.m), c = int(solver->host.c);
        const RidgeDev R = solver->view();
        const NnlsLaunch nn = nnls_variant(c);
        const size_t smem = nnls_smem_bytes(c, nn.cap) * kMtWarps;
        const int64_t n_max = std::min<int64_t>(v, std::max<int64_t>(4096, int64_t((size_t(2) << 30) / (size_t(c) * 8))));
        const int64_t slots = resident_slots(nn.kernel, smem, n_max, "sd.nnls.ctas_per_sm");
        const size_t slot = nnls_slot_doubles(m, nn.cap);
        auto carve_all = [&](Carver& cv, int*& counters, double*& corr, double*& work) {
            counters = cv.take<int>(8);
            corr = cv.take<double>(size_t(n_max) * c);
            work = cv.take<double>(size_t(slots) * slot);
        };
        int* counters = nullptr;
        double *corr = nullptr, *work = nullptr;
        Carver sizing{nullptr};
        carve_all(sizing, counters, corr, work);
        Carver cv{static_cast<char*>(solver->reserve(sizing.used))};
        carve_all(cv, counters, corr, work);
        auto st = static_cast<cudaStream_t>(stream);
        for (int64_t v0 = 0; v0 < v; v0 += n_max) {
            const int64_t n = std::min(n_max, v - v0);
            const SignalDev S{signals + v0 * m, nullptr, nullptr, nullptr, m, 0};
            launch_correlate(S, nullptr, n, nullptr, R, corr, c, st);
            if (status) cuda_check(cudaMemsetAsync(status + v0, 0, size_t(n), st), "cudaMemsetAsync");
            cuda_check(cudaMemsetAsync(counters, 0, sizeof(int), st), "cudaMemsetAsync");
            const unsigned nb = unsigned(std::max<int64_t>(1, std::min<int64_t>(slots / kMtWarps, (n + kMtWarps - 1) / kMtWarps)));
            LaunchScope scope(nn.name, st);
            nn.kernel<<<nb, kMtWarps * 32, smem, st>>>(R, S, nullptr, n, nullptr, corr, c, fods + v0 * c, c,
                                                       status ? status + v0 : nullptr, counters, work, slot);
            cuda_check(cudaGetLastError(), "ridge_nnls_kernel launch");
        }
    });
}

}  // extern "C"
