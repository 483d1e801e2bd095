// Least squares with inequality constraints (MSMT-CSD) on the GPU, one warp per voxel.
//
// Follows cpp/src/sd/lsi.cpp. The design is prepared once on the host in FP64 (make_lsi_design
// :75-125, host_la.hpp): q_t (n x m), back = P R^-1 (n x n), E = G P R^-1 with unit rows
// (k x n), its Gram E E^T (k x k) and absolute row sums. Per voxel (solve_lsi_by :301-338):
//   rotated = q_t s; f = -E rotated scaled to max |f| = 1 (or the unconstrained solution when
//   f = 0); the LDP multipliers u >= 0 by the Lawson-Hanson steps on H = E E^T + f f^T with a
//   growing Cholesky factor and Givens downdates (ldp_multipliers :253-297: the steepest
//   inactive gradient f (1 - f.u) - E E^T u enters, the first on a tie; a pivot below 1e-12 of
//   its diagonal or more than 3 k inner steps sends the voxel to the fallback); the fallback is
//   the QR-based NNLS on the explicit [E^T; f^T] (warp_nnls.cuh); then
//   x = back (scale E^T u / (1 - f.u) + rotated).
//
// Work distribution, four launches on the stream:
//   rows_product_kernel    rotated = q_t s for every voxel (a tiled FP64 product), left in x;
//   lsi_group_kernel       the LDP steps, a group of warps per voxel (see below), x <- scale E^T u /
//                          (1 - f.u) + rotated; a voxel whose factor fails is marked and listed;
//   lsi_group_kernel<.., QR>  the listed voxels (and those past the list's end), with orthonormal rows instead of the
//                          Cholesky factor; what it cannot take either stays marked for
//   lsi_kernel             one warp per marked voxel by the QR-based NNLS (warp_nnls.cuh), also
//                          the whole fit where the group kernel's shared memory does not hold the
//                          problem or only_qr asks for it;
//   rows_product_kernel    x = back x, in place.

#include <algorithm>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "common.cuh"
#include "host_la.hpp"
#include "plain_fp32.cuh"
#include "warp_chol.cuh"
#include "warp_nnls.cuh"

namespace lar {

namespace {

constexpr int kLsiWarps = 4;
constexpr int kFactorCap = 64;   // active columns the Cholesky factor can hold (>= n + 1)
constexpr double kMinRelativePivot = 1e-12;
constexpr uint8_t kMarked = 2;     // converged[] of a voxel still to be fitted by a fallback
constexpr uint8_t kUnlisted = 3;   // the same, for the QR variant, past what its list holds
constexpr int kColsPerLane = 16;  // constraint columns a lane holds gradients for (k <= 512)

struct LsiDevice {
    int m, n, k;
    const double* qt;      // (m, n): q_t transposed, row j holds column j of q_t
    const double* back;    // (n, n)
    const double* et;      // (n, k): E transposed
    const double* e;       // (k, n)
    const double* gram;    // (k, k)
    const double* abs_sums;  // (k,)
};

// Global scratch of one warp: the Cholesky factor and its inverse, the QR-based fallback's
// explicit matrix and workspaces.
inline size_t lsi_slot_doubles(int n, int k) {
    return 2 * size_t(packed_size(kFactorCap))  // L, M
           + 2 * size_t(k)                  // fallback u, z
           + size_t(n + 1) * k              // fallback matrix
           + size_t(kFactorCap) * (n + 1)   // fallback QR columns
           + (size_t(k) + 7) / 8            // fallback flags
           + 64;
}

// Shared memory of one warp: bounds f, multipliers u, candidate z (k each), the factor's vectors
// h, w, y (cap each), small vectors, then the int and byte arrays.
struct LsiWarpLayout {
    int k, cap;
    __host__ __device__ size_t doubles() const { return 3 * size_t(k) + 3 * size_t(cap) + 4 * 64; }
    __host__ __device__ size_t ints() const { return 2 * size_t(cap) + 2 * 64 + 8; }
    __host__ __device__ size_t bytes() const {
        return (doubles() * sizeof(double) + ints() * sizeof(int) + size_t(k) + 15) / 16 * 16;
    }
};

struct LsiWarp {
    double *f, *u, *z, *h, *wv, *y, *L, *M, *rot, *t, *d, *res;
    int *cols, *sorted, *act, *perm;
    int* n_act;
    uint8_t* flag;
};

__device__ LsiWarp carve_lsi(unsigned char* base, const LsiWarpLayout& lay) {
    LsiWarp w;
    double* p = reinterpret_cast<double*>(base);
    w.f = p; p += lay.k;
    w.u = p; p += lay.k;
    w.z = p; p += lay.k;
    w.h = p; p += lay.cap;
    w.wv = p; p += lay.cap;
    w.y = p; p += lay.cap;
    w.L = nullptr;  // in the warp's global slot
    w.M = nullptr;
    w.rot = p; p += 64;
    w.t = p; p += 64;
    w.d = p; p += 64;
    w.res = p; p += 64;
    int* q = reinterpret_cast<int*>(p);
    w.cols = q; q += lay.cap;
    w.sorted = q; q += lay.cap;
    w.act = q; q += 64;
    w.perm = q; q += 64;
    w.n_act = q; q += 8;
    w.flag = reinterpret_cast<uint8_t*>(q);
    return w;
}

// The small per-warp QR state of the fallback.
struct LsiQrShared {
    double tau[kFactorCap], nu[kFactorCap], nd[kFactorCap], rv[kFactorCap + 1];
};

// The LDP multipliers (cpp/src/sd/lsi.cpp:253-297) in w.u. Returns false when a Cholesky pivot
// fails or the inner steps run out (the caller falls back to the QR-based NNLS). The factor of
// H_AA is kept with its inverse (warp_chol.cuh, InvFactor): y = M f_A grows with each append, a
// solve is one triangular matrix-vector product, and a removal is the Givens downdate of both.
// Inlined into the kernel with every argument by value, so that its state stays in registers.
template <int CPL>
__device__ __forceinline__ bool ldp_multipliers(const LsiDevice D, const LsiWarp w, int cap, int* outer_steps,
                                                int lane) {
    constexpr int VPL = kFactorCap / 32;
    const int k = D.k;
    const InvFactor fac{w.L, w.M, w.h, w.wv, w.y, w.cols, cap};
    double norm1 = 0.0;
    for (int j = lane; j < k; j += 32) {
        norm1 = fmax(norm1, D.abs_sums[j] + fabs(w.f[j]));
        w.u[j] = 0.0;
        w.z[j] = 0.0;
        w.flag[j] = 0;
    }
    norm1 = warp_max(norm1);
    const double tol = 10.0 * kEps64 * norm1 * double(max(D.n + 1, k));
    const int max_inner = 3 * k;
    int na = 0, inner = 0, outer = 0;
    __syncwarp();
    auto solve = [&]() {
        if (na <= 32) inv_solve<1>(fac, na, w.z, k, lane);
        else inv_solve<VPL>(fac, na, w.z, k, lane);
    };
    for (;;) {
        double fu = 0.0;
        for (int j = lane; j < k; j += 32) fu += w.f[j] * w.u[j];
        fu = warp_sum(fu);
        // Steepest inactive gradient f (1 - f.u) - sum_c u_c (E E^T)_c over the active columns in
        // increasing order (u is zero elsewhere), the first on a tie.
        double g[CPL];
#pragma unroll
        for (int t = 0; t < CPL; ++t) {
            const int j = lane + 32 * t;
            g[t] = j < k ? w.f[j] * (1.0 - fu) : 0.0;
        }
        for (int q = 0; q < na; ++q) {
            const int c = w.sorted[q];
            const double uc = w.u[c];
            if (uc == 0.0) continue;
            const double* row = D.gram + size_t(c) * k;
#pragma unroll
            for (int t = 0; t < CPL; ++t) {
                const int j = lane + 32 * t;
                if (j < k) g[t] -= uc * row[j];
            }
        }
        double bv = 0.0;
        int bi = -1;
#pragma unroll
        for (int t = 0; t < CPL; ++t) {
            const int j = lane + 32 * t;
            if (j < k && !w.flag[j] && (bi < 0 || g[t] > bv)) { bv = g[t]; bi = j; }
        }
        const int e = warp_argmax_first(bv, bi);
        const double ge = e >= 0 ? __shfl_sync(0xffffffffu, bv, e & 31) : 0.0;
        if (e < 0 || ge <= tol) break;
        ++outer;
        // H(cols[r], e) = (E E^T)(cols[r], e) + f_cols[r] f_e, then append.
        const double fe = w.f[e];
        for (int r = lane; r < na; r += 32) {
            const int c = w.cols[r];
            w.h[r] = D.gram[size_t(c) * k + e] + w.f[c] * fe;
        }
        __syncwarp();
        const double hee = D.gram[size_t(e) * k + e] + fe * fe;
        const bool appended = na < 32 ? inv_append<1>(fac, na, hee, fe, e, kMinRelativePivot, lane)
                                      : inv_append<VPL>(fac, na, hee, fe, e, kMinRelativePivot, lane);
        if (!appended) {
            *outer_steps = outer;
            return false;
        }
        if (lane == 0) {
            w.flag[e] = 1;
            int q = na - 1;
            while (q > 0 && w.sorted[q - 1] > e) { w.sorted[q] = w.sorted[q - 1]; --q; }
            w.sorted[q] = e;
        }
        __syncwarp();
        solve();
        for (;;) {
            // Blocking step over active columns with z <= 0, the first on a tie.
            double sv = 0.0;
            int si = -1;
            for (int q = lane; q < na; q += 32) {
                const int col = w.sorted[q];
                if (w.z[col] > 0.0) continue;
                const double dist = w.u[col] - w.z[col];
                const double st = dist > 0.0 ? w.u[col] / dist : 0.0;
                if (si < 0 || st < sv) { sv = st; si = col; }
            }
            double step;
            const int b = warp_argmin_first(sv, si, &step);
            if (b < 0) break;
            if (++inner > max_inner) {
                *outer_steps = outer;
                return false;
            }
            for (int q = lane; q < na; q += 32) {
                const int col = w.sorted[q];
                w.u[col] += step * (w.z[col] - w.u[col]);
            }
            __syncwarp();
            // The blocking coefficient leaves, and so does any that rounding left near zero.
            if (lane == 0) {
                w.u[b] = 0.0;
                int kept = 0;
                for (int q = 0; q < na; ++q) {
                    const int col = w.sorted[q];
                    if (col == b || fabs(w.u[col]) < tol) {
                        w.flag[col] = 0;
                        w.u[col] = 0.0;
                    } else {
                        w.sorted[kept++] = col;
                    }
                }
            }
            __syncwarp();
            // keep(): drop the factor columns that left, from the last position to the first.
            for (int pos = na - 1; pos >= 0; --pos) {
                if (w.flag[w.cols[pos]]) continue;
                if (na <= 32) inv_remove<1>(fac, na, pos, lane);
                else inv_remove<VPL>(fac, na, pos, lane);
                --na;
                __syncwarp();
            }
            solve();
        }
        for (int j = lane; j < k; j += 32) w.u[j] = w.z[j];
        __syncwarp();
    }
    *outer_steps = outer;
    return true;
}

template <int CPL>
__global__ void __launch_bounds__(kLsiWarps * 32, 4) lsi_kernel(LsiDevice D, const double* __restrict__ signals,
                                                             int64_t v, int only_qr, int marked, int* queue, int cap,
                                                             double* __restrict__ workspace, size_t slot_doubles,
                                                             double* __restrict__ x, uint8_t* __restrict__ converged,
                                                             uint8_t* __restrict__ status,
                                                             int32_t* __restrict__ outer_out,
                                                             uint8_t* __restrict__ active_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ LsiQrShared qr_shared[kLsiWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LsiWarpLayout lay{D.k, cap};
    LsiQrShared& qsh = qr_shared[warp];
    const int m = D.m, n = D.n, k = D.k, rows = n + 1;
    double* slot = workspace + (size_t(blockIdx.x) * kLsiWarps + warp) * slot_doubles;
    LsiWarp w = carve_lsi(smem_raw + warp * lay.bytes(), lay);
    w.L = slot;
    w.M = slot + packed_size(kFactorCap);
    double* u2 = w.M + packed_size(kFactorCap);
    double* z2 = u2 + k;
    double* cmat = z2 + k;                        // (rows, k)
    double* sub = cmat + size_t(rows) * k;        // (kFactorCap, rows)
    uint8_t* flag2 = reinterpret_cast<uint8_t*>(sub + size_t(kFactorCap) * rows);
    // marked: only the voxels a group kernel left marked, looked for 32 at a time.
    int64_t first = 0;
    unsigned todo = 0u;
    for (;;) {
        if (todo == 0u) {
            if (lane == 0) first = atomicAdd(queue, marked ? 32 : 1);
            first = __shfl_sync(0xffffffffu, first, 0);
            if (first >= v) break;
            todo = marked ? __ballot_sync(0xffffffffu, first + lane < v && converged[first + lane] == kMarked) : 1u;
            if (todo == 0u) continue;
        }
        const int64_t voxel = first + __ffs(todo) - 1;
        todo &= todo - 1u;
        const double* s = signals + voxel * m;
        // rotated = q_t s.
        for (int i = lane; i < n; i += 32) {
            double acc = 0.0;
            for (int j = 0; j < m; ++j) acc += D.qt[size_t(j) * n + i] * s[j];
            w.rot[i] = acc;
        }
        __syncwarp();
        // f = -E rotated, scaled by max |f|.
        double scale = 0.0;
        for (int j = lane; j < k; j += 32) {
            double acc = 0.0;
            for (int i = 0; i < n; ++i) acc += D.et[size_t(i) * k + j] * w.rot[i];
            w.f[j] = -acc;
            scale = fmax(scale, fabs(acc));
        }
        scale = warp_max(scale);
        __syncwarp();
        uint8_t st = 0, conv = 1;
        int outer = 0;
        if (!(scale > 0.0)) {
            // f = 0: the unconstrained solution back * rotated.
            for (int i = lane; i < n; i += 32) {
                double acc = 0.0;
                for (int j = 0; j < n; ++j) acc += D.back[size_t(i) * n + j] * w.rot[j];
                x[voxel * n + i] = acc;
            }
            if (active_out)
                for (int j = lane; j < k; j += 32) active_out[voxel * k + j] = 0;
            st = 2;
        } else {
            for (int j = lane; j < k; j += 32) w.f[j] /= scale;
            __syncwarp();
            const double* mult = w.u;
            const bool fast = !only_qr && ldp_multipliers<CPL>(D, w, cap, &outer, lane);
            if (!fast) {
                // QR-based NNLS on the explicit [E^T; f^T] (cpp/src/sd/lsi.cpp:321-332).
                double colmax = 0.0;
                for (int j = lane; j < k; j += 32) {
                    double cs = fabs(w.f[j]);
                    for (int i = 0; i < n; ++i) {
                        const double eij = D.e[size_t(j) * n + i];
                        cmat[size_t(i) * k + j] = eij;
                        cs += fabs(eij);
                    }
                    cmat[size_t(n) * k + j] = w.f[j];
                    colmax = fmax(colmax, cs);
                }
                colmax = warp_max(colmax);
                for (int r = lane; r < rows; r += 32) w.d[r] = (r == n) ? 1.0 : 0.0;
                __syncwarp();
                const double tol = 10.0 * kEps64 * colmax * double(max(rows, k));
                NnlsScratch ns{u2, z2, flag2, w.act, w.n_act, w.res,
                               QrScratch{sub, qsh.tau, qsh.nu, qsh.nd, w.perm, qsh.rv}, kFactorCap};
                const int outcome = warp_nnls_explicit(cmat, rows, k, w.d, tol, 3 * k, ns, lane);
                conv = outcome == 1 ? 1 : 0;
                if (outcome < 0)
                    for (int j = lane; j < k; j += 32) u2[j] = 0.0;
                __syncwarp();
                mult = u2;
                st = 1;
            }
            // x = back (scale E^T u / (1 - f.u) + rotated).
            double fu = 0.0;
            for (int j = lane; j < k; j += 32) fu += w.f[j] * mult[j];
            fu = warp_sum(fu);
            for (int i = lane; i < n; i += 32) {
                double acc = 0.0;
                for (int j = 0; j < k; ++j) {
                    const double mj = mult[j];
                    if (mj != 0.0) acc += D.e[size_t(j) * n + i] * mj;
                }
                w.t[i] = scale * acc / (1.0 - fu) + w.rot[i];
            }
            __syncwarp();
            for (int i = lane; i < n; i += 32) {
                double acc = 0.0;
                for (int j = 0; j < n; ++j) acc += D.back[size_t(i) * n + j] * w.t[j];
                x[voxel * n + i] = acc;
            }
            if (active_out)
                for (int j = lane; j < k; j += 32) active_out[voxel * k + j] = mult[j] != 0.0 ? 1 : 0;
        }
        if (lane == 0) {
            converged[voxel] = conv;
            if (status) status[voxel] = st;
            if (outer_out && !marked) outer_out[voxel] = outer;
        }
        __syncwarp();
    }
}

// ---- the group kernel ----------------------------------------------------------------------
//
// What bounds it: the gradients E (E^T u), 302 x 47 entries in each of ~120 steps per voxel. Read as
// active rows of the 302 x 302 Gram matrix they were 13.9 MB of L2 reads per voxel at their
// latency (lsi_kernel: 19 M cycles per voxel and warp; 484 ms for 100,003 voxels of 47 unknowns and
// 302 constraints, 19.3 ms for 4,099). Here E^T (114 KB) and eight voxels' whole state (14.7 KB
// each) stay in one SM's shared memory: 98.5 ms and 4.9 ms, bound by the shared-memory bandwidth
// of the gradients (~2,000 wavefronts per step, two thirds of them E). Four voxels taking their
// gradients together read E a quarter as often, but waited for one another: 120 ms.
// NW warps share a voxel and split every loop of a step, meeting at named barriers: the QR variant
// takes few voxels, each the length of its chain of steps (2.0 ms on one warp, 1.5 ms on eight;
// lsi_kernel's QR from scratch in every step took 130 ms).
//
// The factor is kept as M = L^-1 alone (packed rows; a row's offset r (r + 1) / 2 puts 16
// consecutive rows of one column in 16 different banks), with y = M f_A and z = M^T y:
// - appending column e: w = M h, d^2 = h_ee - w.w, M's new row [-(w^T M) / d, 1 / d], y_e =
//   (f_e - w.y) / d, z += y_e (new row): the solve is part of the append, in the same order of sums;
// - removing position p: the rotations of rows (k, k + 1) that clear column p of M from the top
//   down have c_k = M(k+1, p) / t_{k+1}, s_k = t_k / t_{k+1}, t_k^2 = sum_{i <= k} M(i, p)^2: one
//   prefix sum and one reciprocal root per lane instead of a chain of hypots, then each lane
//   runs the chain of its own columns.
// With QR, rows Q of an orthonormal basis of the active columns [E_c; f_c] stand beside M: w = Q c
// and the new row is c - Q^T w, orthogonalised twice, so the pivot loses nothing to cancellation.

constexpr int kGroupNW = 1;       // warps per voxel (2: 102 ms on the volume below, 4: 135 ms)
constexpr int kGroups = 8;        // voxels per CTA (one CTA per SM)
constexpr int kQrNW = 8;          // the QR variant: one voxel per CTA
// Voxels the QR variant's list holds (its size does not grow with the call, so that a captured call needs no larger
// scratch); it looks the others up by their mark, so that they are fitted the same way.
constexpr int kRedoCap = 1 << 16;
constexpr double kQrMinPivot = 1e-26;  // squared, relative: below it a column is dependent

struct GroupLayout {
    int n, k, nw, groups;
    bool qr;
    __host__ __device__ int cap() const { return n + 1; }
    __host__ __device__ int kp() const { return k | 1; }       // odd: a column of E^T is conflict-free too
    __host__ __device__ int ldq() const { return (n + 1) | 1; }
    __host__ __device__ int mask_words() const { return (k + 31) / 32; }
    __host__ __device__ size_t voxel_doubles() const {
        const size_t q = qr ? size_t(cap()) * ldq() + n + 1 : 0;
        return size_t(cap()) * (cap() + 1) / 2 + k + 5 * size_t(cap()) + size_t(nw) * cap() + nw + q;
    }
    __host__ __device__ size_t int_off() const { return size_t(n) * kp() + size_t(groups) * voxel_doubles(); }
    __host__ __device__ size_t bytes() const {
        return int_off() * sizeof(double) + size_t(groups) * (nw + cap() + mask_words() + 1) * sizeof(int);
    }
};

// A voxel in shared memory.
struct GroupVoxel {
    double *M, *f, *fpos, *u, *z, *y, *w, *part, *best_v, *Q, *cv;
    int *best_i, *cols, *ticket;
    unsigned* mask;  // active constraints, a bit each
};

__device__ __forceinline__ int tri(int r) { return r * (r + 1) / 2; }

// A warp's place: lane, warp in the group, group in the CTA.
template <int NW>
struct Place {
    int lane, wig, group;
    __device__ __forceinline__ void sync() const {
        if constexpr (NW == 1)
            __syncwarp();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(NW * 32) : "memory");
    }
};

// The group's sum over its warps of each warp's a[t] (entry lane + 32 t), in every warp: through
// g.part (two entries per lane, na <= 64), with the barrier that makes it visible.
template <int NW>
__device__ __forceinline__ void group_sum(const GroupVoxel& g, int cap, int na, const Place<NW>& at, double (&a)[2]) {
    if constexpr (NW > 1) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (at.lane + 32 * t < na) g.part[at.wig * cap + at.lane + 32 * t] = a[t];
        at.sync();
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            if (at.lane + 32 * t >= na) continue;
            double s = g.part[at.lane + 32 * t];
#pragma unroll
            for (int q = 1; q < NW; ++q) s += g.part[q * cap + at.lane + 32 * t];
            a[t] = s;
        }
    }
}

// This warp's share of M h (rows lane + 32 t): the columns j = wig, wig + NW, ..., h in g.w.
template <int NW>
__device__ __forceinline__ void tri_rows(const GroupVoxel& g, int na, const Place<NW>& at, double (&w)[2]) {
    w[0] = w[1] = 0.0;
    const int lane = at.lane;
    const double* row0 = g.M + tri(lane);
    const int low = lane < na ? lane : -1;
#pragma unroll 4
    for (int j = at.wig; j < na; j += NW)
        if (j <= low) w[0] = fma(row0[j], g.w[j], w[0]);
    if (na > 32) {
        const double* row1 = g.M + tri(lane + 32);
        const int high = lane + 32 < na ? lane + 32 : -1;
#pragma unroll 4
        for (int j = at.wig; j < na; j += NW)
            if (j <= high) w[1] = fma(row1[j], g.w[j], w[1]);
    }
}

// This warp's share of v^T M (columns lane + 32 t): the rows r = wig, wig + NW, ...
template <int NW>
__device__ __forceinline__ void tri_columns(const GroupVoxel& g, const double* v, int na, const Place<NW>& at,
                                            double (&out)[2]) {
    out[0] = out[1] = 0.0;
    const int lane = at.lane;
#pragma unroll 4
    for (int r = at.wig; r < na; r += NW)
        if (lane <= r) out[0] = fma(g.M[tri(r) + lane], v[r], out[0]);
    if (na > 32) {
#pragma unroll 4
        for (int r = 32 + (at.wig - 32 % NW + NW) % NW; r < na; r += NW)
            if (lane + 32 <= r) out[1] = fma(g.M[tri(r) + lane + 32], v[r], out[1]);
    }
}

// Appends constraint e (value f_e) to the factor; false, leaving it as it was, on a pivot that is
// not above the limit. g.z grows to the fit on the larger set.
template <bool QR, int NW>
__device__ __forceinline__ bool group_append(const LsiDevice& D, const GroupLayout& lay, const double* et,
                                             const GroupVoxel& g, int& na, int e, const Place<NW>& at) {
    const int n = D.n, kp = lay.kp(), cap = lay.cap(), lane = at.lane;
    const double fe = g.f[e];
    const double hee = D.gram[size_t(e) * D.k + e] + fe * fe;
    if (na >= cap) return false;
    double w[2], d2, ye;
    if constexpr (!QR) {
        // H(cols[r], e) = (E E^T)(cols[r], e) + f_cols[r] f_e, the Gram matrix's row e: each warp the
        // entries its share of M h reads.
        const double* row = D.gram + size_t(e) * D.k;
        for (int r = lane * NW + at.wig; r < na; r += 32 * NW) g.w[r] = row[g.cols[r]] + g.fpos[r] * fe;
        __syncwarp();
        tri_rows<NW>(g, na, at, w);
        group_sum<NW>(g, cap, na, at, w);
        double sq = 0.0, wy = 0.0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int r = lane + 32 * t;
            if (r < na) {
                g.w[r] = w[t];  // every warp writes the same values: the h there are all read
                sq = fma(w[t], w[t], sq);
                wy = fma(w[t], g.y[r], wy);
            }
        }
        sq = warp_sum(sq);
        wy = warp_sum(wy);
        d2 = hee - sq;
        if (!(d2 > kMinRelativePivot * hee)) return false;
        ye = fe - wy;
    } else {
        const int rows = n + 1, ldq = lay.ldq();
        for (int i = lane + 32 * at.wig; i < rows; i += 32 * NW) g.cv[i] = i < n ? et[size_t(i) * kp + e] : fe;
        w[0] = w[1] = 0.0;
        at.sync();
        for (int pass = 0; pass < 2; ++pass) {
            double p[2] = {0.0, 0.0};
            for (int i = at.wig; i < rows; i += NW) {
                const double c = g.cv[i];
                if (lane < na) p[0] = fma(g.Q[lane * ldq + i], c, p[0]);
                if (lane + 32 < na) p[1] = fma(g.Q[(lane + 32) * ldq + i], c, p[1]);
            }
            group_sum<NW>(g, cap, na, at, p);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (lane + 32 * t < na) g.w[lane + 32 * t] = p[t];
                w[t] += p[t];
            }
            at.sync();
            double c[2] = {0.0, 0.0};
            for (int r = at.wig; r < na; r += NW) {
                const double pr = g.w[r];
                if (lane < rows) c[0] = fma(-g.Q[r * ldq + lane], pr, c[0]);
                if (lane + 32 < rows) c[1] = fma(-g.Q[r * ldq + lane + 32], pr, c[1]);
            }
            group_sum<NW>(g, cap, rows, at, c);
            at.sync();
            if (at.wig == 0) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (lane + 32 * t < rows) g.cv[lane + 32 * t] += c[t];
            }
            at.sync();
        }
        d2 = 0.0;
        for (int i = lane; i < rows; i += 32) d2 = fma(g.cv[i], g.cv[i], d2);
        d2 = warp_sum(d2);
        if (!(d2 > kQrMinPivot * hee)) return false;
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (lane + 32 * t < na) g.w[lane + 32 * t] = w[t];
        ye = g.cv[n];  // the right-hand side is the last unit vector
    }
    const double inv_d = rsqrt(d2);
    ye *= inv_d;
    at.sync();  // w is whole, and g.part read
    double row[2];
    tri_columns<NW>(g, g.w, na, at, row);
    group_sum<NW>(g, cap, na, at, row);
    double* mrow = g.M + tri(na);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int j = lane + 32 * t;
        if (j < na && (NW == 1 || at.wig == t)) {
            const double v = -row[t] * inv_d;
            mrow[j] = v;
            g.z[j] = fma(v, ye, g.z[j]);
        }
    }
    if constexpr (QR) {
        double* q = g.Q + na * lay.ldq();
        for (int i = lane + 32 * at.wig; i <= n; i += 32 * NW) q[i] = g.cv[i] * inv_d;
    }
    if (lane == 0 && at.wig == 0) {
        mrow[na] = inv_d;
        g.z[na] = inv_d * ye;
        g.y[na] = ye;
        g.u[na] = 0.0;
        g.fpos[na] = fe;
        g.cols[na] = e;
        g.mask[e >> 5] |= 1u << (e & 31);
    }
    ++na;
    at.sync();
    return true;
}

// Removes position p of the factor's na columns (z is left to the caller). The group has synchronised
// before; it synchronises at the end.
template <bool QR, int NW>
__device__ __forceinline__ void group_remove(const GroupLayout& lay, const GroupVoxel& g, int na, int p,
                                             const Place<NW>& at) {
    const int lane = at.lane;
    // t_k^2 over rows p..na-1 of column p, the prefix sums of its squares (every warp its own).
    double v[2], s[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int i = p + lane + 32 * t;
        v[t] = i < na ? g.M[tri(i) + p] : 0.0;
        s[t] = v[t] * v[t];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, s[0], o);
        if (lane >= o) s[0] += a;
    }
    if (na - p > 32) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double b = __shfl_up_sync(0xffffffffu, s[1], o);
            if (lane >= o) s[1] += b;
        }
        s[1] += __shfl_sync(0xffffffffu, s[0], 31);
    }
    double rt[2], tt[2];
    rt[0] = rsqrt(s[0]);
    tt[0] = s[0] * rt[0];
    rt[1] = tt[1] = 0.0;
    if (na - p > 32) {
        rt[1] = rsqrt(s[1]);
        tt[1] = s[1] * rt[1];
    }
    const double last = __shfl_sync(0xffffffffu, tt[0], 31);
    // Entry k of w and part: c and s of the rotation of rows (k, k + 1), k = p..na-2 (every warp
    // writes the same values); cols, fpos and u move up.
    int c0[2];
    double f0[2], u0[2], a[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        double before = __shfl_up_sync(0xffffffffu, tt[t], 1);
        if (t == 1 && lane == 0) before = last;
        const int k = p + lane + 32 * t - 1;
        if (k >= p && k < na - 1) {
            g.w[k] = v[t] * rt[t];
            g.part[k] = before * rt[t];
        }
        const int q = lane + 32 * t;
        const bool mv = q >= p && q < na - 1;
        c0[t] = mv ? g.cols[q + 1] : 0;
        f0[t] = mv ? g.fpos[q + 1] : 0.0;
        u0[t] = mv ? g.u[q + 1] : 0.0;
        a[t] = q <= p ? g.M[tri(p) + q] : 0.0;
    }
    double ya = g.y[p];
    const int rows = lay.n + 1, ldq = lay.ldq();
    at.sync();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int q = lane + 32 * t;
        if (q >= p && q < na - 1 && (NW == 1 || at.wig == t)) {
            g.cols[q] = c0[t];
            g.fpos[q] = f0[t];
            g.u[q] = u0[t];
        }
    }
    // Column j's chain: row k's new entry is s_k x - c_k v from x = M(k + 1, j) and the carried v, which
    // becomes s_k v + c_k x. Columns 0..31 on warp 0, the others on the last warp. A warp writes row k
    // after reading row k + 1; column 32 becomes column 31, which warp 0 still reads, so with several
    // warps its entries wait in part until the chains have ended.
    if (at.wig == 0 || (at.wig == NW - 1 && na > 32)) {
        const bool first = NW == 1 || at.wig == 0, second = NW == 1 ? na > 32 : at.wig != 0;
        for (int k = p; k < na - 1; ++k) {
            const double c = g.w[k], sn = g.part[k];
            const double* below = g.M + tri(k + 1);
            double* row = g.M + tri(k);
            double x[2] = {0.0, 0.0};
            if (first && lane <= k + 1) x[0] = below[lane];
            if (second && lane + 32 <= k + 1) x[1] = below[lane + 32];
            __syncwarp();
            if (first) {
                if (lane <= k + 1 && lane != p) row[lane < p ? lane : lane - 1] = sn * x[0] - c * a[0];
                a[0] = sn * a[0] + c * x[0];
            }
            if (second) {
                if (lane + 32 <= k + 1 && lane + 32 != p) {
                    const double out = sn * x[1] - c * a[1];
                    if (NW > 1 && lane == 0 && p < 32)
                        g.part[lay.cap() + k] = out;
                    else
                        row[lane + 32 < p ? lane + 32 : lane + 31] = out;
                }
                a[1] = sn * a[1] + c * x[1];
            }
        }
    }
    if (at.wig == NW / 2 && lane == 0) {
        for (int k = p; k < na - 1; ++k) {
            const double c = g.w[k], sn = g.part[k], yx = g.y[k + 1];
            g.y[k] = sn * yx - c * ya;
            ya = sn * ya + c * yx;
        }
    }
    if constexpr (QR) {
        for (int i = lane + 32 * at.wig; i < rows; i += 32 * NW) {
            double qa = g.Q[p * ldq + i];
            for (int k = p; k < na - 1; ++k) {
                const double c = g.w[k], sn = g.part[k], qx = g.Q[(k + 1) * ldq + i];
                g.Q[k * ldq + i] = sn * qx - c * qa;
                qa = sn * qa + c * qx;
            }
        }
    }
    at.sync();
    if (NW > 1 && na > 32 && p < 32) {
        const int k = 31 + lane;
        if (at.wig == 0 && k >= p && k < na - 1) g.M[tri(k) + 31] = g.part[lay.cap() + k];
        at.sync();
    }
}

// The steps of a fit once a constraint has joined (cpp/src/sd/lsi.cpp:270-295): while some
// candidate is not positive, move to the first blocking step, drop what reached zero, fit again;
// then u = z. False when the inner steps run out.
template <bool QR, int NW>
__device__ __forceinline__ bool group_inner(const GroupLayout& lay, const GroupVoxel& g, int& na, int& inner,
                                            int max_inner, double tol, const Place<NW>& at) {
    const int lane = at.lane;
    for (;;) {
        // Every warp takes the same decisions from the same values; warp t writes entry slice t.
        double sv = 0.0, u[2], z[2];
        int si = -1, col[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int q = lane + 32 * t;
            const bool in = q < na;
            u[t] = in ? g.u[q] : 0.0;
            z[t] = in ? g.z[q] : 1.0;
            col[t] = in ? g.cols[q] : -1;
            if (in && !(z[t] > 0.0)) {
                const double dist = u[t] - z[t];
                const double st = dist > 0.0 ? u[t] / dist : 0.0;
                if (si < 0 || st < sv || (st == sv && col[t] < si)) {
                    sv = st;
                    si = col[t];
                }
            }
        }
        at.sync();  // every warp has read u and z
        if (!__any_sync(0xffffffffu, si >= 0)) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
                if (lane + 32 * t < na && (NW == 1 || at.wig == t)) g.u[lane + 32 * t] = z[t];
            at.sync();
            return true;
        }
        if (++inner > max_inner) return false;
        double step;
        const int b = warp_argmin_first(sv, si, &step);
        unsigned gone[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int q = lane + 32 * t;
            bool drop = false;
            if (q < na) {
                u[t] += step * (z[t] - u[t]);
                drop = col[t] == b || fabs(u[t]) < tol;
                if (NW == 1 || at.wig == t) g.u[q] = u[t];
            }
            gone[t] = __ballot_sync(0xffffffffu, drop);
            if (drop && at.wig == 0) atomicAnd(&g.mask[col[t] >> 5], ~(1u << (col[t] & 31)));
        }
        at.sync();
        for (int t = 1; t >= 0; --t)
            while (gone[t]) {
                const int bit = 31 - __clz(gone[t]);
                gone[t] ^= 1u << bit;
                group_remove<QR, NW>(lay, g, na, bit + 32 * t, at);
                --na;
            }
        // z = M^T y.
        double zn[2];
        tri_columns<NW>(g, g.y, na, at, zn);
        group_sum<NW>(g, lay.cap(), na, at, zn);
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (lane + 32 * t < na && (NW == 1 || at.wig == t)) g.z[lane + 32 * t] = zn[t];
        at.sync();
    }
}

// x holds the rotated signals and gets scale E^T u / (1 - f.u) + rotated, for all v voxels, or with QR for those of
// `list` (redo_count of them, as many as it holds) and then those marked kUnlisted, 32 voxels to a ticket of queue[2]. K constraints per thread: 32 NW K >= k.
template <int NW, int GROUPS, int K, bool QR>
__global__ void __launch_bounds__(NW * GROUPS * 32, 1) lsi_group_kernel(
    LsiDevice D, int64_t v, int* queue, int* list, int* list_count, double* __restrict__ x,
    uint8_t* __restrict__ converged, uint8_t* __restrict__ status, int32_t* __restrict__ outer_out,
    uint8_t* __restrict__ active_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* const sm = reinterpret_cast<double*>(smem_raw);
    const int n = D.n, k = D.k;
    const GroupLayout lay{n, k, NW, GROUPS, QR};
    const int kp = lay.kp(), cap = lay.cap(), words = lay.mask_words();
    const int failed = QR ? *list_count : 0;
    if (QR && failed == 0) return;
    const int warp = threadIdx.x >> 5;
    const Place<NW> at{int(threadIdx.x & 31), warp % NW, warp / NW};
    const int lane = at.lane, gtid = at.wig * 32 + lane;
    double* const et = sm;
    GroupVoxel g;
    {
        double* p = sm + size_t(n) * kp + size_t(at.group) * lay.voxel_doubles();
        g.M = p; p += cap * (cap + 1) / 2;
        g.f = p; p += k;
        g.fpos = p; p += cap;
        g.u = p; p += cap;
        g.z = p; p += cap;
        g.y = p; p += cap;
        g.w = p; p += cap;
        g.part = p; p += NW * cap;
        g.best_v = p; p += NW;
        g.Q = p;
        g.cv = p + (QR ? cap * lay.ldq() : 0);
        int* q = reinterpret_cast<int*>(sm + lay.int_off()) + at.group * (NW + cap + words + 1);
        g.best_i = q; q += NW;
        g.cols = q; q += cap;
        g.mask = reinterpret_cast<unsigned*>(q); q += words;
        g.ticket = q;
    }
    for (int i = threadIdx.x; i < n * k; i += blockDim.x) {
        const int r = i / k, c = i - r * k;
        et[size_t(r) * kp + c] = D.et[i];
    }
    __syncthreads();
    const int max_inner = 3 * k;
    bool by_mark = false;
    int64_t first = 0;   // by_mark: the ticket's 32 voxels, and
    unsigned todo = 0u;  // those of them still to be fitted
    for (;;) {
        // The group's next voxel.
        int64_t voxel = first + __ffs(todo) - 1;
        if (todo == 0u) {
            if (gtid == 0) *g.ticket = atomicAdd(by_mark ? queue + 2 : queue, 1);
            at.sync();
            voxel = *g.ticket;
            if constexpr (QR) {
                if (by_mark) {
                    first = 32 * voxel;
                    if (first >= v) break;
                    todo = __ballot_sync(0xffffffffu, first + lane < v && converged[first + lane] == kUnlisted);
                    at.sync();  // every warp has read the ticket and the marks
                    continue;
                }
                if (voxel >= min(failed, kRedoCap)) {
                    if (failed <= kRedoCap) break;
                    by_mark = true;
                    at.sync();
                    continue;
                }
                voxel = list[voxel];
            } else if (voxel >= v) {
                break;
            }
        } else {
            todo &= todo - 1u;
        }
        double rot[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            rot[t] = lane + 32 * t < n ? x[voxel * n + lane + 32 * t] : 0.0;
            if (lane + 32 * t < n) g.z[lane + 32 * t] = rot[t];  // every warp the same (cap > n)
        }
        for (int q = gtid; q < words; q += 32 * NW) g.mask[q] = 0u;
        at.sync();
        // f = -E rotated, scaled by max |f|.
        double scale = 0.0;
        for (int j = gtid; j < k; j += 32 * NW) {
            double acc = 0.0;
#pragma unroll 8
            for (int i = 0; i < n; ++i) acc = fma(et[i * kp + j], g.z[i], acc);
            g.f[j] = -acc;
            scale = fmax(scale, fabs(acc));
        }
        scale = warp_max(scale);
        if (lane == 0) g.best_v[at.wig] = scale;
        at.sync();
#pragma unroll
        for (int q = 0; q < NW; ++q) scale = fmax(scale, g.best_v[q]);
        if (!(scale > 0.0)) {
            // f = 0: the unconstrained solution; x keeps rotated.
            if (active_out)
                for (int j = gtid; j < k; j += 32 * NW) active_out[voxel * k + j] = 0;
            if (gtid == 0) {
                converged[voxel] = 1;
                if (status) status[voxel] = 2;
                if (outer_out) outer_out[voxel] = 0;
            }
            at.sync();
            continue;
        }
        at.sync();  // best_v is read
        double norm1 = 0.0;
        for (int j = gtid; j < k; j += 32 * NW) {
            const double fj = g.f[j] / scale;
            g.f[j] = fj;
            norm1 = fmax(norm1, D.abs_sums[j] + fabs(fj));
        }
        norm1 = warp_max(norm1);
        if (lane == 0) g.best_v[at.wig] = norm1;
        at.sync();
#pragma unroll
        for (int q = 0; q < NW; ++q) norm1 = fmax(norm1, g.best_v[q]);
        const double tol = 10.0 * kEps64 * norm1 * double(max(n + 1, k));
        int na = 0, inner = 0, outer = 0;
        for (;;) {
            // r = E^T u and f.u: each warp its share of the active columns.
            double r[2] = {0.0, 0.0}, fu = 0.0;
            {
                const int i0 = (lane < n ? lane : n - 1) * kp, i1 = (lane + 32 < n ? lane + 32 : n - 1) * kp;
#pragma unroll 4
                for (int q = at.wig; q < na; q += NW) {
                    const int c = g.cols[q];
                    const double uq = g.u[q];
                    r[0] = fma(uq, et[i0 + c], r[0]);
                    r[1] = fma(uq, et[i1 + c], r[1]);
                }
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (lane + 32 * t < na) fu = fma(g.u[lane + 32 * t], g.fpos[lane + 32 * t], fu);
                fu = warp_sum(fu);
            }
            group_sum<NW>(g, cap, n, at, r);
            // The gradient f (1 - f.u) - E E^T u is -E (E^T u + (1 - f.u) / scale rotated); the vector
            // goes to g.w (every warp the same values).
            const double back = (1.0 - fu) / scale;
#pragma unroll
            for (int t = 0; t < 2; ++t)
                if (lane + 32 * t < n) g.w[lane + 32 * t] = fma(back, rot[t], r[t]);
            __syncwarp();
            double bv = 0.0;
            int bi = -1;
            {
                double acc[K];
                int col[K];
#pragma unroll
                for (int t = 0; t < K; ++t) {
                    col[t] = min(gtid + 32 * NW * t, k - 1);
                    acc[t] = 0.0;
                }
#pragma unroll 4
                for (int i = 0; i < n; ++i) {
                    const double rv = g.w[i];
                    const double* ei = et + i * kp;
#pragma unroll
                    for (int t = 0; t < K; ++t) acc[t] = fma(-ei[col[t]], rv, acc[t]);
                }
                // The steepest inactive entry, the first on a tie.
#pragma unroll
                for (int t = 0; t < K; ++t) {
                    const int j = gtid + 32 * NW * t;
                    if (j < k && !((g.mask[j >> 5] >> (j & 31)) & 1u) && (bi < 0 || acc[t] > bv)) {
                        bv = acc[t];
                        bi = j;
                    }
                }
            }
            int e = bi;
            double ge = bv;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, ge, o);
                const int oi = __shfl_xor_sync(0xffffffffu, e, o);
                const bool take = oi >= 0 && (e < 0 || ov > ge || (ov == ge && oi < e));
                ge = take ? ov : ge;
                e = take ? oi : e;
            }
            if constexpr (NW > 1) {
                if (lane == 0) {
                    g.best_v[at.wig] = ge;
                    g.best_i[at.wig] = e;
                }
                at.sync();
                e = -1;
                ge = 0.0;
#pragma unroll
                for (int q = 0; q < NW; ++q) {
                    const double ov = g.best_v[q];
                    const int oi = g.best_i[q];
                    if (oi >= 0 && (e < 0 || ov > ge || (ov == ge && oi < e))) {
                        ge = ov;
                        e = oi;
                    }
                }
            }
            if (e < 0 || ge <= tol) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (lane + 32 * t < n && (NW == 1 || at.wig == t))
                        x[voxel * n + lane + 32 * t] = scale * r[t] / (1.0 - fu) + rot[t];
                if (active_out)
                    for (int j = gtid; j < k; j += 32 * NW)
                        active_out[voxel * k + j] = (g.mask[j >> 5] >> (j & 31)) & 1u;
                if (gtid == 0) {
                    converged[voxel] = 1;
                    if (status) status[voxel] = QR ? 1 : 0;
                    if (outer_out && !QR) outer_out[voxel] = outer;
                }
                break;
            }
            ++outer;
            if (!group_append<QR, NW>(D, lay, et, g, na, e, at) ||
                !group_inner<QR, NW>(lay, g, na, inner, max_inner, tol, at)) {
                if (gtid == 0) {
                    uint8_t mark = kMarked;
                    if (!QR) {
                        if (outer_out) outer_out[voxel] = outer;
                        const int slot = atomicAdd(list_count, 1);
                        if (slot < kRedoCap)
                            list[slot] = int(voxel);
                        else
                            mark = kUnlisted;
                    }
                    converged[voxel] = mark;
                }
                break;
            }
        }
        at.sync();  // the group is done with this voxel's state
    }
}

// out(v, j) = sum_i in(v, i) b(i, j) for 32 rows and all n <= 16 RC columns per CTA, each entry
// summed in increasing i; out may be in (a CTA's rows are read before they are written).
template <int RC>
__global__ void __launch_bounds__(128) rows_product_kernel(const double* in, int64_t v, int m,
                                                           const double* __restrict__ b, int n, double* out) {
    constexpr int kRows = 32, kDepth = 16, TC = 16 * RC;
    __shared__ double a_t[kDepth][kRows + 1];
    __shared__ double b_t[kDepth][TC];
    const int tid = threadIdx.x, tv = tid & 7, tc = tid >> 3;
    const int64_t v0 = int64_t(blockIdx.x) * kRows;
    double acc[4][RC];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < RC; ++q) acc[p][q] = 0.0;
    for (int i0 = 0; i0 < m; i0 += kDepth) {
        const int depth = min(kDepth, m - i0);
        for (int e = tid; e < kRows * kDepth; e += 128) {
            const int r = e / kDepth, i = e % kDepth;
            a_t[i][r] = (v0 + r < v && i < depth) ? in[(v0 + r) * m + i0 + i] : 0.0;
        }
        for (int e = tid; e < kDepth * TC; e += 128) {
            const int i = e / TC, j = e % TC;
            b_t[i][j] = (i < depth && j < n) ? b[size_t(i0 + i) * n + j] : 0.0;
        }
        __syncthreads();
        for (int i = 0; i < depth; ++i) {
            double av[4], bv[RC];
#pragma unroll
            for (int p = 0; p < 4; ++p) av[p] = a_t[i][tv + 8 * p];
#pragma unroll
            for (int q = 0; q < RC; ++q) bv[q] = b_t[i][tc + 16 * q];
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < RC; ++q) acc[p][q] = fma(av[p], bv[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int64_t row = v0 + tv + 8 * p;
        if (row >= v) continue;
#pragma unroll
        for (int q = 0; q < RC; ++q)
            if (tc + 16 * q < n) out[row * n + tc + 16 * q] = acc[p][q];
    }
}

void launch_rows_product(const double* in, int64_t v, int m, const double* b, int n, double* out, cudaStream_t st) {
    LaunchScope scope("rows_product_kernel", st);
    const unsigned grid = unsigned((v + 31) / 32);
    if (n <= 16) rows_product_kernel<1><<<grid, 128, 0, st>>>(in, v, m, b, n, out);
    else if (n <= 32) rows_product_kernel<2><<<grid, 128, 0, st>>>(in, v, m, b, n, out);
    else if (n <= 48) rows_product_kernel<3><<<grid, 128, 0, st>>>(in, v, m, b, n, out);
    else rows_product_kernel<4><<<grid, 128, 0, st>>>(in, v, m, b, n, out);
    cuda_check(cudaGetLastError(), "rows_product_kernel launch");
}

using GroupKernel = void (*)(LsiDevice, int64_t, int*, int*, int*, double*, uint8_t*, uint8_t*, int32_t*, uint8_t*);

// The group kernels of a problem, or null where their shared memory does not hold it or k is past
// their threads' constraints.
struct GroupPlan {
    GroupKernel main = nullptr, qr = nullptr;
    size_t main_smem = 0, qr_smem = 0;
};

GroupPlan group_plan(int n, int k) {
    GroupPlan p;
    constexpr size_t limit = 227 * 1024;
    constexpr int kMainK = (320 + 32 * kGroupNW - 1) / (32 * kGroupNW), kQrK = 2;
    const GroupLayout main{n, k, kGroupNW, kGroups, false}, qr{n, k, kQrNW, 1, true};
    if (k > 320 || main.bytes() > limit || qr.bytes() > limit) return p;
    p.main = lsi_group_kernel<kGroupNW, kGroups, kMainK, false>;
    p.qr = lsi_group_kernel<kQrNW, 1, kQrK, true>;
    p.main_smem = main.bytes();
    p.qr_smem = qr.bytes();
    return p;
}

}  // namespace

}  // namespace lar

struct lar_lsi_design_s {
    lar::host::LsiDesignHost host;
    lar::DeviceArray<double> qt, back, back_t, et, e, gram, abs_sums;
    // FP32 copies for the plain single-precision fit (the comparison baseline).
    lar::DeviceArray<float> qt32, back32, et32, e32, gram32, abs_sums32;
    void* scratch = nullptr;
    size_t scratch_bytes = 0;
    ~lar_lsi_design_s() {
        if (scratch) cudaFree(scratch);
    }
};

using namespace lar;

extern "C" {

int lar_lsi_design_create(const double* a, int64_t m, int64_t n, const double* g, int64_t k, double ridge,
                          lar_lsi_design* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(a != nullptr && m > 0 && n > 0, "a must be a non-empty (m, n) array");
        require(g != nullptr && k > 0, "g must be a non-empty (k, n) array");
        require(n + 1 <= 64, "the LSI fit takes at most 63 parameters");
        require(k <= 512, "the LSI fit takes at most 512 constraints");
        require(m <= (int64_t(1) << 20) && k <= (int64_t(1) << 16), "the LSI design is too large");
        auto h = std::make_unique<lar_lsi_design_s>();
        h->host = host::prepare_lsi_design(a, m, n, g, k, ridge);
        const auto& d = h->host;
        std::vector<double> qt(size_t(m * n)), et(size_t(n * k));
        for (int64_t i = 0; i < n; ++i)
            for (int64_t j = 0; j < m; ++j) qt[size_t(j * n + i)] = d.q_t[size_t(i * m + j)];
        for (int64_t j = 0; j < k; ++j)
            for (int64_t i = 0; i < n; ++i) et[size_t(i * k + j)] = d.e[size_t(j * n + i)];
        h->qt.upload(qt.data(), qt.size());
        h->back.upload(d.back.data(), d.back.size());
        std::vector<double> back_t(size_t(n * n));
        for (int64_t i = 0; i < n; ++i)
            for (int64_t j = 0; j < n; ++j) back_t[size_t(j * n + i)] = d.back[size_t(i * n + j)];
        h->back_t.upload(back_t.data(), back_t.size());
        h->et.upload(et.data(), et.size());
        h->e.upload(d.e.data(), d.e.size());
        h->gram.upload(d.gram.data(), d.gram.size());
        h->abs_sums.upload(d.abs_sums.data(), d.abs_sums.size());
        auto upload32 = [](DeviceArray<float>& dst, const std::vector<double>& src) {
            const std::vector<float> f(src.begin(), src.end());
            dst.upload(f.data(), f.size());
        };
        upload32(h->qt32, qt);
        upload32(h->back32, d.back);
        upload32(h->et32, et);
        upload32(h->e32, d.e);
        upload32(h->gram32, d.gram);
        upload32(h->abs_sums32, d.abs_sums);
        *out = h.release();
    });
}

void lar_lsi_design_destroy(lar_lsi_design design) { delete design; }

int lar_lsi_design_matrices(lar_lsi_design design, double* q_t, double* back, double* e, double* gram,
                            double* abs_sums) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        const auto& d = design->host;
        if (q_t) std::copy(d.q_t.begin(), d.q_t.end(), q_t);
        if (back) std::copy(d.back.begin(), d.back.end(), back);
        if (e) std::copy(d.e.begin(), d.e.end(), e);
        if (gram) std::copy(d.gram.begin(), d.gram.end(), gram);
        if (abs_sums) std::copy(d.abs_sums.begin(), d.abs_sums.end(), abs_sums);
    });
}

int lar_fit_lsi(lar_lsi_design design, const double* signals, int64_t v, int only_qr, double* x,
                uint8_t* converged, uint8_t* status, int32_t* outer, uint8_t* active, void* stream) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(signals && x && converged, "signals, x and converged must not be NULL");
        const auto& h = design->host;
        const int cap = int(std::min<int64_t>(kFactorCap, (h.n + 1 + 7) / 8 * 8));
        const LsiWarpLayout lay{int(h.k), cap};
        const size_t smem = lay.bytes() * kLsiWarps;
        require(smem <= 200 * 1024, "the LSI problem has too many constraints for the shared-memory solver");
        // The group kernels take the fit where E^T and eight voxels fit in shared memory and the list
        // holds voxel numbers (msmt at lmax 8: 47 unknowns, 302 constraints, 226 KB); lsi_kernel takes the
        // other sizes, and the voxels whose factor fails in both group kernels.
        const GroupPlan plan = only_qr || v >= (int64_t(1) << 31) ? GroupPlan{} : group_plan(int(h.n), int(h.k));
        const bool grouped = plan.main != nullptr;
        // Constraint columns per lane: 10 up to 320 constraints (302 with the 300-direction grid),
        // else kColsPerLane.
        auto kernel = h.k <= 320 ? lsi_kernel<10> : lsi_kernel<kColsPerLane>;
        allow_smem(kernel, smem);
        int per_sm = 1;  // the marked voxels are few: one CTA per SM looks for them
        if (!grouped)
            cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kLsiWarps * 32, smem),
                       "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((v + kLsiWarps - 1) / kLsiWarps,
                                                                      int64_t(sm_count()) * ctas_per_sm(per_sm, "lsi.ctas_per_sm")));
        const int slots = int(blocks) * kLsiWarps;
        const size_t slot = lsi_slot_doubles(int(h.n), int(h.k));
        const size_t lists = 256 + (grouped ? size_t(kRedoCap) * sizeof(int) : 0);
        const size_t need = lists + size_t(slots) * slot * sizeof(double);
        if (need > design->scratch_bytes) {
            if (design->scratch) cuda_check(cudaFree(design->scratch), "cudaFree");
            design->scratch = nullptr;
            design->scratch_bytes = 0;
            cuda_check(cudaMalloc(&design->scratch, need), "cudaMalloc (LSI scratch)");
            design->scratch_bytes = need;
        }
        auto st = static_cast<cudaStream_t>(stream);
        char* base = static_cast<char*>(design->scratch);
        // [0] lsi_kernel's queue, [1] and [2] the group kernels', [3] the listed voxels, [4] the QR variant's marks.
        int* counters = reinterpret_cast<int*>(base);
        cuda_check(cudaMemsetAsync(base, 0, 5 * sizeof(int), st), "cudaMemsetAsync");
        LsiDevice D{int(h.m), int(h.n), int(h.k), design->qt.ptr, design->back.ptr, design->et.ptr,
                    design->e.ptr, design->gram.ptr, design->abs_sums.ptr};
        if (grouped) {
            int* redo = reinterpret_cast<int*>(base + 256);
            launch_rows_product(signals, v, D.m, D.qt, D.n, x, st);
            allow_smem(plan.main, plan.main_smem);
            allow_smem(plan.qr, plan.qr_smem);
            // One CTA per SM (its shared memory); a small call spreads its voxels over the SMs.
            const unsigned grid = unsigned(std::min<int64_t>(v, sm_count()));
            {
                LaunchScope scope("lsi_group_kernel", st);
                plan.main<<<grid, kGroupNW * kGroups * 32, plan.main_smem, st>>>(
                    D, v, counters + 1, redo, counters + 3, x, converged, status, outer, active);
                cuda_check(cudaGetLastError(), "lsi_group_kernel launch");
            }
            {
                LaunchScope scope("lsi_group_qr_kernel", st);
                plan.qr<<<unsigned(std::min<int64_t>(v, sm_count())), kQrNW * 32, plan.qr_smem, st>>>(
                    D, v, counters + 2, redo, counters + 3, x, converged, status, outer, active);
                cuda_check(cudaGetLastError(), "lsi_group_qr_kernel launch");
            }
            launch_rows_product(x, v, D.n, design->back_t.ptr, D.n, x, st);
        }
        LaunchScope scope("lsi_kernel", st);
        kernel<<<unsigned(blocks), kLsiWarps * 32, smem, st>>>(
            D, signals, v, grouped ? 1 : only_qr, grouped ? 1 : 0, counters, cap,
            reinterpret_cast<double*>(base + lists), slot, x, converged, status, outer, active);
        cuda_check(cudaGetLastError(), "lsi_kernel launch");
    });
}

int lar_fit_lsi_plain_fp32(lar_lsi_design design, const float* signals, int64_t v, float* x, uint8_t* status,
                           void* stream) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(signals && x, "signals and x must not be NULL");
        const auto& h = design->host;
        const PlainLsi D{int(h.m), int(h.n), int(h.k), design->qt32.ptr, design->back32.ptr, design->et32.ptr,
                         design->e32.ptr, design->gram32.ptr, design->abs_sums32.ptr};
        launch_plain_lsi(D, signals, v, x, status, static_cast<cudaStream_t>(stream));
    });
}

}  // extern "C"
