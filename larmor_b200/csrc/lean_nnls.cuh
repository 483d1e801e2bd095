// The ridge NNLS of one voxel on a warp, for active sets of at most 32 columns: the Lawson-Hanson
// steps, rules and tolerances of ridge_nnls in multi_tissue.cu (cpp/src/sd/nnls.cpp:362-418) with the
// fewest instructions and the shortest chain per step. Lane r owns the r-th active column (its
// number, value x, candidate z and row r of M); the kernel's columns are dealt to the lanes CPL each.
//
// What bounds it: instructions and their latency (a fit is ~14 steps on 8 active of 44 columns at low
// resolution, 22 on 12 of 300 at high). With the factor and its inverse both kept, in global slots, and two voxels
// per warp, a low-resolution fit took 18 k warp instructions; here 7.3 k, and a warp's state is 6.1 KB of shared
// memory: sixteen warps per SM at low resolution (one CTA; with the 44 x 44 Gram matrix it takes 115,840 bytes, and
// two CTAs and the kilobyte that each reserves 256 bytes more than an SM has; up to 43 columns two run), twenty at
// high. 250,000 voxels of 280 measurements, ten rounds: low resolution 70.3 -> 26.6 ms, high 35.6 -> 13.6 ms; 8,191
// voxels (latency): 12.8 -> 2.9 ms and 1.66 -> 0.65 ms. Eight voxels per warp with their gradients as one FP64
// tensor-core product was slower at every size (42 ms, 10.5 ms): the voxels' other loops diverge.
//
// - The factor is M = L^-1 alone (packed rows in shared memory) with y = M c_A and z = M^T y. Appending
//   column e: w = M h, then one loop over the rows gives w^T M, w.w and w.y at once (every lane reads
//   the pairs (w_r, y_r), so nothing is reduced by shuffles); the solve is the update z += y_e m of
//   the new row m, in the same order of sums.
// - Removing position p: with v = M(., p) and t_k^2 = sum_{i <= k} v_i^2 from row p on, row k becomes
//   (t_k M(k+1, .) - (v_{k+1} / t_k) sum_{i <= k} v_i M(i, .)) / t_{k+1}, which are the Givens
//   rotations of rows (k, k + 1) that clear column p, composed: one prefix sum over the lanes, then
//   each lane runs down its own column.
// - The steepest column and the blocking step are found with integer reductions on the bits of
//   the (non-negative) doubles: high word, low word, index.
//
// A voxel whose fit needs the QR fallback (a pivot below the tolerance) or more than 32 active columns
// is not finished here: the caller hands it to the full-factor kernel, which fits it from the start.
#pragma once

#include "common.cuh"

namespace lar {

constexpr int kLeanCap = 32;
constexpr int kLeanTri = kLeanCap * (kLeanCap + 1) / 2;
// A warp's doubles: M, the pairs (w, y), (x, column), (t_k / t_{k+1}, v_{k+1} / (t_k t_{k+1})), v and h.
constexpr int kLeanWarpDoubles = kLeanTri + 3 * 2 * kLeanCap + 2 * kLeanCap;

struct LeanWarp {
    double* M;
    double2 *wy, *xc, *ab;
    double *v, *h;
    __device__ __forceinline__ explicit LeanWarp(double* base) {
        wy = reinterpret_cast<double2*>(base);
        xc = wy + kLeanCap;
        ab = xc + kLeanCap;
        v = reinterpret_cast<double*>(ab + kLeanCap);
        h = v + kLeanCap;
        M = h + kLeanCap;
    }
};

__device__ __forceinline__ int lean_tri(int r) { return r * (r + 1) / 2; }

// The lane whose non-negative key is largest (LARGEST) or smallest, the smallest index on a tie, over
// the lanes with idx >= 0: their key and index in every lane; idx < 0 when there is none.
template <bool LARGEST>
__device__ __forceinline__ void lean_pick(double& key, int& idx) {
    constexpr unsigned kAll = 0xffffffffu;
    const bool in = idx >= 0;
    const unsigned hi = unsigned(__double2hiint(key)), lo = unsigned(__double2loint(key));
    unsigned bh, bl;
    if constexpr (LARGEST) {
        bh = __reduce_max_sync(kAll, in ? hi : 0u);
        bl = __reduce_max_sync(kAll, in && hi == bh ? lo : 0u);
    } else {
        bh = __reduce_min_sync(kAll, in ? hi : 0xffffffffu);
        bl = __reduce_min_sync(kAll, in && hi == bh ? lo : 0xffffffffu);
    }
    idx = int(__reduce_min_sync(kAll, in && hi == bh && lo == bl ? unsigned(idx) : 0x7fffffffu));
    if (idx == 0x7fffffff) idx = -1;
    key = __hiloint2double(int(bh), int(bl));
}

// Fits corr on the Gram matrix (row stride ldg, in shared or global memory) of c <= 32 CPL columns:
// out (c) gets the solution. False, leaving out alone, when the voxel needs the full-factor kernel.
template <int CPL>
__device__ __forceinline__ bool lean_nnls(const double* gram, int ldg, int c, double tol, double min_pivot,
                                          const double* __restrict__ corr, const LeanWarp q, double* __restrict__ out,
                                          int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    double cj[CPL];
    unsigned busy = 0u;  // bit t: column lane + 32 t has joined (or does not exist)
#pragma unroll
    for (int t = 0; t < CPL; ++t) {
        const int j = lane + 32 * t;
        cj[t] = j < c ? corr[j] : 0.0;
        if (j >= c) busy |= 1u << t;
    }
    const int max_inner = 3 * c;
    int na = 0, inner = 0, col = 0;
    double x = 0.0, z = 1.0;
    for (;;) {
        // The gradient corr - G x, and its largest positive entry at a column that has not joined.
        double g[CPL];
#pragma unroll
        for (int t = 0; t < CPL; ++t) g[t] = cj[t];
#pragma unroll (CPL > 4 ? 2 : 4)
        for (int r = 0; r < na; ++r) {
            const double2 p = q.xc[r];
            const double* row = gram + __double2loint(p.y) + lane;
#pragma unroll
            for (int t = 0; t < CPL; ++t)
                if (lane + 32 * t < c) g[t] = fma(-p.x, row[32 * t], g[t]);
        }
        double best = 0.0;
        int e = -1;
#pragma unroll
        for (int t = 0; t < CPL; ++t) {
            // (A NaN counts as positive, so that it reaches the result.)
            if (!((busy >> t) & 1u) && !(g[t] <= 0.0) && (e < 0 || g[t] > best)) {
                best = fabs(g[t]);
                e = lane + 32 * t;
            }
        }
        lean_pick<true>(best, e);
        if (e < 0 || best <= tol) break;
        if (na >= kLeanCap) return false;
        // w = M h.
        const double gee = gram[size_t(e) * ldg + e];
        if (lane < na) q.h[lane] = gram[size_t(e) * ldg + col];
        const double ce = corr[e];
        __syncwarp();
        double w = 0.0;
        {
            const double* row = q.M + lean_tri(lane);
            const int mine = lane < na ? lane : -1;
#pragma unroll 4
            for (int j = 0; j < na; ++j) {
                const double hj = q.h[j];
                if (j <= mine) w = fma(row[j], hj, w);
            }
        }
        if (lane < na) q.wy[lane].x = w;
        __syncwarp();
        double u = 0.0, sq = 0.0, wy = 0.0;
#pragma unroll 4
        for (int r = 0; r < na; ++r) {
            const double2 p = q.wy[r];
            if (lane <= r) u = fma(q.M[lean_tri(r) + lane], p.x, u);
            sq = fma(p.x, p.x, sq);
            wy = fma(p.x, p.y, wy);
        }
        const double pivot = gee - sq;
        if (!(pivot > min_pivot * gee)) return false;
        const double inv = rsqrt(pivot), ye = (ce - wy) * inv;
        const double m = lane == na ? inv : -u * inv;
        if (lane <= na) q.M[lean_tri(na) + lane] = m;
        z = lane < na ? fma(m, ye, z) : lane == na ? m * ye : z;
        if (lane == na) {
            x = 0.0;
            col = e;
            q.wy[na].y = ye;
        }
        if (lane == (e & 31)) busy |= 1u << (e >> 5);
        ++na;
        __syncwarp();
        // While a candidate is not positive: towards the fit until the first active column reaches
        // zero; it and every active column below the tolerance leave.
        while (__any_sync(kAll, lane < na && z <= 0.0)) {
            if (++inner > max_inner) {
                // The last least-squares fit is the answer (cpp/src/sd/nnls.cpp:204-207).
                for (int j = lane; j < c; j += 32) out[j] = 0.0;
                __syncwarp();
                if (lane < na) out[col] = z;
                return true;
            }
            const bool blocks = lane < na && z <= 0.0;
            const double dist = x - z;
            double step = blocks && dist > 0.0 ? x / dist : 0.0;
            int b = blocks ? col : -1;
            lean_pick<false>(step, b);
            bool drop = false;
            if (lane < na) {
                x += step * (z - x);
                drop = col == b || !(fabs(x) >= tol);
            }
            unsigned gone = __ballot_sync(kAll, drop);
            while (gone) {
                const int pos = 31 - __clz(gone);
                gone ^= 1u << pos;
                const int left = __shfl_sync(kAll, col, pos);
                if (lane == (left & 31)) busy &= ~(1u << (left >> 5));
                const double v = lane >= pos && lane < na ? q.M[lean_tri(lane) + pos] : 0.0;
                double s = v * v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double a = __shfl_up_sync(kAll, s, o);
                    if (lane >= o) s += a;
                }
                // Lane r: 1 / t_r and t_r; row r - 1 needs t_{r-1} / t_r and v_r / (t_{r-1} t_r).
                const double rt = rsqrt(s);
                const double rt_up = __shfl_up_sync(kAll, rt, 1), t_up = __shfl_up_sync(kAll, s * rt, 1);
                if (lane > pos && lane < na) q.ab[lane - 1] = make_double2(t_up * rt, v * rt_up * rt);
                if (lane < na) q.v[lane] = v;
                const double x_down = __shfl_down_sync(kAll, x, 1);
                const int col_down = __shfl_down_sync(kAll, col, 1);
                __syncwarp();
                // Column `lane` of M (lane 31, or the first idle one, runs y's): row k + 1 is read before
                // any lane writes row k, and written a step later.
                double mine = lane <= pos ? q.M[lean_tri(pos) + lane] : 0.0, sum = 0.0;
                double ym = q.wy[pos].y, ysum = 0.0;
                for (int k = pos; k < na - 1; ++k) {
                    const double2 ab = q.ab[k];
                    const double vk = q.v[k];
                    const double below = lane <= k + 1 ? q.M[lean_tri(k + 1) + lane] : 0.0, yb = q.wy[k + 1].y;
                    sum = fma(vk, mine, sum);
                    ysum = fma(vk, ym, ysum);
                    __syncwarp();
                    if (lane <= k + 1 && lane != pos) q.M[lean_tri(k) + lane - (lane > pos)] = ab.x * below - ab.y * sum;
                    if (lane == 0) q.wy[k].y = ab.x * yb - ab.y * ysum;
                    mine = below;
                    ym = yb;
                }
                if (lane >= pos) {
                    x = x_down;
                    col = col_down;
                }
                --na;
                __syncwarp();
            }
            // z = M^T y.
            z = 0.0;
#pragma unroll 4
            for (int r = 0; r < na; ++r) {
                const double yr = q.wy[r].y;
                if (lane <= r) z = fma(q.M[lean_tri(r) + lane], yr, z);
            }
        }
        if (lane < na) {
            x = z;
            q.xc[lane] = make_double2(z, __hiloint2double(0, col * ldg));
        }
        __syncwarp();
    }
    for (int j = lane; j < c; j += 32) out[j] = 0.0;
    __syncwarp();
    if (lane < na) out[col] = x;
    return true;
}

}  // namespace lar
