// Log-signal least-squares fits of DTI and DKI on the GPU: ordinary, iteratively reweighted
// (IRLS) and, for DKI, re-fitted under constraints. Follows the per-voxel algorithm of
// cpp/src/dwi/log_fit.cpp (reweighted_fit :114-147, fit_log_signal_block :245-269) and the
// maps of src/larmor/dwi/dti.py:170-235.
//
// Layout: the masked signals are (v, n) row-major, one voxel's n samples contiguous, as the
// reference's chunk arrays are. The per-table design (unit-norm columns X (n, p), its
// pseudo-inverse, constraints) is small and shared by every voxel: each CTA stages X and the pseudo-inverse
// once into shared memory.
//
// DTI (p = 7): two to eight neighbouring lanes per voxel (small_lanes). A lane accumulates the 28
// normal-matrix entries and 7 right-hand sides in registers over its share of the measurements (or some of the
// entries over a share it has in common with others), a butterfly sums the lanes' shares, each lane solves the 7 x 7 system by
// L D L^T in registers, and the first finishes with the tensor's eigen-decomposition (cyclic Jacobi) and the DTI
// maps.

#include <cmath>
#include <cstdio>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "host_la.hpp"
#include "log_fit.cuh"
#include "batch.cuh"
#include "log_fit_warp.cuh"
#include "tensor_maps.cuh"

// Device scratch of a design handle: the violator list and the constrained re-fit's warp
// slots, grown on demand. Calls on one handle must not overlap on the GPU.
struct LogScratch {
    void* base = nullptr;
    size_t bytes = 0;
    ~LogScratch() {
        if (base) cudaFree(base);
    }
    void* reserve(size_t need) {
        if (need > bytes) {
            if (base) lar::cuda_check(cudaFree(base), "cudaFree");
            base = nullptr;
            bytes = 0;
            lar::cuda_check(cudaMalloc(&base, need), "cudaMalloc (log-fit scratch)");
            bytes = need;
        }
        return base;
    }
};

struct lar_log_design_s {
    lar::host::LogDesignHost host;
    LogScratch scratch;
    lar::LogDesignDevice<double> d64;
    lar::LogDesignDevice<float> d32;
    lar::DeviceArray<double> x64, pinvt64, g64, scales64;
    lar::DeviceArray<float> x32, pinvt32, g32, scales32;
};

namespace lar {

namespace {

// ---- per-thread helpers ----------------------------------------------------------------

template <class T, int P>
__device__ __forceinline__ bool all_finite(const T (&v)[P]) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < P; ++i) ok &= isfinite(v[i]);
    return ok;
}

// ---- the IRLS of the 7-column design ------------------------------------------------------

constexpr int kSmallThreads = 128;  // most of a CTA
constexpr int kSmallCtas = 3;  // an SM's, by registers (a third more, spilling: no faster)

// How a voxel's lanes share its sums over the measurements. Each sum is the sum of C partial sums, of the
// measurements j = c mod C in increasing j, added in a butterfly of the distances C / 2, ..., 1; C depends on the
// table alone, so a voxel's fit has the same bits in a slice, in a shard and in the whole volume. kCxR are C R lanes, R
// of them sharing a class (normal_equations_shared).
// Measured, microseconds, at 2,003 / 5,000 / 8,000 / 12,000 / 16,000 / 24,000 / 79,912 voxels:
//   n = 13: k2x1 65, 66, 66, 77, 75, 93, 215; k2x2 75, 81, 85, 95, 132, 152; k2x4 55, 65, 92, 104, 130, 174
//   n = 31: k2x1 74, 73, 73, 96, 97, 100, 261; k2x2 63, 65, 69, 90, 118, 140, 382; k2x4 43, 51, 76, 95, 116, 162, 476;
//           k8x1 39, 47, 70, 87, 103, 142, 405
//   n = 94: k2x1 172, 172, 182, 194, 217, 237, 636; k2x2 116, 123, 139, 167, 246, 293, 778; k2x4 74, 100, 154, 186, 240,
//           324, 961; k8x1 67, 82, 124, 150, 191, 254, 746
//   n = 120: k2x1 182 to 924; k8x1 66, 93, 138, 167, 210, 287, 844
// (one lane: 107 at 2,003 and 321 at 79,912 voxels of 31; four classes in four lanes: 50 and 296.)
// The ordinary fit, an unweighted call's and the one a weighted fit starts from and falls back to, has eight classes
// everywhere, one, two or four to a lane, so that the two have the same bits. An unweighted call is its seven sums and
// the maps, on eight lanes in small calls and on four or two in larger ones (k8x1, kPlain4, kPlain2): 2,003 voxels of 31
// measurements 13, 13, 18, 79,912 of them 100, 45, 37; of 134 20, 26, 41 and 172, 127, 180. Past 500 measurements a
// batch's CTA would not hold the signals of two lanes' voxels.
enum class Lanes { kPlain2, kPlain4, k2x1, k2x2, k2x4, k8x1 };
__host__ __device__ constexpr bool plain(Lanes lanes) { return lanes == Lanes::kPlain2 || lanes == Lanes::kPlain4; }
__host__ __device__ constexpr int class_count(Lanes lanes) { return lanes == Lanes::k8x1 ? 8 : 2; }
constexpr int kOrdinaryClasses = 8;
__host__ __device__ constexpr int lane_count(Lanes lanes) {
    return lanes == Lanes::kPlain2 || lanes == Lanes::k2x1 ? 2 : lanes == Lanes::kPlain4 || lanes == Lanes::k2x2 ? 4 : 8;
}
__host__ __device__ inline Lanes small_lanes(int64_t v, int n, bool weighted) {
    if (!weighted) return n > 500 || v <= 6000 ? Lanes::k8x1 : v <= 20000 || n >= 80 ? Lanes::kPlain4 : Lanes::kPlain2;
    if (n >= 96) return Lanes::k8x1;
    return v <= 6000 ? Lanes::k2x4 : v <= 14000 && n >= 28 ? Lanes::k2x2 : Lanes::k2x1;
}

// f with the lanes as a compile-time constant.
template <class F>
__host__ __device__ inline void with_lanes(Lanes lanes, const F& f) {
    switch (lanes) {
        case Lanes::kPlain2: f(std::integral_constant<Lanes, Lanes::kPlain2>{}); break;
        case Lanes::kPlain4: f(std::integral_constant<Lanes, Lanes::kPlain4>{}); break;
        case Lanes::k2x1: f(std::integral_constant<Lanes, Lanes::k2x1>{}); break;
        case Lanes::k2x2: f(std::integral_constant<Lanes, Lanes::k2x2>{}); break;
        case Lanes::k2x4: f(std::integral_constant<Lanes, Lanes::k2x4>{}); break;
        default: f(std::integral_constant<Lanes, Lanes::k8x1>{});
    }
}

__host__ __device__ constexpr int small_ctas(Lanes lanes) { return plain(lanes) ? 2 * kSmallCtas : kSmallCtas; }

// Row strides in shared memory: of x and pinv^T (7 entries in whole 16-byte loads, eight rows of which
// fall in distinct banks), and of the log signals of `voxels` voxels.
template <class T>
__host__ __device__ constexpr int row_ld() { return sizeof(T) == 8 ? 10 : 12; }
__host__ __device__ constexpr int voxel_ld(int voxels) { return voxels + 1; }

template <class T>
size_t small_bytes(int n, int voxels) {
    return size_t(n) * (2 * row_ld<T>() + voxel_ld(voxels)) * sizeof(T);
}

// The first 8 entries of a row.
__device__ __forceinline__ void load_row(const double* row, double (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 two = reinterpret_cast<const double2*>(row)[i];
        x[2 * i] = two.x;
        x[2 * i + 1] = two.y;
    }
}
__device__ __forceinline__ void load_row(const float* row, float (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float4 four = reinterpret_cast<const float4*>(row)[i];
        x[4 * i] = four.x;
        x[4 * i + 1] = four.y;
        x[4 * i + 2] = four.z;
        x[4 * i + 3] = four.w;
    }
}

// Packed index of (a, b), a <= b, in the upper triangle stored row by row.
__host__ __device__ constexpr int packed(int a, int b, int p) { return a * p - a * (a - 1) / 2 + (b - a); }

__host__ __device__ constexpr int packed_row(int k, int p) {
    int a = 0;
    while (k >= packed(a + 1, a + 1, p)) ++a;
    return a;
}
__host__ __device__ constexpr int packed_column(int k, int p) {
    return k - packed(packed_row(k, p), packed_row(k, p), p) + packed_row(k, p);
}

// Solves the symmetric system g x = b (g packed, P x P) in place in b by L D L^T. Returns false
// when a pivot is exactly zero, the weighted normal equations being singular (weights that
// underflow to zero on most measurements), as the reference's zero LU pivot test does
// (cpp/src/dwi/log_fit.cpp:128-133).
// Every index is fixed at compile time by loops from 0 with a test: loops from j + 1 were not unrolled, and
// the matrix lay in local memory, written and read in each iteration (half a gigabyte at 79,912 voxels).
template <class T, int P>
__device__ __forceinline__ bool ldlt_solve(T (&g)[P * (P + 1) / 2], T (&b)[P]) {
    // In place: g(j, j) <- 1 / d_j, g(j, i) (j < i) <- L(i, j); behind column j its update is taken from the rest.
    bool ok = true;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const T d = g[packed(j, j, P)];
        ok &= (d != T(0));
        const T inv = T(1) / d;
        T l[P];
#pragma unroll
        for (int i = 0; i < P; ++i)
            if (i > j) {
                l[i] = g[packed(j, i, P)] * inv;
                b[i] = fma(-l[i], b[j], b[i]);
            }
#pragma unroll
        for (int i = 0; i < P; ++i)
#pragma unroll
            for (int k = 0; k < P; ++k)
                if (i > j && k >= i) g[packed(i, k, P)] = fma(-l[i], g[packed(j, k, P)], g[packed(i, k, P)]);
#pragma unroll
        for (int i = 0; i < P; ++i)
            if (i > j) g[packed(j, i, P)] = l[i];
        b[j] *= inv;
    }
    if (!ok) return false;
#pragma unroll
    for (int i = P - 1; i >= 0; --i)
#pragma unroll
        for (int k = 0; k < P; ++k)
            if (k > i) b[i] = fma(-g[packed(i, k, P)], b[k], b[i]);
    return true;
}

// The sum of C classes, or of the C sums that lanes hold of theirs, lane g of the voxel holding that of g % C in v, the
// same bits in each lane (mask: the voxel's lanes).
template <int C, class T, int N>
__device__ __forceinline__ void class_sum(T (&v)[N], unsigned mask) {
#pragma unroll
    for (int o = C / 2; o > 0; o /= 2)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(mask, v[i], o);
}

// The maximum over a voxel's G lanes, in each.
template <int G, class T>
__device__ __forceinline__ T lanes_max(T v, unsigned mask) {
#pragma unroll
    for (int o = 1; o < G; o *= 2) v = fmax(v, __shfl_xor_sync(mask, v, o));
    return v;
}

template <class T>
__device__ __forceinline__ T predict(const T (&x)[8], const T (&q)[7]) {
    T pred = T(0);
#pragma unroll
    for (int a = 0; a < 7; ++a) pred = fma(x[a], q[a], pred);
    return pred;
}

// The weighted normal matrix m and right-hand side r of one voxel, weights exp(2 (x p - mx)), the same bits in each
// of its lanes (g: this one). Each lane sums all 35 entries of its class.
template <class T, int C>
__device__ __forceinline__ void normal_equations(const T* __restrict__ xs, int n, const T* __restrict__ ys, int stride,
                                                 const T (&p)[7], T mx, int g, unsigned mask, T (&m)[28], T (&r)[7]) {
    constexpr int P = 7, PP = 28, LD = row_ld<T>();
#pragma unroll
    for (int k = 0; k < PP; ++k) m[k] = T(0);
#pragma unroll
    for (int a = 0; a < P; ++a) r[a] = T(0);
    for (int j = g; j < n; j += C) {
        T x[8];
        load_row(xs + j * LD, x);
        const T w = dev_exp<T>(T(2) * (predict(x, p) - mx));
        const T y = ys[j * stride];
        // The products x_a x_b come from the row itself: a table of them was four times the loads.
        T wx[P];
#pragma unroll
        for (int a = 0; a < P; ++a) {
            wx[a] = w * x[a];
            r[a] = fma(wx[a], y, r[a]);
        }
#pragma unroll
        for (int k = 0; k < PP; ++k) m[k] = fma(wx[packed_row(k, P)], x[packed_column(k, P)], m[k]);
    }
    class_sum<C>(m, mask);
    class_sum<C>(r, mask);
}

// Row k of part `part` of R of the rows of [x, y], and the first column it is summed from (an entry or more below the
// diagonal too for some parts, which no one reads): two parts 0, 3, 4, 7 and 1, 2, 5, 6 from the columns 0, 2, 4, 6;
// four parts 0, 7 and 1, 6 and 2, 5 and 3, 4 from the columns 0, 4.
__host__ __device__ constexpr int part_row(int R, int part, int k) {
    if (R == 4) return k == 0 ? part : 7 - part;
    return 2 * k + (k & 1 ? 1 - part : part);
}
__host__ __device__ constexpr int part_column(int R, int k) { return R * k; }

// The same from C R lanes: of the class that R lanes share, each takes every R-th exponential, four of them before
// the sums (one at a time for a remainder), and the sums of 8 / R rows of [x, y]^T W [x, y].
template <class T, int C, int R>
__device__ __forceinline__ void normal_equations_shared(const T* __restrict__ xs, int n, const T* __restrict__ ys,
                                                        int stride, const T (&p)[7], T mx, int g, unsigned mask,
                                                        T (&m)[28], T (&r)[7]) {
    constexpr int P = 7, LD = row_ld<T>(), kRows = 8 / R;
    const int c = g % C, part = g / C, first = int(threadIdx.x % 32) - g + c;  // the class's lane of part 0
    T acc[kRows][8];
#pragma unroll
    for (int k = 0; k < kRows; ++k)
#pragma unroll
        for (int b = 0; b < 8; ++b) acc[k][b] = T(0);
    // The sums of `ahead` measurements per lane of each class, from measurement j0 of all.
    auto block = [&](auto ahead, int j0) {
        constexpr int kAhead = decltype(ahead)::value;
        T mine[kAhead], x[8];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            load_row(xs + min(j0 + c + (R * u + part) * C, n - 1) * LD, x);
            mine[u] = dev_exp<T>(T(2) * (predict(x, p) - mx));
        }
#pragma unroll
        for (int u = 0; u < R * kAhead; ++u) {
            const T from = __shfl_sync(mask, mine[u / R], first + C * (u % R));
            const int j = j0 + c + C * u, at = min(j, n - 1);
            const T w = j < n ? from : T(0);  // adds zeros past the last
            load_row(xs + at * LD, x);
            x[7] = ys[at * stride];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                // The part's row: of four parts from shared memory again (selecting it took a third of the loop).
                T row;
                if (R == 4)
                    row = k == 0 ? xs[at * LD + part] : part == 0 ? x[7] : xs[at * LD + 7 - part];
                else
                    row = part == 0 ? x[part_row(R, 0, k)] : x[part_row(R, 1, k)];
                const T wx = w * row;
#pragma unroll
                for (int b = 0; b < 8; ++b)
                    if (b >= part_column(R, k)) acc[k][b] = fma(wx, x[b], acc[k][b]);
            }
        }
    };
    for (int j0 = 0; j0 < n;) {
        if (n - j0 > 3 * R * C) {
            block(std::integral_constant<int, 4>{}, j0);
            j0 += 4 * R * C;
        } else {
            block(std::integral_constant<int, 1>{}, j0);
            j0 += R * C;
        }
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) class_sum<C>(acc[k], mask);
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int a = part_row(R, q, k);
            if (a >= P) continue;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                if (b < a) continue;
                const T entry = __shfl_sync(mask, acc[k][b], first + C * q);
                if (b < P)
                    m[packed(a, b, P)] = entry;
                else
                    r[a] = entry;
            }
        }
}

// Fits one voxel from its log signals ys[j * stride] on its lanes, and leaves its scaled parameters in p
// (the same in every lane); returns the number of weighted fits. Follows reweighted_fit
// (cpp/src/dwi/log_fit.cpp:114-147) from the ordinary fit pinv y (:251).
// What bounds it: the latencies of a measurement's chain (a product, an exponential, the sums) with twelve warps
// in an SM, and the lanes that wait for their warp's slowest voxel.
template <class T, Lanes LANES>
__device__ __forceinline__ int fit_voxel_small(const T* __restrict__ xs, const T* __restrict__ pinvt, int n,
                                               const T* __restrict__ ys, int stride, bool weighted, int max_rw, T tol,
                                               T (&p)[7]) {
    constexpr int P = 7, PP = 28, LD = row_ld<T>(), G = lane_count(LANES), C = class_count(LANES);
    const int g = int(threadIdx.x) % G;
    const unsigned mask = ((1u << G) - 1u) << (threadIdx.x % 32 - g);
    auto ordinary = [&] {
        constexpr int K = kOrdinaryClasses / G;  // classes of a lane
        T sum[K][P];
#pragma unroll
        for (int q = 0; q < K; ++q)
#pragma unroll
            for (int a = 0; a < P; ++a) sum[q][a] = T(0);
#pragma unroll 2
        for (int j0 = g; j0 < n; j0 += kOrdinaryClasses)
#pragma unroll
            for (int q = 0; q < K; ++q) {
                const int j = j0 + q * G;
                if (q > 0 && j >= n) continue;
                const T y = ys[j * stride];
                T row[8];
                load_row(pinvt + j * LD, row);
#pragma unroll
                for (int a = 0; a < P; ++a) sum[q][a] = fma(row[a], y, sum[q][a]);
            }
#pragma unroll
        for (int o = K / 2; o > 0; o /= 2)
#pragma unroll
            for (int q = 0; q < o; ++q)
#pragma unroll
                for (int a = 0; a < P; ++a) sum[q][a] += sum[q + o][a];
#pragma unroll
        for (int a = 0; a < P; ++a) p[a] = sum[0][a];
        class_sum<G>(p, mask);
    };
    ordinary();
    if constexpr (plain(LANES)) return 0;
    if (!weighted || !all_finite(p)) return 0;
    T mx = -INFINITY;
#pragma unroll 2
    for (int j = g; j < n; j += G) {
        T x[8];
        load_row(xs + j * LD, x);
        mx = fmax(mx, predict(x, p));
    }
    mx = lanes_max<G>(mx, mask);
    int it = 0;
    for (; it < max_rw; ++it) {
        T m[PP], r[P];
        if constexpr (G > C)
            normal_equations_shared<T, C, G / C>(xs, n, ys, stride, p, mx, g, mask, m, r);
        else
            normal_equations<T, C>(xs, n, ys, stride, p, mx, g, mask, m, r);
        if (!ldlt_solve<T, P>(m, r) || !all_finite(r)) {
            ordinary();
            return it + 1;
        }
        T change = T(0), mx_next = -INFINITY;
#pragma unroll 2
        for (int j = g; j < n; j += G) {
            T x[8];
            load_row(xs + j * LD, x);
            const T po = predict(x, p), pn = predict(x, r);
            change = fmax(change, fabs(pn - po));
            mx_next = fmax(mx_next, pn);
        }
        change = lanes_max<G>(change, mask);
        mx = lanes_max<G>(mx_next, mask);
#pragma unroll
        for (int a = 0; a < P; ++a) p[a] = r[a];
        if (!(change > tol)) return it + 1;
    }
    return it;
}

// Stages x and pinv^T (n, p) into shared memory; returns the end.
template <class T>
__device__ __forceinline__ T* stage_design(const LogDesignDevice<T>& d, T* sm) {
    constexpr int P = 7, LD = row_ld<T>();
    for (int i = threadIdx.x; i < d.n * 8; i += blockDim.x) {
        const int j = i / 8, a = i % 8;
        sm[j * LD + a] = a < P ? d.x[j * P + a] : T(0);
        sm[(d.n + j) * LD + a] = a < P ? d.pinvt[j * P + a] : T(0);
    }
    return sm + 2 * d.n * LD;
}

// The log signals of `count` voxels from `first`, measurement-major, the loads along the rows.
template <class T, class Src>
__device__ __forceinline__ void stage_signals(const Src& src, int64_t first, int count, int n, T* ys, int ld) {
    for (int i = threadIdx.x; i < count * n; i += blockDim.x) {
        const int local = i / n;
        ys[(i - local * n) * ld + local] = src.template entry<T>(first + local, first * n + i);
    }
}

template <class T, Lanes LANES, class Src>
__global__ void __launch_bounds__(kSmallThreads, small_ctas(LANES)) fit_log_small_kernel(LogDesignDevice<T> d, Src src, int64_t v,
                                                                     int weighted, int max_rw, T tol,
                                                                     double* __restrict__ params,
                                                                     uint8_t* __restrict__ broke,
                                                                     int32_t* __restrict__ iterations) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);
    constexpr int G = lane_count(LANES);
    const int n = d.n, voxels = blockDim.x / G, ld = voxel_ld(voxels), local = threadIdx.x / G;
    T* ys = stage_design<T>(d, sm);
    const int64_t first = int64_t(blockIdx.x) * voxels;
    const int count = int(v - first < int64_t(voxels) ? v - first : int64_t(voxels));
    stage_signals<T>(src, first, count, n, ys, ld);
    __syncthreads();
    if (local >= count) return;
    const int64_t voxel = first + local;
    T p[7];
    const int it = fit_voxel_small<T, LANES>(sm, sm + n * row_ld<T>(), n, ys + local, ld, weighted != 0, max_rw, tol, p);
    if (threadIdx.x % G) return;
#pragma unroll
    for (int a = 0; a < 7; ++a) params[voxel * 7 + a] = double(p[a]) / d.scales64[a];
    broke[voxel] = 0;
    if (iterations) iterations[voxel] = it;
}

template <class T, Lanes LANES>
__global__ void __launch_bounds__(kSmallThreads, small_ctas(LANES)) fit_dti_maps_kernel(LogDesignDevice<T> d, FlooredSource src,
                                                                    int64_t v, int weighted, int max_rw, T tol,
                                                                    float* __restrict__ maps,
                                                                    uint8_t* __restrict__ npd,
                                                                    double* __restrict__ params) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);
    constexpr int G = lane_count(LANES);
    const int n = d.n, voxels = blockDim.x / G, ld = voxel_ld(voxels), local = threadIdx.x / G;
    T* ys = stage_design<T>(d, sm);
    const int64_t first = int64_t(blockIdx.x) * voxels;
    const int count = int(v - first < int64_t(voxels) ? v - first : int64_t(voxels));
    stage_signals<T>(src, first, count, n, ys, ld);
    __syncthreads();
    if (local >= count) return;
    const int64_t voxel = first + local;
    T p[7];
    fit_voxel_small<T, LANES>(sm, sm + n * row_ld<T>(), n, ys + local, ld, weighted != 0, max_rw, tol, p);
    if (threadIdx.x % G) return;
    T dt[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) dt[a] = p[a + 1] / d.scales[a + 1];
    if (params) {
#pragma unroll
        for (int a = 0; a < 7; ++a) params[voxel * 7 + a] = double(p[a]) / d.scales64[a];
    }
    dti_maps<T>(dt, voxel, v, maps, npd);
}

// The DTI family of a batch (batch.cuh): a persistent grid whose CTAs take tickets of
// dti_ticket_voxels(v, n) voxels of one volume from a device counter across every DTI volume; a CTA
// restages the design when its ticket moves to another volume. Per voxel the same fit and maps
// as fit_dti_maps_kernel (FP64).
template <Lanes LANES>
__device__ __noinline__ void batch_dti_ticket(const DtiBatchJob& job, int64_t ticket, int weighted, int max_rw,
                                              double tol, double* sm) {
    constexpr int G = lane_count(LANES);
    const int n = job.d.n, local = threadIdx.x / G;
    constexpr int kVoxels = kDtiBatchThreads / G, kLd = voxel_ld(kVoxels), LD = row_ld<double>();
    double* ys = sm + 2 * n * LD;
    const int64_t first = ticket * kVoxels;
    const int count = int(job.v - first < int64_t(kVoxels) ? job.v - first : int64_t(kVoxels));
    stage_signals<double>(FlooredSource{job.s, job.floor, n}, first, count, n, ys, kLd);
    __syncthreads();
    if (local < count) {
        double p[7];
        fit_voxel_small<double, LANES>(sm, sm + n * LD, n, ys + local, kLd, weighted != 0, max_rw, tol, p);
        if (threadIdx.x % G == 0) {
            double dt[6];
#pragma unroll
            for (int a = 0; a < 6; ++a) dt[a] = p[a + 1] / job.d.scales[a + 1];
            dti_maps<double>(dt, first + local, job.v, job.maps, job.npd);
        }
    }
}

__global__ void __launch_bounds__(kDtiBatchThreads, kSmallCtas * kSmallThreads / kDtiBatchThreads)
    batch_dti_kernel(const DtiBatchJob* __restrict__ jobs, const int64_t* __restrict__ first, int n_jobs, int weighted,
                     int max_rw, double tol, int* __restrict__ queue) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long ticket;
    double* sm = reinterpret_cast<double*>(smem_raw);
    const int64_t total = first[n_jobs];
    int cur = -1;
    for (;;) {
        if (threadIdx.x == 0) ticket = atomicAdd(reinterpret_cast<unsigned long long*>(queue), 1ull);
        __syncthreads();
        const int64_t t = ticket;
        if (t >= total) break;
        const int j = ticket_job(first, n_jobs, t);
        const DtiBatchJob& job = jobs[j];
        if (j != cur) {
            stage_design<double>(job.d, sm);
            cur = j;
        }
        with_lanes(small_lanes(job.v, job.d.n, weighted != 0), [&](auto lanes) {
            batch_dti_ticket<decltype(lanes)::value>(job, t - first[j], weighted, max_rw, tol, sm);
        });
        __syncthreads();
    }
}

template <class T>
const LogDesignDevice<T>& device_view(const lar_log_design_s* h);
template <>
const LogDesignDevice<double>& device_view<double>(const lar_log_design_s* h) { return h->d64; }
template <>
const LogDesignDevice<float>& device_view<float>(const lar_log_design_s* h) { return h->d32; }

// Threads per CTA of the shared-memory fits: few for a small call, so that it spreads over the SMs, else
// kSmallThreads, whose voxels share the staged design (20,000 voxels of 270 measurements: 639 us, with 64 threads
// 735); fewer when the design and the CTA's signals do not fit in shared memory (tables of more than about 700 measurements).
template <class T>
int small_threads(int64_t v, int n, int lanes) {
    const int64_t want = launch_setting("dti.voxels_per_cta");
    int threads = v <= 6000 ? 64 : kSmallThreads;
    if (want == 16 || want == 32 || want == 64) threads = int(std::min<int64_t>(kSmallThreads, want * lanes));
    while (threads > 16 && small_bytes<T>(n, threads / lanes) > 227 * 1024) threads /= 2;
    return threads;
}

template <class Kernel>
void set_smem(Kernel kernel, size_t bytes) {
    require(bytes <= 227 * 1024, "the design has too many measurements for the shared-memory fit");
    allow_smem(kernel, bytes);
}

// Scratch layout for a constrained fit of v voxels: [count, two queues] ints, voxel ids, scaled
// parameters, then the warp slots of the re-fit.
struct ScratchPlan {
    size_t ids_off, params_off, slots_off, total;
    int slots;
};

inline ScratchPlan plan_scratch(const lar::host::LogDesignHost& h, int64_t v) {
    ScratchPlan s{};
    const size_t align = 256;
    auto up = [&](size_t x) { return (x + align - 1) / align * align; };
    s.ids_off = align;
    s.params_off = up(s.ids_off + size_t(v) * sizeof(int64_t));
    s.slots_off = up(s.params_off + size_t(v) * h.p * sizeof(double));
    // As many warp slots as warps of the re-fit fit on the GPU at once.
    const int64_t cap = constrained_resident_warps(int(h.n), int(h.p), h.dki);
    s.slots = int(std::max<int64_t>(4, std::min<int64_t>((v + 3) / 4 * 4, cap)));
    s.total = s.slots_off + size_t(s.slots) * constrained_slot_doubles(int(h.n), int(h.p), int(h.m)) * sizeof(double);
    return s;
}

template <class T, class Src>
void launch_general(lar_log_design_s* h, const Src& src, int64_t v, int weighted, int max_rw, double tol,
                    double* params, uint8_t* broke, int32_t* iterations, cudaStream_t stream) {
    const auto& d = device_view<T>(h);
    require(h->host.p <= 32, "the log fit takes at most 32 parameters");
    ViolatorList<T> vl;
    ViolatorList<double> vl64;
    ScratchPlan plan{};
    char* base = nullptr;
    if (h->host.m > 0) {
        require(h->host.p <= 31, "the constrained log fit takes at most 31 parameters");
        require(v < (int64_t(1) << 31), "at most 2^31 - 1 voxels per constrained call");
        plan = plan_scratch(h->host, v);
        base = static_cast<char*>(h->scratch.reserve(plan.total));
        cuda_check(cudaMemsetAsync(base, 0, 3 * sizeof(int), stream), "cudaMemsetAsync");
        vl.count = reinterpret_cast<int*>(base);
        vl.capacity = int(v);
        vl.voxel = reinterpret_cast<int64_t*>(base + plan.ids_off);
        vl.params = reinterpret_cast<double*>(base + plan.params_off);
        vl64.count = vl.count;
        vl64.capacity = vl.capacity;
        vl64.voxel = vl.voxel;
        vl64.params = vl.params;
    }
    launch_log_warp<T>(d, src, v, weighted, max_rw, tol, params, broke, iterations, vl, stream);
    if (h->host.m > 0) {
        launch_constrained<Src>(h->d64, src, weighted, vl64, int(v), reinterpret_cast<int*>(base) + 1,
                                reinterpret_cast<double*>(base + plan.slots_off), plan.slots, params, stream);
    }
}

template <class T>
void launch_fit(lar_log_design_s* h, const double* log_s, int64_t v, int weighted,
                int max_rw, double tol, double* params, uint8_t* broke, int32_t* iterations,
                cudaStream_t stream) {
    const auto& d = device_view<T>(h);
    const int p = int(h->host.p);
    LogSource src{log_s, h->host.n};
    if (p == 7 && h->host.m == 0) {
        auto run = [&](auto kernel, int lanes) {
            const int threads = small_threads<T>(v, d.n, lanes), voxels = threads / lanes;
            const size_t sm = small_bytes<T>(d.n, voxels);
            set_smem(kernel, sm);
            const int64_t grid = (v + voxels - 1) / voxels;
            LaunchScope scope("fit_log_small_kernel", stream);
            kernel<<<unsigned(grid), threads, sm, stream>>>(d, src, v, weighted, max_rw, T(tol), params, broke,
                                                            iterations);
            cuda_check(cudaGetLastError(), "fit_log_small_kernel launch");
        };
        with_lanes(small_lanes(v, d.n, weighted != 0), [&](auto lanes) {
            constexpr Lanes kLanes = decltype(lanes)::value;
            run(fit_log_small_kernel<T, kLanes, LogSource>, lane_count(kLanes));
        });
        return;
    }
    launch_general<T>(h, src, v, weighted, max_rw, tol, params, broke, iterations, stream);
}

template <class T>
void launch_dti_maps(const lar_log_design_s* h, const float* s, const double* floor, int64_t v,
                     int weighted, int max_rw, double tol, float* maps, uint8_t* npd,
                     double* params, cudaStream_t stream) {
    const auto& d = device_view<T>(h);
    FlooredSource src{s, floor, h->host.n};
    auto run = [&](auto kernel, int lanes) {
        const int threads = small_threads<T>(v, d.n, lanes), voxels = threads / lanes;
        const size_t sm = small_bytes<T>(d.n, voxels);
        set_smem(kernel, sm);
        const int64_t grid = (v + voxels - 1) / voxels;
        LaunchScope scope("fit_dti_maps_kernel", stream);
        kernel<<<unsigned(grid), threads, sm, stream>>>(d, src, v, weighted, max_rw, T(tol), maps, npd, params);
        cuda_check(cudaGetLastError(), "fit_dti_maps_kernel launch");
    };
    with_lanes(small_lanes(v, d.n, weighted != 0), [&](auto lanes) {
        constexpr Lanes kLanes = decltype(lanes)::value;
        run(fit_dti_maps_kernel<T, kLanes>, lane_count(kLanes));
    });
}

}  // namespace

int dti_ticket_voxels(int64_t v, int n, bool weighted) {
    return kDtiBatchThreads / lane_count(small_lanes(v, n, weighted));
}

size_t batch_dti_smem(int64_t v, int n, bool weighted) {
    return small_bytes<double>(n, dti_ticket_voxels(v, n, weighted));
}

void launch_batch_dti(const DtiBatchJob* jobs, const int64_t* first, int n_jobs, size_t sm, int64_t tickets,
                      int weighted, int max_rw, double tol, int* queue, cudaStream_t stream) {
    if (n_jobs == 0 || tickets == 0) return;
    auto kernel = batch_dti_kernel;
    set_smem(kernel, sm);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kDtiBatchThreads, sm),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const int64_t grid = std::min<int64_t>(tickets, int64_t(sm_count()) * std::max(per_sm, 1));
    cuda_check(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), stream), "cudaMemsetAsync");
    LaunchScope scope("batch_dti_kernel", stream);
    kernel<<<unsigned(grid), kDtiBatchThreads, sm, stream>>>(jobs, first, n_jobs, weighted, max_rw, tol, queue);
    cuda_check(cudaGetLastError(), "batch_dti_kernel launch");
}

namespace {

template <class T>
void upload_design(lar_log_design_s* h, DeviceArray<T>& x, DeviceArray<T>& pinvt, DeviceArray<T>& g,
                   DeviceArray<T>& scales, LogDesignDevice<T>& view) {
    const auto& hd = h->host;
    const int64_t n = hd.n, p = hd.p, m = hd.m;
    std::vector<T> xv(static_cast<size_t>(n * p)), pt(static_cast<size_t>(n * p)), gv(static_cast<size_t>(2 * m * p)), sv(static_cast<size_t>(p));
    for (int64_t i = 0; i < n; ++i)
        for (int64_t a = 0; a < p; ++a) {
            xv[size_t(i * p + a)] = T(hd.x[size_t(i * p + a)]);
            pt[size_t(i * p + a)] = T(hd.pinv[size_t(a * n + i)]);
        }
    // g (m, p) row-major, then its transpose (p, m).
    for (int64_t c = 0; c < m; ++c)
        for (int64_t a = 0; a < p; ++a) {
            gv[size_t(c * p + a)] = T(hd.g[size_t(c * p + a)]);
            gv[size_t(m * p + a * m + c)] = T(hd.g[size_t(c * p + a)]);
        }
    for (int64_t a = 0; a < p; ++a) sv[size_t(a)] = T(hd.scales[size_t(a)]);
    x.upload(xv.data(), xv.size());
    pinvt.upload(pt.data(), pt.size());
    g.upload(gv.data(), gv.size());
    scales.upload(sv.data(), sv.size());
    view.n = int(n);
    view.p = int(p);
    view.m = int(m);
    view.x = x.ptr;
    view.pinvt = pinvt.ptr;
    view.g = g.ptr;
    view.gt = m > 0 ? g.ptr + m * p : nullptr;
    view.scales = scales.ptr;
}

}  // namespace

void launch_dki_maps(const double* params, int64_t v, float* maps, uint8_t* npd, cudaStream_t stream);

}  // namespace lar

using namespace lar;

namespace lar {
LogDesignDevice<double> log_design_view(const lar_log_design_s* h) { return h->d64; }
}  // namespace lar

extern "C" {

int lar_log_design_create(const double* x, int64_t n, int64_t p, const double* g, int64_t m,
                          lar_log_design* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(x != nullptr && n > 0 && p > 0, "x must be a non-empty (n, p) array");
        require(m >= 0 && (m == 0 || g != nullptr), "g must be (m, p) with m >= 0");
        require(n >= p, "x must be (n, p) with n >= p: got (" + std::to_string(n) + ", " + std::to_string(p) + ")");
        auto h = std::make_unique<lar_log_design_s>();
        h->host = host::prepare_log_design(x, n, p, g, m);
        double bound = 0.0;
        h->host.dki = dki_constraint_bound(h->host.g.data(), m, p, &bound);
        upload_design<double>(h.get(), h->x64, h->pinvt64, h->g64, h->scales64, h->d64);
        upload_design<float>(h.get(), h->x32, h->pinvt32, h->g32, h->scales32, h->d32);
        h->d64.dki = h->host.dki;
        h->d64.bound = bound;
        h->d64.scales64 = h->scales64.ptr;
        h->d32.scales64 = h->scales64.ptr;
        *out = h.release();
    });
}

void lar_log_design_destroy(lar_log_design design) { delete design; }

int lar_log_design_violators(lar_log_design design, int64_t* count) {
    return guarded([&] {
        require(design != nullptr && count != nullptr, "design and count must not be NULL");
        int n = 0;
        if (design->host.m > 0 && design->scratch.base != nullptr)
            cuda_check(cudaMemcpy(&n, design->scratch.base, sizeof(int), cudaMemcpyDeviceToHost),
                       "cudaMemcpy (violator count)");
        *count = n;
    });
}

int lar_fit_log_signal(lar_log_design design, const double* log_s, int64_t v, int weighted,
                       int64_t max_iter, double tol, int precision, double* params,
                       uint8_t* broke, int32_t* iterations, void* stream) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        require(v >= 0, "v must be at least 0");
        require(max_iter >= 0, "max_iter must be at least 0");
        require(precision == LAR_FP64 || precision == LAR_FP32, "precision must be LAR_FP64 or LAR_FP32");
        if (v == 0) return;
        require(log_s && params && broke, "log_s, params and broke must not be NULL");
        const int rw = int(std::min<int64_t>(max_iter, 1 << 20));
        auto s = static_cast<cudaStream_t>(stream);
        if (precision == LAR_FP64)
            launch_fit<double>(design, log_s, v, weighted, rw, tol, params, broke, iterations, s);
        else
            launch_fit<float>(design, log_s, v, weighted, rw, tol, params, broke, iterations, s);
    });
}

int lar_fit_dti_maps(lar_log_design design, const float* signals, const double* floor,
                     int64_t v, int weighted, int64_t max_iter, double tol, int precision,
                     float* maps, uint8_t* npd, double* params, void* stream) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        require(design->host.p == 7 && design->host.m == 0,
                "the DTI maps need the 7-column DTI design without constraints");
        require(v >= 0, "v must be at least 0");
        require(max_iter >= 0, "max_iter must be at least 0");
        require(precision == LAR_FP64 || precision == LAR_FP32, "precision must be LAR_FP64 or LAR_FP32");
        if (v == 0) return;
        require(signals && floor && maps && npd, "signals, floor, maps and npd must not be NULL");
        const int rw = int(std::min<int64_t>(max_iter, 1 << 20));
        auto s = static_cast<cudaStream_t>(stream);
        if (precision == LAR_FP64)
            launch_dti_maps<double>(design, signals, floor, v, weighted, rw, tol, maps, npd, params, s);
        else
            launch_dti_maps<float>(design, signals, floor, v, weighted, rw, tol, maps, npd, params, s);
    });
}

int lar_dki_maps(const double* params, int64_t v, float* maps, uint8_t* npd, void* stream) {
    return guarded([&] {
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(params && maps && npd, "params, maps and npd must not be NULL");
        launch_dki_maps(params, v, maps, npd, static_cast<cudaStream_t>(stream));
    });
}

int lar_fit_dki_maps(lar_log_design design, const float* signals, const double* s0, const double* floor,
                     const uint8_t* is_b0, int64_t v, int weighted, int64_t max_iter, double tol,
                     int precision, float* maps, uint8_t* npd, uint8_t* broke, double* params,
                     void* stream) {
    return guarded([&] {
        require(design != nullptr, "design must not be NULL");
        require(design->host.p == 22, "the DKI maps need the 22-column DKI design");
        require(v >= 0, "v must be at least 0");
        require(max_iter >= 0, "max_iter must be at least 0");
        require(precision == LAR_FP64 || precision == LAR_FP32, "precision must be LAR_FP64 or LAR_FP32");
        if (v == 0) return;
        require(signals && floor && is_b0 && maps && npd && broke && params,
                "signals, floor, is_b0, maps, npd, broke and params must not be NULL");
        const int rw = int(std::min<int64_t>(max_iter, 1 << 20));
        auto st = static_cast<cudaStream_t>(stream);
        CappedSource src{signals, s0, floor, is_b0, design->host.n};
        if (precision == LAR_FP64)
            launch_general<double>(design, src, v, weighted, rw, tol, params, broke, nullptr, st);
        else
            launch_general<float>(design, src, v, weighted, rw, tol, params, broke, nullptr, st);
        launch_dki_maps(params, v, maps, npd, st);
    });
}

}  // extern "C"
