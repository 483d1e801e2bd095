// Single-shell constrained spherical deconvolution (CSD) on the GPU: _core.fit_csd
// (cpp/src/python/sd.cpp:171-209) over cpp/src/sd/csd.cpp. Per voxel: the linear estimate
// f = initial s, the projection M^T s, then up to max_iter solves of
// (M^T M + norm_weight I + C_S^T C_S) f = M^T s, S the rows of C where C f < threshold, until
// S repeats (Tournier et al., NeuroImage 35 (2007) 1459-1472).
//
// Mapping: one warp per voxel, voxels grid-strided over a resident grid.
//
// Up to 48 coefficients (csd_tiles_kernel) the constraint matrix lies in the CTA's shared memory for all its
// warps, and the system is only ever in registers, as the lower 8x8 tiles of the FP64 tensor cores'
// accumulators (mma.sync m8n8k4, lane (r, p) holds entries (r, 2p) and (r, 2p + 1)). An accumulator tile
// is both an A operand and, transposed, a B operand of two k-steps, the even and the odd columns, without a
// shuffle. So the blocked Cholesky stays on the tensor cores: X = A (L^-1)^T below a diagonal tile,
// T -= X X^T behind it; only the 8x8 diagonal tiles are eliminated lane by lane, giving their inverse
// factors, which the two triangular solves use as well. What bounds it: the C_S^T C_S products and the
// latencies of the diagonal tiles: 500,040 voxels, 45 coefficients, 300 constraints, 4.6 solves each of 134
// constrained rows, 44.7 ms, of which the products take 26 at the tensor cores' rate (as csd_kernel does it
// below: 138 ms).
//
// For larger systems and constraint sets (csd_kernel) the system is packed in the warp's shared memory (lower
// triangle, row-major). Each iteration rebuilds it as the Gram matrix plus C_S^T C_S on the tensor cores, rows
// staged eight at a time in shared memory. A left-looking Cholesky factorisation (one row per lane) and two
// column-oriented triangular solves follow. The amplitudes C f read C^T, so that the lanes (one
// direction each) load coalesced.

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "common.cuh"

namespace lar {
namespace {

constexpr int kCsdStage = 8;   // constraint rows staged per pass of the system build (two k-steps of 4)
constexpr int kCsdBatch = 8;   // tiles accumulated at once by build_batched
constexpr int kTileRows = 6;   // most tile rows of csd_tiles_kernel: c <= 48 (lmax <= 8)
constexpr int kTileWarps = 16;  // (44.7 ms at the size below; 12 warps of 168 registers: 46.6, 14: 50)

struct CsdDev {
    const double* initial_t;     // (m, c0)
    const double* forward;       // (m, c)
    const double* constraint;    // (k, c)
    const double* constraint_t;  // (c, k)
    const double* gram;          // packed (c (c + 1) / 2): M^T M + norm_weight I
    int m, c, c0, k, max_iter;
    double threshold;
};

__host__ __device__ inline int packed_count(int c) { return c * (c + 1) / 2; }

// The staged rows' stride: c rounded up to whole 8-column tiles.
__host__ __device__ inline int padded8(int c) { return (c + 7) / 8 * 8; }

// Shared memory of one warp: the packed system, f, the right-hand side, y, the staged rows
// (padded to whole 8-column tiles), then the two lists of constrained directions.
__host__ __device__ inline size_t csd_warp_bytes(int c, int k) {
    const size_t doubles = size_t(packed_count(c)) + 3 * size_t(c) + size_t(kCsdStage) * padded8(c);
    return (doubles * 8 + 2 * size_t(k) * 2 + 15) / 16 * 16;
}

// D += A B for one 8x8x4 FP64 tile on the tensor cores: a lane holds A(lane / 4, lane % 4),
// B(lane % 4, lane / 4) and D(lane / 4, 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Stages the constrained rows cur[q0, q0 + kCsdStage) of C into rows (kCsdStage, cp), zero-padded.
__device__ __forceinline__ int stage_rows(const CsdDev& P, const uint16_t* cur, int n_cur, int q0, double* rows,
                                          int cp, int lane) {
    const int nr = min(kCsdStage, n_cur - q0);
    __syncwarp();
    for (int t = lane; t < kCsdStage * cp; t += 32) {
        const int r = t / cp, j = t - r * cp;
        rows[t] = (r < nr && j < P.c) ? P.constraint[size_t(cur[q0 + r]) * P.c + j] : 0.0;
    }
    __syncwarp();
    return nr;
}

// csd_tiles_kernel's row stride in C, odd so that 32 lanes' rows are in different banks, with the columns past c
// zero, and its last row all zero; then the Gram matrix in tiles.
template <int T>
struct TileShape {
    static constexpr int kTiles = T * (T + 1) / 2, kLd = 8 * T + 1;
    static __host__ __device__ size_t doubles(int k) { return size_t(k + 1) * kLd + (size_t(k + 1) * kLd & 1) + 64 * kTiles; }
    static __host__ __device__ size_t list_bytes(int k) { return size_t((k + 7) / 4 * 4) * 2; }
    static __host__ __device__ size_t bytes(int k) {
        return doubles(k) * 8 + kTileWarps * (2 * size_t(8 * T) * 8 + list_bytes(k));
    }
};

__device__ __forceinline__ constexpr int tile_of(int i, int j) { return i * (i + 1) / 2 + j; }

// The sum over a quad's four lanes, in each.
__device__ __forceinline__ double quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// The sum over the eight rows, in each.
__device__ __forceinline__ double row_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// The inverse Cholesky factor of the symmetric 8x8 tile (a0, a1) in its place: Gaussian elimination of
// [A | I] without the square roots, whose rows are scaled at the end. Not inlined: six copies overran the
// instruction cache (54.4 ms against 46.6 with twelve warps).
__device__ __noinline__ double2 invert_diagonal(double a0, double a1, int lane) {
    const int r = lane >> 2, p = lane & 3;
    double e0 = r == 2 * p ? 1.0 : 0.0, e1 = r == 2 * p + 1 ? 1.0 : 0.0, d = 1.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double ak = k & 1 ? a1 : a0;
        const double pivot = __shfl_sync(0xffffffffu, ak, 4 * k + k / 2);
        const double mine = __shfl_sync(0xffffffffu, ak, 4 * r + k / 2);
        if (r == k) d = pivot;
        if (k == 7) break;
        const double r0 = __shfl_sync(0xffffffffu, a0, 4 * k + p), r1 = __shfl_sync(0xffffffffu, a1, 4 * k + p);
        const double s0 = __shfl_sync(0xffffffffu, e0, 4 * k + p), s1 = __shfl_sync(0xffffffffu, e1, 4 * k + p);
        const double factor = r > k ? -mine * (1.0 / pivot) : 0.0;
        a0 = fma(factor, r0, a0);
        a1 = fma(factor, r1, a1);
        e0 = fma(factor, s0, e0);
        e1 = fma(factor, s1, e1);
    }
    const double scale = 1.0 / sqrt(d);
    return make_double2(e0 * scale, e1 * scale);
}

// (a0, a1) += A B^T of two tiles in the accumulators' layout.
__device__ __forceinline__ void mma_tiles(double (&d)[2], double a0, double a1, const double (&b)[2]) {
    mma_f64(d[0], d[1], a0, b[0]);
    mma_f64(d[0], d[1], a1, b[1]);
}

// f of H f = rhs, both of 8 T entries in shared memory, H the lower tiles in acc (destroyed).
template <int T>
__device__ __forceinline__ void solve_tiles(double (&acc)[T * (T + 1) / 2][2], const double* rhs, double* f, int lane) {
    const int r = lane >> 2, p = lane & 3;
    double part[T], y[T];  // of L y = rhs: this lane's share of row r's sum so far, and y, by row
#pragma unroll
    for (int b = 0; b < T; ++b) part[b] = 0.0;
#pragma unroll
    for (int b = 0; b < T; ++b) {
        double(&inv)[2] = acc[tile_of(b, b)];
        const double2 factor = invert_diagonal(inv[0], inv[1], lane);
        inv[0] = factor.x;
        inv[1] = factor.y;
        const double t = rhs[8 * b + r] - quad_sum(part[b]);
        const double t0 = __shfl_sync(0xffffffffu, t, 8 * p), t1 = __shfl_sync(0xffffffffu, t, 8 * p + 4);
        y[b] = quad_sum(fma(inv[0], t0, inv[1] * t1));
        const double y0 = __shfl_sync(0xffffffffu, y[b], 8 * p), y1 = __shfl_sync(0xffffffffu, y[b], 8 * p + 4);
#pragma unroll
        for (int i = b + 1; i < T; ++i) {
            double(&x)[2] = acc[tile_of(i, b)];
            double next[2] = {0.0, 0.0};
            mma_tiles(next, x[0], x[1], inv);
            x[0] = next[0];
            x[1] = next[1];
            part[i] = fma(x[0], y0, fma(x[1], y1, part[i]));
        }
#pragma unroll
        for (int i = b + 1; i < T; ++i)
#pragma unroll
            for (int j = b + 1; j <= i; ++j)
                mma_tiles(acc[tile_of(i, j)], -acc[tile_of(i, b)][0], -acc[tile_of(i, b)][1], acc[tile_of(j, b)]);
    }
    // L^T f = y, from the last block: y becomes f, by row.
#pragma unroll
    for (int b = T - 1; b >= 0; --b) {
        double u0 = 0.0, u1 = 0.0;
#pragma unroll
        for (int i = b + 1; i < T; ++i) {
            u0 = fma(acc[tile_of(i, b)][0], y[i], u0);
            u1 = fma(acc[tile_of(i, b)][1], y[i], u1);
        }
        u0 = row_sum(u0);
        u1 = row_sum(u1);
        // By row again: entry r is the lane r / 2's of its parity.
        const double w0 = __shfl_sync(0xffffffffu, u0, r >> 1), w1 = __shfl_sync(0xffffffffu, u1, r >> 1);
        const double z = y[b] - (r & 1 ? w1 : w0);
        const double f0 = row_sum(acc[tile_of(b, b)][0] * z), f1 = row_sum(acc[tile_of(b, b)][1] * z);
        const double v0 = __shfl_sync(0xffffffffu, f0, r >> 1), v1 = __shfl_sync(0xffffffffu, f1, r >> 1);
        y[b] = r & 1 ? v1 : v0;
        if (p == 0) f[8 * b + r] = y[b];
    }
}

template <int T>
__global__ void __launch_bounds__(kTileWarps * 32, 1)
    csd_tiles_kernel(CsdDev P, const double* __restrict__ signals, int64_t v, double* __restrict__ fods,
                     uint8_t* __restrict__ converged_out) {
    using Shape = TileShape<T>;
    constexpr int kLd = Shape::kLd, kTiles = Shape::kTiles, kAtOnce = 5;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, c = P.c, k = P.k;
    double* cm = reinterpret_cast<double*>(smem);  // (k + 1, kLd)
    double* gram = cm + Shape::doubles(k) - 64 * kTiles;
    double* rhs = cm + Shape::doubles(k) + w * 2 * 8 * T;
    double* f = rhs + 8 * T;
    auto* rows = reinterpret_cast<uint16_t*>(smem + Shape::doubles(k) * 8 + kTileWarps * 2 * size_t(8 * T) * 8 +
                                             w * Shape::list_bytes(k));
    for (int e = tid; e < (k + 1) * kLd; e += kTileWarps * 32) {
        const int d = e / kLd, j = e % kLd;
        cm[e] = d < k && j < c ? P.constraint[size_t(d) * c + j] : 0.0;
    }
    for (int e = tid; e < 64 * kTiles; e += kTileWarps * 32) {
        int t = e / 64, bi = 0;
        while (t > bi) t -= ++bi;
        const int i = 8 * bi + e % 64 / 8, j = 8 * t + e % 8, hi = max(i, j), lo = min(i, j);
        gram[e] = hi < c ? P.gram[hi * (hi + 1) / 2 + lo] : (hi == lo ? 1.0 : 0.0);
    }
    __syncthreads();
    // The voxels go round the CTAs first, so that a small call has a warp on every SM.
    const int64_t n_warps = int64_t(gridDim.x) * kTileWarps;
    for (int64_t voxel = int64_t(w) * gridDim.x + blockIdx.x; voxel < v; voxel += n_warps) {
        const double* s = signals + voxel * P.m;
        for (int j = lane; j < 8 * T; j += 32) {
            double pj = 0.0, fj = 0.0;
            if (j < c)
                for (int i = 0; i < P.m; ++i) {
                    const double si = __ldg(s + i);
                    pj = fma(__ldg(P.forward + size_t(i) * c + j), si, pj);
                    if (j < P.c0) fj = fma(__ldg(P.initial_t + size_t(i) * P.c0 + j), si, fj);
                }
            rhs[j] = pj;
            f[j] = fj;
        }
        __syncwarp();
        unsigned prev = 0;  // word `lane` of the last constrained set
        bool conv = P.max_iter == 0;
        for (int it = 0; it < P.max_iter; ++it) {
            // The constrained directions, in increasing order, and as bits.
            int n_cur = 0;
            unsigned cur = 0;
            for (int d0 = 0; d0 < k; d0 += 32 * kAtOnce) {
                double a[kAtOnce];
                const double* at[kAtOnce];
#pragma unroll
                for (int u = 0; u < kAtOnce; ++u) {
                    a[u] = 0.0;
                    at[u] = cm + min(d0 + 32 * u + lane, k) * kLd;
                }
                for (int j = 0; j < c; ++j) {
                    const double fj = f[j];
#pragma unroll
                    for (int u = 0; u < kAtOnce; ++u) a[u] = fma(at[u][j], fj, a[u]);
                }
#pragma unroll
                for (int u = 0; u < kAtOnce; ++u) {
                    const int d = d0 + 32 * u + lane;
                    const bool below = d < k && a[u] < P.threshold;
                    const unsigned b = __ballot_sync(0xffffffffu, below);
                    if (below) rows[n_cur + __popc(b & ((1u << lane) - 1u))] = uint16_t(d);
                    if (lane == d0 / 32 + u) cur = b;
                    n_cur += __popc(b);
                }
            }
            if (lane < 4) rows[n_cur + lane] = uint16_t(k);  // the zero row, to a whole k-step
            __syncwarp();
            if (it > 0 && __all_sync(0xffffffffu, cur == prev)) {
                conv = true;
                break;
            }
            prev = cur;
            double acc[kTiles][2];
#pragma unroll
            for (int t = 0; t < kTiles; ++t) acc[t][0] = acc[t][1] = 0.0;
            for (int q = 0; q < n_cur; q += 4) {
                const double* row = cm + rows[q + (lane & 3)] * kLd + (lane >> 2);
                double x[T];
#pragma unroll
                for (int b = 0; b < T; ++b) x[b] = row[8 * b];
#pragma unroll
                for (int bi = 0; bi < T; ++bi)
#pragma unroll
                    for (int bj = 0; bj <= bi; ++bj) mma_f64(acc[tile_of(bi, bj)][0], acc[tile_of(bi, bj)][1], x[bi], x[bj]);
            }
#pragma unroll
            for (int t = 0; t < kTiles; ++t) {
                const double2 g = *reinterpret_cast<const double2*>(gram + 64 * t + 2 * lane);
                acc[t][0] += g.x;
                acc[t][1] += g.y;
            }
            solve_tiles<T>(acc, rhs, f, lane);
            __syncwarp();
        }
        for (int j = lane; j < c; j += 32) fods[voxel * c + j] = f[j];
        if (lane == 0) converged_out[voxel] = conv;
        __syncwarp();
    }
}

// H = gram + C_S^T C_S in T tile rows, all their lower tiles accumulated over one pass of the constrained rows.
template <int T>
__device__ __forceinline__ void build_once(const CsdDev& P, const uint16_t* cur, int n_cur, double* rows, double* H,
                                        int lane) {
    constexpr int cp = 8 * T;
    double acc[T * (T + 1) / 2][2];
#pragma unroll
    for (int t = 0; t < T * (T + 1) / 2; ++t) acc[t][0] = acc[t][1] = 0.0;
    for (int q0 = 0; q0 < n_cur; q0 += kCsdStage) {
        stage_rows(P, cur, n_cur, q0, rows, cp, lane);
#pragma unroll
        for (int kk = 0; kk < kCsdStage; kk += 4) {
            const double* rk = rows + (kk + (lane & 3)) * cp + (lane >> 2);
            double v[T];
#pragma unroll
            for (int b = 0; b < T; ++b) v[b] = rk[8 * b];
#pragma unroll
            for (int bi = 0; bi < T; ++bi)
#pragma unroll
                for (int bj = 0; bj <= bi; ++bj) mma_f64(acc[tile_of(bi, bj)][0], acc[tile_of(bi, bj)][1], v[bi], v[bj]);
        }
    }
    const int c = P.c;
#pragma unroll
    for (int bi = 0; bi < T; ++bi)
#pragma unroll
        for (int bj = 0; bj <= bi; ++bj)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 8 * bi + (lane >> 2), j = 8 * bj + 2 * (lane & 3) + h;
                if (i < c && j <= i) {
                    const int e = i * (i + 1) / 2 + j;
                    H[e] = P.gram[e] + acc[tile_of(bi, bj)][h];
                }
            }
}

// H = gram + C_S^T C_S for any c: the lower tiles kCsdBatch at a time, the rows staged again
// for each batch.
__device__ __noinline__ void build_batched(const CsdDev& P, const uint16_t* cur, int n_cur, double* rows, double* H,
                                           int lane) {
    const int c = P.c, cp = padded8(c), tiles = cp / 8, n_tiles = tiles * (tiles + 1) / 2;
    for (int t0 = 0; t0 < n_tiles; t0 += kCsdBatch) {
        double acc[kCsdBatch][2];
        int off_r[kCsdBatch], off_c[kCsdBatch];
#pragma unroll
        for (int t = 0; t < kCsdBatch; ++t) {
            acc[t][0] = acc[t][1] = 0.0;
            int idx = t0 + t, r = 0;  // tile t0 + t of the lower triangle, row by row
            while (idx > r) {
                idx -= r + 1;
                ++r;
            }
            off_r[t] = 8 * r;
            off_c[t] = 8 * idx;
        }
        for (int q0 = 0; q0 < n_cur; q0 += kCsdStage) {
            stage_rows(P, cur, n_cur, q0, rows, cp, lane);
#pragma unroll
            for (int kk = 0; kk < kCsdStage; kk += 4) {
                const double* rk = rows + (kk + (lane & 3)) * cp + (lane >> 2);
#pragma unroll
                for (int t = 0; t < kCsdBatch; ++t)
                    if (t0 + t < n_tiles) mma_f64(acc[t][0], acc[t][1], rk[off_r[t]], rk[off_c[t]]);
            }
        }
#pragma unroll
        for (int t = 0; t < kCsdBatch; ++t) {
            if (t0 + t >= n_tiles) continue;
            const int i = off_r[t] + (lane >> 2);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = off_c[t] + 2 * (lane & 3) + h;
                if (i < c && j <= i) {
                    const int e = i * (i + 1) / 2 + j;
                    H[e] = P.gram[e] + acc[t][h];
                }
            }
        }
    }
}

// TILES: the system's tile rows, built by build_once, or 0 for build_batched.
template <int TILES>
__global__ void csd_kernel(CsdDev P, const double* __restrict__ signals, int64_t v, double* __restrict__ fods,
                           uint8_t* __restrict__ converged_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int c = P.c, k = P.k, npk = packed_count(c);
    unsigned char* base = smem + size_t(w) * csd_warp_bytes(c, k);
    double* H = reinterpret_cast<double*>(base);
    double* f = H + npk;
    double* rhs = f + c;
    double* y = rhs + c;
    double* rows = y + c;
    auto* list_a = reinterpret_cast<uint16_t*>(rows + kCsdStage * padded8(c));
    uint16_t* list_b = list_a + k;
    const int64_t n_warps = int64_t(gridDim.x) * warps;
    for (int64_t voxel = int64_t(blockIdx.x) * warps + w; voxel < v; voxel += n_warps) {
        const double* s = signals + voxel * P.m;
        for (int j = lane; j < c; j += 32) {
            double pj = 0.0, fj = 0.0;
            for (int i = 0; i < P.m; ++i) {
                const double si = s[i];
                pj = fma(P.forward[size_t(i) * c + j], si, pj);
                if (j < P.c0) fj = fma(P.initial_t[size_t(i) * P.c0 + j], si, fj);
            }
            rhs[j] = pj;
            f[j] = fj;
        }
        __syncwarp();
        uint16_t* cur = list_a;
        uint16_t* prev = list_b;
        int n_prev = -1;
        bool conv = P.max_iter == 0;
        for (int it = 0; it < P.max_iter; ++it) {
            // The constrained directions, in increasing order.
            int n_cur = 0;
            for (int d0 = 0; d0 < k; d0 += 32) {
                const int d = d0 + lane;
                bool below = false;
                if (d < k) {
                    double a = 0.0;
                    for (int j = 0; j < c; ++j) a = fma(P.constraint_t[size_t(j) * k + d], f[j], a);
                    below = a < P.threshold;
                }
                const unsigned b = __ballot_sync(0xffffffffu, below);
                if (below) cur[n_cur + __popc(b & ((1u << lane) - 1u))] = uint16_t(d);
                n_cur += __popc(b);
            }
            __syncwarp();
            if (n_prev == n_cur) {
                bool same = true;
                for (int q = lane; q < n_cur; q += 32) same &= cur[q] == prev[q];
                if (__all_sync(0xffffffffu, same)) {
                    conv = true;
                    break;
                }
            }
            // The system: the Gram matrix plus C_S^T C_S, the constrained rows' product on the
            // tensor cores over the rows staged kCsdStage at a time (zero-padded to whole tiles
            // and k-steps).
            if constexpr (TILES > 0)
                build_once<TILES>(P, cur, n_cur, rows, H, lane);
            else
                build_batched(P, cur, n_cur, rows, H, lane);
            __syncwarp();
            // Left-looking Cholesky, packed in place: column j's entries from the finished
            // columns, one row per lane; lane 0 holds the diagonal.
            for (int j = 0; j < c; ++j) {
                const double* lj = H + j * (j + 1) / 2;
                double val[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = j + lane + 32 * u;
                    val[u] = 0.0;
                    if (i < c) {
                        const double* li = H + i * (i + 1) / 2;
                        double a = li[j];
                        for (int q = 0; q < j; ++q) a -= li[q] * lj[q];
                        val[u] = a;
                    }
                }
                const double d = sqrt(__shfl_sync(0xffffffffu, val[0], 0));
                __syncwarp();
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = j + lane + 32 * u;
                    if (i < c) H[i * (i + 1) / 2 + j] = i == j ? d : val[u] / d;
                }
                for (int i = j + 64 + lane; i < c; i += 32) {
                    const double* li = H + i * (i + 1) / 2;
                    double a = li[j];
                    for (int q = 0; q < j; ++q) a -= li[q] * lj[q];
                    H[i * (i + 1) / 2 + j] = a / d;
                }
                __syncwarp();
            }
            // L y = rhs, then L^T f = y.
            for (int q = lane; q < c; q += 32) y[q] = rhs[q];
            __syncwarp();
            for (int i = 0; i < c; ++i) {
                const double yi = y[i] / H[i * (i + 1) / 2 + i];
                __syncwarp();
                if (lane == 0) y[i] = yi;
                for (int r = i + 1 + lane; r < c; r += 32) y[r] -= H[r * (r + 1) / 2 + i] * yi;
                __syncwarp();
            }
            for (int i = c - 1; i >= 0; --i) {
                const int row = i * (i + 1) / 2;
                const double fi = y[i] / H[row + i];
                __syncwarp();
                if (lane == 0) f[i] = fi;
                for (int r = lane; r < i; r += 32) y[r] -= H[row + r] * fi;
                __syncwarp();
            }
            uint16_t* t = prev;
            prev = cur;
            cur = t;
            n_prev = n_cur;
        }
        for (int j = lane; j < c; j += 32) fods[voxel * c + j] = f[j];
        if (lane == 0) converged_out[voxel] = conv;
        __syncwarp();
    }
}

// Launches csd_tiles_kernel<T> when C fits the shared memory.
template <int T>
bool launch_tiles(const CsdDev& P, const double* signals, int64_t v, double* fods, uint8_t* converged,
                  cudaStream_t st) {
    const size_t smem = TileShape<T>::bytes(P.k);
    if (P.k > 1024 || smem > 220 * 1024) return false;  // (a set is a word per lane)
    allow_smem(csd_tiles_kernel<T>, smem);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, csd_tiles_kernel<T>, kTileWarps * 32, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const int64_t blocks =
        std::max<int64_t>(1, std::min<int64_t>(v, int64_t(sm_count()) * ctas_per_sm(per_sm, "csd.ctas_per_sm")));
    LaunchScope scope("csd_kernel", st);
    csd_tiles_kernel<T><<<unsigned(blocks), kTileWarps * 32, smem, st>>>(P, signals, v, fods, converged);
    cuda_check(cudaGetLastError(), "csd_tiles_kernel launch");
    return true;
}

}  // namespace
}  // namespace lar

// The matrices of one shell's CSD fit on the device (the reference's CsdProblem,
// cpp/src/sd/csd.hpp:10-24).
struct lar_csd_s {
    int m = 0, c = 0, c0 = 0, k = 0, max_iter = 0;
    double threshold = 0.0;
    lar::DeviceArray<double> initial_t, forward, constraint, constraint_t, gram;
};

using namespace lar;

extern "C" {

int lar_csd_create(const double* initial, int64_t c0, int64_t m, const double* forward, int64_t c,
                   const double* constraint, int64_t k, double norm_weight, double threshold, int64_t max_iter,
                   lar_csd* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(m > 0 && c > 0 && k > 0 && c0 >= 0, "the matrices must not be empty");
        require(c0 <= c, "initial must not have more rows than forward has columns");
        require(c <= 255 && k <= 65535, "at most 255 coefficients and 65535 constraint directions");
        require(max_iter >= 0, "max_iter must be at least 0");
        require(forward && constraint && (c0 == 0 || initial), "the matrices must not be NULL");
        require(csd_warp_bytes(int(c), int(k)) <= 220 * 1024,
                "the system does not fit one warp's shared memory: too many coefficients or directions");
        auto h = std::make_unique<lar_csd_s>();
        h->m = int(m);
        h->c = int(c);
        h->c0 = int(c0);
        h->k = int(k);
        h->max_iter = int(max_iter);
        h->threshold = threshold;
        std::vector<double> it(static_cast<size_t>(m * std::max<int64_t>(c0, 1)), 0.0);
        std::vector<double> ct(static_cast<size_t>(c * k));
        std::vector<double> gram(static_cast<size_t>(packed_count(int(c))));
        for (int64_t r = 0; r < c0; ++r)
            for (int64_t i = 0; i < m; ++i) it[size_t(i * c0 + r)] = initial[r * m + i];
        for (int64_t d = 0; d < k; ++d)
            for (int64_t j = 0; j < c; ++j) ct[size_t(j * k + d)] = constraint[d * c + j];
        // cpp/src/sd/csd.cpp:13-14: M^T M with norm_weight on its diagonal.
        for (int64_t i = 0; i < c; ++i)
            for (int64_t j = 0; j <= i; ++j) {
                double acc = 0.0;
                for (int64_t r = 0; r < m; ++r) acc += forward[r * c + i] * forward[r * c + j];
                gram[size_t(i * (i + 1) / 2 + j)] = acc + (i == j ? norm_weight : 0.0);
            }
        h->initial_t.upload(it.data(), it.size());
        h->forward.upload(forward, size_t(m * c));
        h->constraint.upload(constraint, size_t(k * c));
        h->constraint_t.upload(ct.data(), ct.size());
        h->gram.upload(gram.data(), gram.size());
        *out = h.release();
    });
}

void lar_csd_destroy(lar_csd csd) { delete csd; }

int lar_fit_csd(lar_csd csd, const double* signals, int64_t v, double* fods, uint8_t* converged, void* stream) {
    return guarded([&] {
        require(csd != nullptr, "csd must not be NULL");
        require(v >= 0, "v must be at least 0");
        if (v == 0) return;
        require(signals && fods && converged, "signals, fods and converged must not be NULL");
        auto st = static_cast<cudaStream_t>(stream);
        const CsdDev P{csd->initial_t.ptr, csd->forward.ptr, csd->constraint.ptr, csd->constraint_t.ptr,
                       csd->gram.ptr, csd->m, csd->c, csd->c0, csd->k, csd->max_iter, csd->threshold};
        // The accumulators hold systems of up to 48 coefficients, in as few tiles as cover them.
        if (csd->c <= 16 && launch_tiles<2>(P, signals, v, fods, converged, st)) return;
        if (csd->c > 16 && csd->c <= 32 && launch_tiles<4>(P, signals, v, fods, converged, st)) return;
        if (csd->c > 32 && csd->c <= 8 * kTileRows && launch_tiles<kTileRows>(P, signals, v, fods, converged, st)) return;
        const size_t per_warp = csd_warp_bytes(csd->c, csd->k);
        const int warps = int(std::max<size_t>(1, std::min<size_t>(4, (200 * 1024) / per_warp)));
        const size_t smem = per_warp * warps;
        // Systems of four to six tile rows whose constraints are too many for the CTA's shared memory (past some
        // 475 directions at 45 coefficients): one pass of the rows, where the batches stage them two or three times
        // (20,000 voxels: 45 coefficients on 642 directions 12.1 against 32.9 ms, 28 on 900 6.5 against 16.0). With
        // fewer tile rows one batch is one pass; with more the accumulators would not fit.
        const int tiles = padded8(csd->c) / 8;
        auto kernel = tiles == 4 ? csd_kernel<4> : tiles == 5 ? csd_kernel<5> : tiles == 6 ? csd_kernel<6> : csd_kernel<0>;
        allow_smem(kernel, smem);
        int per_sm = 0;
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        const int64_t blocks = std::max<int64_t>(
            1, std::min<int64_t>((v + warps - 1) / warps, int64_t(sm_count()) * ctas_per_sm(per_sm, "csd.ctas_per_sm")));
        LaunchScope scope("csd_kernel", st);
        kernel<<<unsigned(blocks), warps * 32, smem, st>>>(P, signals, v, fods, converged);
        cuda_check(cudaGetLastError(), "csd_kernel launch");
    });
}

}  // extern "C"
