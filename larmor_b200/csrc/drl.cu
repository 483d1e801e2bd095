// Damped Richardson-Lucy (dRL) deconvolution on the GPU: FodSolver.drl + fit_single_tissue
// (cpp/src/python/sd.cpp:127-145, cpp/src/sd/solver.cpp:9-12) over damped_richardson_lucy
// (cpp/src/sd/drl.cpp:39-100). Dell'Acqua F et al., NeuroImage 49 (2010) 1446-1458.
//
// Each voxel starts every amplitude at `init`. An iteration computes the prediction p = K^T K f
// and moves each amplitude to max(f (1 + u (K^T s - p) / (p + 1e-16)), 1e-6). The damping is
// u = 1 - strength (1 - f^8 / (f^8 + nu^8)), with strength = max(1 - 4 std(s), 0). A voxel
// stops when its amplitudes change in total by no more than 1e-4 of its largest signal value.
//
// Mapping: a CTA of 8 warps takes 8 RT voxels at a time (32 up to 320 directions, 16 up to 640; fewer in a
// list's last wave, launch_narrow)
// and keeps their FODs F (8 RT, c) and K^T s (8 RT, c) in shared memory for all their
// iterations. An iteration is one product F K^T K on the FP64 tensor cores: mma.sync m8n8k4
// over the RT 8-voxel row tiles and the 8-direction column tiles, which the warps take
// round-robin. K^T K (c x c, 720 KB at c = 300) stays in L2. A warp's columns are no other warp's, so it
// reads them straight into its fragments, one to three groups of eight k ahead of their use and the
// first before the update, and the warps meet only around the update: through a shared-memory stage, with
// two barriers per eight k, the tensor cores stood still most of the time. The two k-steps of a group take
// its even and its odd k, so that a lane's two operands lie side by side in a row of K^T K and of F (16-byte
// loads). K^T s is the same product of the signals with K^T. The update is the epilogue, on the
// accumulators, after a barrier, since every warp reads all of F. Each voxel's change is reduced in
// a fixed order, so the stopping test does not depend on the schedule. Converged voxels keep their
// FOD while the tile's others iterate.
//
// What bounds it: the FP64 pipe. 100,003 voxels, 300 directions, 200 iterations: 134 ms, of which the
// products take 97 at the tensor cores' rate and 8 more for the columns past the 38th tile (through the
// stage: 261 ms). With 32 voxels to a CTA and 8 warps nothing hides the update behind another tile's
// products: two CTAs would need K^T K's traffic twice.
//
// Up to 64 directions the whole K^T K (at most 36 KB) is loaded once per CTA instead
// (drl_resident_kernel), and the CTA then fits in half an SM.
//
// The multi-tissue rounds (GRL, cpp/src/sd/multi_tissue.cpp:40-95) run the same solve on a list
// of voxels whose signal is the anisotropic part max(s w - W_iso f_iso, 0) of the round.

#include <algorithm>
#include <cmath>

#include <math_constants.h>

#include "common.cuh"
#include "drl.cuh"

namespace lar {
namespace {

constexpr int kDrlWarps = 8;
constexpr int kGroup = 8;  // k values of a group: two k-steps
// RT 8-voxel row tiles per CTA, up to MAXCT column tiles per warp, for c <= 8 * kDrlWarps * MAXCT directions.
constexpr int kNarrowRt = 4, kNarrowCt = 5;   // 32 voxels, c <= 320
constexpr int kWideRt = 2, kWideCt = 10;      // 16 voxels, c <= 640
constexpr int kNarrowMaxC = 8 * kDrlWarps * kNarrowCt;
constexpr int kWideMaxC = 8 * kDrlWarps * kWideCt;
// Up to 64 directions (the low-resolution kernels of the multi-tissue rounds) all of K^T K stays
// in shared memory for the CTA's life: 32 voxels, one column tile per warp, two CTAs per SM.
constexpr int kResidentMaxC = 8 * kDrlWarps;

// Row strides (doubles) for cp columns, in the resident kernel of F and K^T s, and of K^T K: the padding puts
// the 8 rows of an A fragment, and the 4 rows of a B fragment, in different banks. In the streaming kernel of
// F and K^T s: 8 more than a multiple of 16, so that two rows' 64 bytes of a fragment are in different banks.
__host__ __device__ inline int drl_ldf(int cp) { return cp + 4; }
__host__ __device__ inline int drl_ldg(int cp) { return cp + 8; }
__host__ __device__ inline int drl_lds(int cp) { return cp % 16 == 8 ? cp : cp + 8; }

__device__ __forceinline__ double power_8(double x) {
    const double x2 = x * x, x4 = x2 * x2;
    return x4 * x4;
}

__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Entry i of the signal of `voxel` that dRL deconvolves.
__device__ __forceinline__ double signal_at(const DrlSignal& S, int64_t voxel, int i) {
    const double si = S.s[voxel * S.m + i];
    if (S.w == nullptr) return si;
    const double ws = __dmul_rn(si, S.w[i]);
    double r = 0.0;
    for (int t = 0; t < S.ci; ++t) r = fma(S.wiso[size_t(i) * S.ci + t], S.fiso[voxel * S.ci + t], r);
    return fmax(ws - r, 0.0);
}

// The voxels of a tile from list entry p0, each one's damping strength (1 - 4 x the sample standard
// deviation, at least 0) and stopping threshold (1e-4 x its largest non-NaN signal value).
template <int ROWS>
struct DrlTile {
    double part[kDrlWarps][ROWS];
    double strength[ROWS], threshold[ROWS];
    int active[ROWS];
    int64_t vox[ROWS];
};

template <int ROWS>
__device__ __forceinline__ void open_tile(DrlTile<ROWS>& t, const DrlSignal& S, int m, const int* __restrict__ list,
                                          int64_t p0, int64_t count) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < ROWS) t.vox[tid] = p0 + tid < count ? (list ? int64_t(list[p0 + tid]) : p0 + tid) : -1;
    __syncthreads();
    for (int r = warp; r < ROWS; r += kDrlWarps) {
        const int64_t voxel = t.vox[r];
        if (voxel < 0) {
            if (lane == 0) {
                t.active[r] = 0;
                t.strength[r] = t.threshold[r] = 0.0;
            }
            continue;
        }
        double sum = 0.0, mx = -CUDART_INF;
        bool any = false;
        for (int i = lane; i < m; i += 32) {
            const double si = signal_at(S, voxel, i);
            sum += si;
            if (!isnan(si)) {
                mx = any ? fmax(mx, si) : si;
                any = true;
            }
        }
        const double mean = warp_sum(sum) / m;
        double ss = 0.0;
        for (int i = lane; i < m; i += 32) {
            const double si = signal_at(S, voxel, i);
            ss += (si - mean) * (si - mean);
        }
        ss = warp_sum(ss);
        const bool all_nan = !__any_sync(0xffffffffu, any);
        mx = warp_max(any ? mx : -CUDART_INF);
        if (lane == 0) {
            t.strength[r] = fmax(1.0 - 4.0 * sqrt(ss / double(m - 1)), 0.0);
            t.threshold[r] = 1e-4 * (all_nan ? CUDART_NAN : mx);
            t.active[r] = 1;
        }
    }
}

// The update's relative step as it is written (cpp/src/sd/drl.cpp:13-20).
__device__ __noinline__ double plain_step(double f8, double nu8, double strength, double ks, double pred) {
    return (1.0 - strength * (1.0 - f8 / (f8 + nu8))) * ((ks - pred) / (pred + 1e-16));
}

// Whether |x| lies between about 1e-200 and 1e200 (by its exponent).
__device__ __forceinline__ bool mid_range(double x) {
    return ((unsigned(__double2hiint(x)) >> 20) & 0x7ffu) - 359u <= 1328u;
}

// The damped update of the still-active voxels from the prediction acc (column tile t of the warp in
// acc[.][t]), each one's total change into part, and whether any voxel is still active. The damping
// 1 - strength (1 - f^8 / (f^8 + nu^8)) and the ratio (K^T s - p) / (p + 1e-16) have the product of their
// denominators below one fraction bar, and a lane's two entries share one reciprocal of both products (Montgomery,
// Math. Comp. 48 (1987) 243-264): 100,003 voxels of 300 directions, 200 iterations, 133.6 ms, with a reciprocal each
// 138.5, with a division each 143.5. Where that is 0, out of the middle of the range or not a number, the two are
// taken as written.
template <int RT, int CT>
__device__ __forceinline__ bool update_tile(DrlTile<8 * RT>& tile, const double (&acc)[RT][CT][2], double* F,
                                            const double* KS, int ld, int c, double nu8) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
        const int r = 8 * rt + (lane >> 2);
        double change = 0.0;
        if (tile.active[r]) {
            const double off = (1.0 - tile.strength[r]) * nu8;
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                const int d = 8 * (warp + kDrlWarps * t) + 2 * (lane & 3);
                double* at = F + r * ld + d;
                double2 f = make_double2(1.0, 1.0), ks = make_double2(0.0, 0.0);
                if (d < c) {  // a column of no one's is neither read nor written
                    f = *reinterpret_cast<const double2*>(at);
                    ks = *reinterpret_cast<const double2*>(KS + (at - F));
                }
                double below[2], step[2], to[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double f8 = power_8(h ? f.y : f.x), pred = acc[rt][t][h];
                    below[h] = (f8 + nu8) * (pred + 1e-16);
                    step[h] = (f8 + off) * ((h ? ks.y : ks.x) - pred);
                }
                const double both = below[0] * below[1], inverse = __drcp_rn(both);
                step[0] *= inverse * below[1];
                step[1] *= inverse * below[0];
                if (!mid_range(both)) {
                    step[0] = plain_step(power_8(f.x), nu8, tile.strength[r], ks.x, acc[rt][t][0]);
                    step[1] = plain_step(power_8(f.y), nu8, tile.strength[r], ks.y, acc[rt][t][1]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double fh = h ? f.y : f.x;
                    to[h] = fmax(fh * (1.0 + step[h]), 1e-6);
                    if (d + h < c) change += fabs(to[h] - fh);
                }
                if (d < c) at[0] = to[0];
                if (d + 1 < c) at[1] = to[1];
            }
        }
        change += __shfl_xor_sync(0xffffffffu, change, 1);
        change += __shfl_xor_sync(0xffffffffu, change, 2);
        if ((lane & 3) == 0) tile.part[warp][r] = change;
    }
    __syncthreads();
    int alive = 0;
    if (tid < 8 * RT && tile.active[tid]) {
        double total = 0.0;
        for (int w = 0; w < kDrlWarps; ++w) total += tile.part[w][tid];
        alive = !(total <= tile.threshold[tid]);
        tile.active[tid] = alive;
    }
    return __syncthreads_or(alive);
}

// x(list[p], :) = the dRL FOD of voxel list[p] for p < count (min(count, *count_dev) when
// count_dev is given); no list: voxel p itself.
__global__ void __launch_bounds__(kDrlWarps * 32, 2)
    drl_resident_kernel(DrlDev P, DrlSignal S, const int* __restrict__ list, int64_t count,
                        const int* __restrict__ count_dev, double* __restrict__ x, int64_t ldx) {
    constexpr int RT = kNarrowRt, kRows = 8 * RT;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ DrlTile<kRows> tile;
    if (count_dev) count = min(count, int64_t(*count_dev));
    const int c = P.c, m = P.m, cp = (c + 7) / 8 * 8, ldf = drl_ldf(cp), ldg = drl_ldg(cp);
    double* F = reinterpret_cast<double*>(smem);  // (kRows, ldf)
    double* KS = F + kRows * ldf;                 // (kRows, ldf)
    double* GS = KS + kRows * ldf;                // (cp, ldg)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double nu8 = power_8(P.nu);
    // All of K^T K, zero past c (made visible by the barrier at the first tile's start).
    for (int e = threadIdx.x; e < cp * ldg; e += blockDim.x) {
        const int k = e / ldg, d = e - k * ldg;
        GS[e] = (k < c && d < c) ? P.gram[size_t(k) * c + d] : 0.0;
    }
    for (int64_t p0 = int64_t(blockIdx.x) * kRows; p0 < count; p0 += int64_t(gridDim.x) * kRows) {
        open_tile(tile, S, m, list, p0, count);
        // K^T s and the start.
        for (int e = tid; e < kRows * ldf; e += blockDim.x) {
            const int r = e / ldf, d = e - r * ldf;
            const int64_t voxel = tile.vox[r];
            const bool real = voxel >= 0 && d < c;
            double ks = 0.0;
            if (real) {
                const double* kt = P.k_t + size_t(d) * m;
                for (int i = 0; i < m; ++i) ks = fma(kt[i], signal_at(S, voxel, i), ks);
            }
            KS[e] = ks;
            F[e] = real ? P.init : 0.0;
        }
        __syncthreads();
        for (int it = 0; it < P.n_iter; ++it) {
            // The prediction K^T K f of every voxel of the tile (K^T K is symmetric: its column
            // block is read as rows).
            double acc[RT][1][2];
#pragma unroll
            for (int rt = 0; rt < RT; ++rt) acc[rt][0][0] = acc[rt][0][1] = 0.0;
            if (8 * warp < cp)
                for (int k0 = 0; k0 < cp; k0 += 4) {
                    const int kk = k0 + (lane & 3);
                    const double b = GS[kk * ldg + 8 * warp + (lane >> 2)];
#pragma unroll
                    for (int rt = 0; rt < RT; ++rt)
                        mma_f64(acc[rt][0][0], acc[rt][0][1], F[(8 * rt + (lane >> 2)) * ldf + kk], b);
                }
            // The update overwrites F: every warp is done reading it first.
            __syncthreads();
            if (!update_tile<RT, 1>(tile, acc, F, KS, ldf, c, nu8)) break;
        }
        for (int e = tid; e < kRows * ldf; e += blockDim.x) {
            const int r = e / ldf, d = e - r * ldf;
            const int64_t voxel = tile.vox[r];
            if (voxel >= 0 && d < c) x[voxel * ldx + d] = F[e];
        }
        __syncthreads();
    }
}

// Columns 8 (warp + 8 t) + {0..7}, t < CT, of A B^T for a tile's rows A (8 RT, k) in shared memory and B
// (n, k) row-major in global memory: B's fragments through registers, DEPTH groups of eight k in flight.
template <int RT, int CT>
struct StreamedProduct {
    static constexpr int DEPTH = CT >= 4 ? 2 : 4;
    double2 b[DEPTH][CT];
    const double* row[CT];  // of this lane's column in tile t, at its first k
    int k;                  // k values, and this lane's next group is at k0
    bool wide;              // rows of B start on 16 bytes

    __device__ __forceinline__ void open(const double* __restrict__ B, int64_t ldb, int n, int from, int count) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        k = count;
        wide = ldb % 2 == 0 && from % 2 == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0;
#pragma unroll
        for (int t = 0; t < CT; ++t)  // a column past the last reads the last, and no one its product
            row[t] = B + int64_t(min(8 * (warp + kDrlWarps * t) + (lane >> 2), n - 1)) * ldb + from + 2 * (lane & 3);
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) fetch(u, u * kGroup);
    }

    __device__ __forceinline__ void fetch(int u, int k0) {
        if (k0 >= k) return;
        const int at = k0 + 2 * (threadIdx.x & 3);
        if (wide && k0 + kGroup <= k) {
#pragma unroll
            for (int t = 0; t < CT; ++t) b[u][t] = __ldcg(reinterpret_cast<const double2*>(row[t] + k0));
        } else {
#pragma unroll
            for (int t = 0; t < CT; ++t)
                b[u][t] = make_double2(at < k ? __ldcg(row[t] + k0) : 0.0, at + 1 < k ? __ldcg(row[t] + k0 + 1) : 0.0);
        }
    }

    // acc += the product; A has zeros from column k to the end of its last group.
    __device__ __forceinline__ void run(double (&acc)[RT][CT][2], const double* A, int ld) {
        const int lane = threadIdx.x & 31;
        const double* mine = A + (lane >> 2) * ld + 2 * (lane & 3);
        for (int k0 = 0; k0 < k; k0 += DEPTH * kGroup) {
#pragma unroll
            for (int u = 0; u < DEPTH; ++u) {
                const int at = k0 + u * kGroup;
                if (at < k) {
                    double2 a[RT];
#pragma unroll
                    for (int rt = 0; rt < RT; ++rt) a[rt] = *reinterpret_cast<const double2*>(mine + 8 * rt * ld + at);
#pragma unroll
                    for (int t = 0; t < CT; ++t)
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt) mma_f64(acc[rt][t][0], acc[rt][t][1], a[rt].x, b[u][t].x);
#pragma unroll
                    for (int t = 0; t < CT; ++t)
#pragma unroll
                        for (int rt = 0; rt < RT; ++rt) mma_f64(acc[rt][t][0], acc[rt][t][1], a[rt].y, b[u][t].y);
                    fetch(u, at + DEPTH * kGroup);
                }
            }
        }
    }
};

template <int RT, int CT>
__global__ void __launch_bounds__(kDrlWarps * 32, 1)
    drl_kernel(DrlDev P, DrlSignal S, const int* __restrict__ list, int64_t count, const int* __restrict__ count_dev,
               double* __restrict__ x, int64_t ldx) {
    constexpr int kRows = 8 * RT;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ DrlTile<kRows> tile;
    if (count_dev) count = min(count, int64_t(*count_dev));
    const int c = P.c, m = P.m, cp = (c + 7) / 8 * 8, ld = drl_lds(cp);
    double* F = reinterpret_cast<double*>(smem);  // (kRows, ld)
    double* KS = F + kRows * ld;                  // (kRows, ld)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double nu8 = power_8(P.nu);
    StreamedProduct<RT, CT> product;
    double acc[RT][CT][2];
    auto clear = [&] {
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int t = 0; t < CT; ++t) acc[rt][t][0] = acc[rt][t][1] = 0.0;
    };
    for (int64_t p0 = int64_t(blockIdx.x) * kRows; p0 < count; p0 += int64_t(gridDim.x) * kRows) {
        open_tile(tile, S, m, list, p0, count);
        // K^T s: the signals in F, cp measurements at a time.
        clear();
        for (int from = 0; from < m; from += cp) {
            const int here = min(cp, m - from);
            product.open(P.k_t, m, c, from, here);
            for (int e = tid; e < kRows * cp; e += blockDim.x) {
                const int r = e / cp, i = e - r * cp;
                const int64_t voxel = tile.vox[r];
                F[r * ld + i] = voxel >= 0 && i < here ? signal_at(S, voxel, from + i) : 0.0;
            }
            __syncthreads();
            product.run(acc, F, ld);
            __syncthreads();
        }
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                const int d = 8 * (warp + kDrlWarps * t) + 2 * (lane & 3);
                if (d < cp)
                    *reinterpret_cast<double2*>(KS + (8 * rt + (lane >> 2)) * ld + d) =
                        make_double2(acc[rt][t][0], acc[rt][t][1]);
            }
        for (int e = tid; e < kRows * cp; e += blockDim.x) {
            const int r = e / cp, d = e - r * cp;
            F[r * ld + d] = tile.vox[r] >= 0 && d < c ? P.init : 0.0;
        }
        if (P.n_iter > 0) product.open(P.gram, c, c, 0, c);
        __syncthreads();
        for (int it = 0; it < P.n_iter; ++it) {
            // The prediction K^T K f of every voxel of the tile.
            clear();
            product.run(acc, F, ld);
            if (it + 1 < P.n_iter) product.open(P.gram, c, c, 0, c);
            // The update overwrites F: every warp is done reading it first.
            __syncthreads();
            if (!update_tile<RT, CT>(tile, acc, F, KS, ld, c, nu8)) break;
        }
        for (int e = tid; e < kRows * cp; e += blockDim.x) {
            const int r = e / cp, d = e - r * cp;
            const int64_t voxel = tile.vox[r];
            if (voxel >= 0 && d < c) x[voxel * ldx + d] = F[r * ld + d];
        }
        __syncthreads();
    }
}

template <int RT, typename Kernel>
void launch_variant(Kernel kernel, const DrlDev& P, const DrlSignal& S, const int* list, int64_t count,
                    const int* count_dev, double* x, int64_t ldx, cudaStream_t st, const char* name, size_t smem) {
    allow_smem(kernel, smem);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kDrlWarps * 32, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const int64_t tiles = (count + 8 * RT - 1) / (8 * RT);
    const int64_t blocks =
        std::max<int64_t>(1, std::min<int64_t>(tiles, int64_t(sm_count()) * ctas_per_sm(per_sm, "drl.ctas_per_sm")));
    LaunchScope scope(name, st);
    kernel<<<unsigned(blocks), kDrlWarps * 32, smem, st>>>(P, S, list, count, count_dev, x, ldx);
    cuda_check(cudaGetLastError(), "drl_kernel launch");
}

// The streaming kernel with RT row tiles and as many column tiles per warp as c needs: the products of a warp's
// columns past c are wasted.
template <int RT>
void launch_streamed(const DrlDev& P, const DrlSignal& S, const int* list, int64_t count, const int* count_dev,
                     double* x, int64_t ldx, cudaStream_t st) {
    const int ct = (P.c + 8 * kDrlWarps - 1) / (8 * kDrlWarps);
    const size_t smem = 2 * size_t(8 * RT) * drl_lds((P.c + 7) / 8 * 8) * sizeof(double);
    launch_variant<RT>(ct <= 2   ? drl_kernel<RT, 2>
                       : ct == 3 ? drl_kernel<RT, 3>
                       : ct == 4 ? drl_kernel<RT, 4>
                                 : drl_kernel<RT, kNarrowCt>,
                       P, S, list, count, count_dev, x, ldx, st, "drl_kernel", smem);
}

// Up to 320 directions: whole waves of 32-voxel tiles, a CTA on every SM, then what is left of the list in tiles
// small enough to be one wave too. A tile's time is nearly its rows', so a wave of few 32-voxel
// tiles takes as long as a full one (300 directions, 200 iterations: 6.1 ms for any number of 32-voxel tiles up to
// a wave; 2.6 ms for 1,184 voxels and 3.5 for 2,368 in the smaller ones, whose warps read all of K^T K for
// fewer products). A count on the device is not known here.
void launch_narrow(const DrlDev& P, const DrlSignal& S, const int* list, int64_t count, const int* count_dev, double* x,
                   int64_t ldx, cudaStream_t st) {
    const int64_t wave = int64_t(sm_count()) * 8;
    const int64_t rest = count_dev != nullptr ? count : count % (4 * wave), whole = count - rest;
    if (count_dev != nullptr || rest > 2 * wave || rest == 0) {
        launch_streamed<4>(P, S, list, count, count_dev, x, ldx, st);
        return;
    }
    if (whole > 0) launch_streamed<4>(P, S, list, whole, nullptr, x, ldx, st);
    DrlSignal after = S;
    if (list != nullptr) {
        list += whole;
    } else {
        after.s += whole * S.m;
        if (S.fiso != nullptr) after.fiso += whole * S.ci;
        x += whole * ldx;
    }
    if (rest > wave)
        launch_streamed<2>(P, after, list, rest, nullptr, x, ldx, st);
    else
        launch_streamed<1>(P, after, list, rest, nullptr, x, ldx, st);
}

}  // namespace

size_t drl_smem_bytes(int c) {
    const int cp = (c + 7) / 8 * 8;
    if (c <= kResidentMaxC) return (2 * size_t(8 * kNarrowRt) * drl_ldf(cp) + size_t(cp) * drl_ldg(cp)) * sizeof(double);
    const size_t rows = c <= kNarrowMaxC ? 8 * kNarrowRt : 8 * kWideRt;
    return 2 * rows * drl_lds(cp) * sizeof(double);
}

bool drl_fits(int c) { return c >= 1 && c <= kWideMaxC; }

void launch_drl_listed(const DrlDev& P, const DrlSignal& S, const int* list, int64_t count, const int* count_dev,
                       double* x, int64_t ldx, cudaStream_t st) {
    if (count == 0) return;
    if (P.gtc != nullptr && drl_tc_fits(P.c) && drl_tc_fits_measurements(P.c, P.m)) {
        launch_drl_tc(P, P.gtc, S, list, count, count_dev, x, ldx, P.err, st);
        return;
    }
    if (P.c <= kResidentMaxC)
        launch_variant<kNarrowRt>(drl_resident_kernel, P, S, list, count, count_dev, x, ldx, st, "drl_kernel_resident",
                                  drl_smem_bytes(P.c));
    else if (P.c <= kNarrowMaxC)
        launch_narrow(P, S, list, count, count_dev, x, ldx, st);
    else
        launch_variant<kWideRt>(P.c <= 8 * kDrlWarps * 7 ? drl_kernel<kWideRt, 7> : drl_kernel<kWideRt, kWideCt>, P, S,
                                list, count, count_dev, x, ldx, st, "drl_kernel_wide", drl_smem_bytes(P.c));
}

void launch_drl(const DrlDev& P, const double* signals, int64_t v, double* fods, cudaStream_t st) {
    launch_drl_listed(P, DrlSignal{signals, nullptr, nullptr, nullptr, P.m, 0}, nullptr, v, nullptr, fods, P.c, st);
}

}  // namespace lar
