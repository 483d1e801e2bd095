// FOD peaks on the GPU: the amplitude of a tournier-basis SH series and its derivatives on the
// sphere (cpp/src/sh/harmonics.cpp:139-196), the Newton climb to a peak (cpp/src/sh/peaks.cpp:
// 31-78) and the peak search of each voxel from the local maxima of its amplitudes on a sphere
// (cpp/src/sh/peaks.cpp:80-133), behind _core.sh_derivatives, _core.climb and _core.peaks_chunk
// (cpp/src/python/sh.cpp:69-176).
//
// Layout and mapping:
// - The Legendre table is built one degree at a time: row l of P(l, m) needs only rows l-1 and
//   l-2 (the recurrence runs along the degree for each order), and the derivative terms of
//   degree l need only row l (the ladder formulas mix orders m-2..m+2 of one degree). So three
//   rows of LCAP+1 values stay in registers instead of a (lmax+1)^2 table.
// - The constants that depend only on (l, m) (the diagonal start, the recurrence factors, the
//   ladder factors, combined per term) are tables in constant memory, computed on the host from the
//   reference's formulas and uploaded once per device.
// - The search runs in passes over one list of all the chunk's climbs (see "the peak search in
//   passes" below): a voxel has ~5-15 local maxima of very uneven climb lengths, so one warp
//   per voxel left most lanes idle; the pool of climbs keeps every lane on a climb, and the
//   merge per voxel runs on one thread in the reference's order.

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

#include <math_constants.h>

#include "common.cuh"

namespace lar {
namespace {

constexpr int kShMaxLmax = 20;
constexpr int kShDim = kShMaxLmax + 1;
constexpr double kSamePeak = 0.99;  // cpp/src/sh/peaks.cpp:12

struct ShConstants {
    double diagonal[kShDim];             // P(m, m) / sin^m theta, with the Condon-Shortley sign
    double first_up[kShDim];             // P(m + 1, m) = first_up[m] cos P(m, m)
    double rec_a[kShDim][kShDim];        // P(l, m) = rec_a cos P(l-1, m) - rec_b P(l-2, m), l > m + 1
    double rec_b[kShDim][kShDim];
    // With u = sqrt((l - m) (l + m + 1)) and d = sqrt((l + m) (l - m + 1)) of (l, m):
    double half_up[kShDim][kShDim];      // dP/dtheta = half_up P(l, m+1) - half_down P(l, m-1)
    double half_down[kShDim][kShDim];
    double tt_0[kShDim][kShDim];         // d2P/dtheta2 = tt_0 P(l, m) + tt_lo P(l, m-2) + tt_hi P(l, m+2)
    double tt_lo[kShDim][kShDim];
    double tt_hi[kShDim][kShDim];
    double zonal_up[kShDim];             // the same of m = 0: zonal_up P(l, 1); zonal_hi P(l, 2) - zonal_0 P(l, 0)
    double zonal_hi[kShDim];
    double zonal_0[kShDim];
};

__constant__ ShConstants c_sh;

// The factors of cpp/src/sh/harmonics.cpp:29-66 and :102-137, combined per (l, m), in double on the host.
ShConstants host_constants() {
    ShConstants k;
    std::memset(&k, 0, sizeof(k));
    const double pi = 3.14159265358979323846;
    auto up = [](int l, int m) { return std::sqrt(double((l - m) * (l + m + 1))); };
    auto down = [](int l, int m) { return std::sqrt(double((l + m) * (l - m + 1))); };
    auto factor = [](int l, int m) { return std::sqrt((4.0 * l * l - 1.0) / (double(l) * l - double(m) * m)); };
    double ratio = 1.0;
    for (int m = 0; m <= kShMaxLmax; ++m) {
        const double mf = m;
        if (m > 0) ratio *= (2.0 * mf - 1.0) / (2.0 * mf);
        k.diagonal[m] = (m % 2 == 1 ? -1.0 : 1.0) * std::sqrt((2.0 * mf + 1.0) / (4.0 * pi) * ratio);
        k.first_up[m] = std::sqrt(2.0 * mf + 3.0);
        for (int l = m + 2; l <= kShMaxLmax; ++l) {
            k.rec_a[l][m] = factor(l, m);
            k.rec_b[l][m] = factor(l, m) / factor(l - 1, m);
        }
    }
    for (int l = 0; l <= kShMaxLmax; ++l) {
        k.zonal_up[l] = up(l, 0);
        k.zonal_hi[l] = l >= 2 ? up(l, 0) * up(l, 1) / 2.0 : 0.0;
        k.zonal_0[l] = double(l) * (l + 1) / 2.0;
        for (int m = 1; m <= l; ++m) {
            k.half_up[l][m] = up(l, m) / 2.0;
            k.half_down[l][m] = down(l, m) / 2.0;
            // u^2 + d^2 = 2 (l (l + 1) - m^2); for m = 1, P(l, -1) = -P(l, 1) joins it.
            k.tt_0[l][m] = -(2.0 * (double(l) * (l + 1) - double(m) * m) + (m == 1 ? double(l) * (l + 1) : 0.0)) / 4.0;
            k.tt_lo[l][m] = m >= 2 ? down(l, m) * down(l, m - 1) / 4.0 : 0.0;
            k.tt_hi[l][m] = m + 2 <= l ? up(l, m) * up(l, m + 1) / 4.0 : 0.0;
        }
    }
    return k;
}

void ensure_constants() {
    static std::mutex mu;
    static bool ready[64] = {};
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    require(dev >= 0 && dev < 64, "device index out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (ready[dev]) return;
    static const ShConstants k = host_constants();
    cuda_check(cudaMemcpyToSymbol(c_sh, &k, sizeof(k)), "cudaMemcpyToSymbol");
    ready[dev] = true;
}

// The workspaces of the peak search come from a stream-ordered pool of the library's own per
// device that keeps freed memory for the next call (the device's default pool returns it to the
// driver at every synchronisation, and the search synchronises once per call).
cudaMemPool_t workspace_pool() {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    require(dev >= 0 && dev < 64, "device index out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        cuda_check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
        uint64_t keep = ~uint64_t(0);
        cuda_check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute");
        pools[dev] = pool;
    }
    return pools[dev];
}

__host__ __device__ inline int n_coeffs(int lmax, bool full) {
    return full ? (lmax + 1) * (lmax + 1) : (lmax + 1) * (lmax + 2) / 2;
}

__device__ __forceinline__ int coefficient_index(int l, int m, bool full) {
    return full ? l * l + l + m : l * (l + 1) / 2 + m;
}

// A series in global memory, and one in a lane's column of its warp's shared memory.
struct GlobalSeries {
    const double* at;
    __device__ __forceinline__ double operator[](int i) const { return __ldg(at + i); }
};

constexpr int kColumnLd = 33;

struct ColumnSeries {
    const double* at;
    __device__ __forceinline__ double operator[](int i) const { return at[i * kColumnLd]; }
};

struct ShDerivatives {
    double f, t, p, tt, tp, pp;
};

// f, df/dtheta, df/dphi / sin, d2f/dtheta2, d2f/dtheta dphi / sin, d2f/dphi2 / sin^2 given sin and cos of
// theta and phi; the pole limits where sin theta < 1e-4. lmax <= LCAP. The sines and cosines of m phi
// come from those of phi by the angle addition, the powers of sin theta from each other: with the
// trigonometry, the per-order sincos and the divisions the climbs of 500,040 voxels took twice the time
// (11.5 ms against 5.5).
template <int LCAP, typename Coefficients>
__device__ __forceinline__ ShDerivatives sh_derivatives(Coefficients sh, int lmax, bool full,
                                                        double st, double ct, double sp, double cp) {
    const bool pole = st < 1e-4;
    double sm[LCAP + 1], cm[LCAP + 1];
    sm[1] = sp;
    cm[1] = cp;
#pragma unroll
    for (int m = 2; m <= LCAP; ++m) {
        cm[m] = cm[m - 1] * cp - sm[m - 1] * sp;
        sm[m] = sm[m - 1] * cp + cm[m - 1] * sp;
    }
    double p2[LCAP + 1], p1[LCAP + 1], p0[LCAP + 1], power = 1.0;
    ShDerivatives z{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, r = z;  // the orders 0, and the others without their sqrt(2)
#pragma unroll
    for (int l = 0; l <= LCAP; ++l) {
        if (l > lmax) break;
        // Row l of the Legendre table (cpp/src/sh/harmonics.cpp:70-88).
#pragma unroll
        for (int m = 0; m <= l; ++m) {
            if (m == l)
                p0[m] = c_sh.diagonal[m] * power;
            else if (m == l - 1)
                p0[m] = c_sh.first_up[m] * ct * p1[m];
            else
                p0[m] = c_sh.rec_a[l][m] * ct * p1[m] - c_sh.rec_b[l][m] * p2[m];
        }
        power *= st;
        if (full || l % 2 == 0) {
            // The terms of degree l (cpp/src/sh/harmonics.cpp:102-137, 150-186).
            const double zonal = sh[coefficient_index(l, 0, full)];
            z.f = fma(zonal, p0[0], z.f);
            if (l > 0) {
                z.t = fma(zonal, c_sh.zonal_up[l] * p0[1], z.t);
                z.tt = fma(zonal, (l >= 2 ? c_sh.zonal_hi[l] * p0[l >= 2 ? 2 : 0] : 0.0) - c_sh.zonal_0[l] * p0[0], z.tt);
            }
#pragma unroll
            for (int m = 1; m <= l; ++m) {
                const double mf = m;
                const double cc = sh[coefficient_index(l, m, full)];
                const double sc = sh[coefficient_index(l, -m, full)];
                const double ang = cc * cm[m] + sc * sm[m];
                const double ang_p = sc * cm[m] - cc * sm[m];
                const double pv = p0[m];
                const double pt = (m < l ? c_sh.half_up[l][m] * p0[m < l ? m + 1 : m] : 0.0) -
                                  c_sh.half_down[l][m] * p0[m - 1];
                double ptt = c_sh.tt_0[l][m] * pv;
                if (m >= 2) ptt = fma(c_sh.tt_lo[l][m], p0[m >= 2 ? m - 2 : 0], ptt);
                if (m + 2 <= l) ptt = fma(c_sh.tt_hi[l][m], p0[m + 2 <= l ? m + 2 : m], ptt);
                r.f = fma(ang, pv, r.f);
                r.t = fma(ang, pt, r.t);
                r.tt = fma(ang, ptt, r.tt);
                const double mp = mf * pv;
                r.p = fma(ang_p, pole ? pt : mp, r.p);
                r.tp = fma(ang_p, mf * pt, r.tp);
                r.pp = fma(-ang, mf * mp, r.pp);
            }
        }
#pragma unroll
        for (int m = 0; m <= l; ++m) {
            p2[m] = p1[m];
            p1[m] = p0[m];
        }
    }
    constexpr double kRoot2 = 1.41421356237309504880;
    r.f = fma(kRoot2, r.f, z.f);
    r.t = fma(kRoot2, r.t, z.t);
    r.tt = fma(kRoot2, r.tt, z.tt);
    if (pole) {
        r.p *= kRoot2;
        r.tp = r.pp = 0.0;
    } else {
        const double inv = 1.0 / st;
        r.p *= kRoot2 * inv;
        r.tp *= kRoot2 * inv;
        r.pp *= kRoot2 * inv * inv;
    }
    return r;
}

// One step of the Newton climb of cpp/src/sh/peaks.cpp:36-72 from the unit vector (x, y, z):
// moves it along the gradient by the capped Newton step and renormalises it; returns the step
// and, in *f, the amplitude before it. The sines and cosines of acos(z) and atan2(y, x) are algebraic in
// the vector.
template <int LCAP, typename Coefficients>
__device__ __forceinline__ double climb_step(Coefficients sh, int lmax, bool full, double& x, double& y, double& z,
                                             double max_step, double* f) {
    const double ct = z < -1.0 ? -1.0 : (1.0 < z ? 1.0 : z);  // std::clamp
    const double st = sqrt((1.0 - ct) * (1.0 + ct));
    double xs = x, ys = y, rho2 = x * x + y * y;
    if (!(rho2 > 1e-280 && rho2 < 1e280)) {  // squares out of range: scaled first
        const double m = fmax(fabs(x), fabs(y));
        xs = m > 0.0 ? x / m : copysign(1.0, x);  // on the axis, atan2's 0 or pi by the sign of x
        ys = m > 0.0 ? y / m : y;
        rho2 = xs * xs + ys * ys;
    }
    const double rho_inv = 1.0 / sqrt(rho2), cp = xs * rho_inv, sp = ys * rho_inv;
    const ShDerivatives h = sh_derivatives<LCAP>(sh, lmax, full, st, ct, sp, cp);
    const double gnorm = sqrt(h.t * h.t + h.p * h.p);
    double at = 0.0, ap = 0.0;
    if (gnorm != 0.0) {
        const double inv = 1.0 / gnorm;
        at = h.t * inv;
        ap = h.p * inv;
    }
    const double slope = at * h.t + ap * h.p;
    const double curv = at * at * h.tt + 2.0 * at * ap * h.tp + ap * ap * h.pp;
    double step = curv != 0.0 ? fabs(slope / curv) : 0.0;
    step = fmin(step, max_step);
    x += step * (at * (ct * cp) + ap * (-sp));
    y += step * (at * (ct * sp) + ap * cp);
    z += step * (at * (-st) + ap * 0.0);
    const double inv = 1.0 / sqrt(x * x + y * y + z * z);
    x *= inv;
    y *= inv;
    z *= inv;
    *f = h.f;
    return step;
}

// The Newton climb of cpp/src/sh/peaks.cpp:31-78: true with the direction after the first step
// shorter than tol and the amplitude before it; false after max_iters steps.
template <int LCAP>
__device__ bool climb(const double* __restrict__ sh, int lmax, bool full, double x, double y, double z, int max_iters,
                      double tol, double max_step, double* out, double* amp) {
    for (int it = 0; it < max_iters; ++it) {
        double f;
        if (climb_step<LCAP>(GlobalSeries{sh}, lmax, full, x, y, z, max_step, &f) < tol) {
            out[0] = x;
            out[1] = y;
            out[2] = z;
            *amp = f;
            return true;
        }
    }
    return false;
}

template <int LCAP>
__global__ void __launch_bounds__(128) sh_derivatives_kernel(const double* __restrict__ coeffs, int64_t n, int64_t ldc,
                                                             int lmax, int full, const double* __restrict__ theta,
                                                             const double* __restrict__ phi, double* __restrict__ out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // Legendre::at_elevation takes cos and sin of theta (cpp/src/sh/harmonics.cpp:92-94).
    double st, ct, sp, cp;
    sincos(theta[i], &st, &ct);
    sincos(phi[i], &sp, &cp);
    const ShDerivatives r = sh_derivatives<LCAP>(GlobalSeries{coeffs + i * ldc}, lmax, full != 0, st, ct, sp, cp);
    double* o = out + i * 6;
    o[0] = r.f;
    o[1] = r.t;
    o[2] = r.p;
    o[3] = r.tt;
    o[4] = r.tp;
    o[5] = r.pp;
}

template <int LCAP>
__global__ void __launch_bounds__(128) climb_kernel(const double* __restrict__ coeffs, int64_t n, int64_t ldc, int lmax,
                                                    int full, const double* __restrict__ starts, int max_iters,
                                                    double tol, double max_step, double* __restrict__ dirs,
                                                    double* __restrict__ amps) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d[3], a;
    if (!climb<LCAP>(coeffs + i * ldc, lmax, full != 0, starts[3 * i], starts[3 * i + 1], starts[3 * i + 2],
                     max_iters, tol, max_step, d, &a)) {
        d[0] = d[1] = d[2] = a = CUDART_NAN;
    }
    dirs[3 * i] = d[0];
    dirs[3 * i + 1] = d[1];
    dirs[3 * i + 2] = d[2];
    amps[i] = a;
}

// ---- the peak search in passes ------------------------------------------------------------
//
// (1) peak_count_kernel: per voxel its local maxima with a positive amplitude, as a bit per vertex, and
//     their number (0 when nv is 0 or the first amplitude is not finite: cpp/src/sh/peaks.cpp:87-89);
// (2) scan_blocks_kernel + scan_sums_kernel: their exclusive prefix sums, the offsets of the
//     voxels' climbs in one list, and the total;
// (3) peak_fill_kernel: the starts (voxel, vertex) at those offsets, in vertex order, one for two opposite
//     maxima of an even series;
// (4) climb_pool_kernel: every climb of the list, one Newton step per pass of a lane, a lane
//     whose climb ends taking the next from a device counter, so the lanes stay busy however
//     uneven the climbs' lengths and the voxels' start counts are;
// (5) peak_merge_kernel: per voxel its climbs merged in start order into a found list kept in
//     place at the front of its span (cpp/src/sh/peaks.cpp:94-116), then the n_peaks largest,
//     ties to the earlier entry (a stable sort), above both thresholds (:118-132).

constexpr int kScanItems = 4;
constexpr int kScanBlock = 1024;
constexpr int kScanSpan = kScanItems * kScanBlock;  // voxels per scan block

__device__ __forceinline__ bool local_max(const double* __restrict__ amp, const int* __restrict__ nb, int v) {
    const double here = amp[v];
    bool is_max = here > 0.0;
    for (int j = 0; j < 6 && is_max; ++j) is_max = amp[nb[6 * v + j]] <= here;
    return is_max;
}

// Whether local maximum v is left to its opposite vertex, which comes first (antipodes is NULL for a series
// with odd degrees). Every term of an even series' climb from -v is that from v, or its negative,
// exactly, so both end at opposite vectors with the same amplitude and the merge drops the second: one
// climb serves both, unless it meets a pole, where the terms' limits are not symmetric (climb_pool_kernel).
__device__ __forceinline__ bool left_to_antipode(const unsigned* mask, const int* __restrict__ antipodes, int v) {
    if (antipodes == nullptr) return false;
    const int a = antipodes[v];
    return a >= 0 && a < v && (mask[a >> 5] >> (a & 31) & 1u);
}

// The climbs of word w: its bits without those.
__device__ __forceinline__ unsigned climbs_of(const unsigned* mask, int w, const int* __restrict__ antipodes) {
    unsigned kept = mask[w];
    for (unsigned b = antipodes != nullptr ? kept : 0u; b; b &= b - 1u) {
        const int bit = __ffs(b) - 1;
        if (left_to_antipode(mask, antipodes, 32 * w + bit)) kept &= ~(1u << bit);
    }
    return kept;
}

// A warp per voxel, for spheres whose tile does not fit.
__global__ void __launch_bounds__(128) peak_count_kernel(const double* __restrict__ on_sphere, int64_t n, int64_t lds,
                                                         const int* __restrict__ neighbours,
                                                         const int* __restrict__ antipodes, int nv,
                                                         int* __restrict__ counts, unsigned* __restrict__ masks) {
    const int lane = threadIdx.x & 31;
    const int64_t voxel = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (voxel >= n) return;
    const double* amp = on_sphere + voxel * lds;
    const int words = (nv + 31) / 32;
    unsigned* mask = masks + voxel * words;
    int count = 0;
    if (nv > 0 && isfinite(amp[0])) {
        for (int w = 0; w < words; ++w) {
            const int v = 32 * w + lane;
            const unsigned b = __ballot_sync(0xffffffffu, v < nv && local_max(amp, neighbours, v));
            if (lane == 0) mask[w] = b;
        }
        __syncwarp();
        for (int w = lane; w < words; w += 32) count += __popc(climbs_of(mask, w, antipodes));
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0) counts[voxel] = count;
}

// The same with the amplitudes of 16 voxels in shared memory, a vertex to a row: a lane compares its own
// voxel's, so that the gathers of a half warp are 16 consecutive doubles. The gathers bound it: read through
// the L1 in vertex order, a warp's 32 lie on nearly as many lines (500,040 voxels on 642 vertices: 1.45 ms
// against 1.88; the amplitudes' bytes alone take 0.39).
constexpr int kTileVoxels = 16;
constexpr int kTileLd = kTileVoxels + 1;
constexpr int kTileThreads = 256;

__global__ void __launch_bounds__(kTileThreads) peak_count_tile_kernel(const double* __restrict__ on_sphere,
                                                                      int64_t n, int64_t lds,
                                                                      const int* __restrict__ neighbours,
                                                                      const int* __restrict__ antipodes, int nv,
                                                                      int* __restrict__ counts,
                                                                      unsigned* __restrict__ masks) {
    extern __shared__ __align__(16) double tile[];  // (nv, kTileLd), then the masks (kTileVoxels, words)
    __shared__ int count[kTileVoxels];
    const int words = (nv + 31) / 32;
    auto* mask = reinterpret_cast<unsigned*>(tile + size_t(nv) * kTileLd);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t v0 = int64_t(blockIdx.x) * kTileVoxels;
    const int here = int(min(int64_t(kTileVoxels), n - v0));
    for (int row = warp; row < here; row += kTileThreads / 32) {
        const double* amp = on_sphere + (v0 + row) * lds;
        for (int v = lane; v < nv; v += 32) {
            const unsigned to = unsigned(__cvta_generic_to_shared(tile + size_t(v) * kTileLd + row));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(amp + v) : "memory");
        }
    }
    if (threadIdx.x < kTileVoxels) count[threadIdx.x] = 0;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int voxel = lane & 15, half = lane >> 4;
    const double* mine = tile + voxel;
    const bool live = voxel < here && isfinite(mine[0]);
    for (int w = warp; w < words; w += kTileThreads / 32) {
        unsigned bits = 0;
        const int first = 32 * w + 16 * half;
#pragma unroll 4
        for (int k = 0; k < 16; ++k) {
            const int v = min(first + k, nv - 1);
            const int2* nb = reinterpret_cast<const int2*>(neighbours + 6 * size_t(v));
            const int2 n0 = __ldg(nb), n1 = __ldg(nb + 1), n2 = __ldg(nb + 2);
            const double amp = mine[v * kTileLd];
            // All seven at once: a chain of early exits waits for each gather in turn.
            const bool is_max = (amp > 0.0) & (mine[n0.x * kTileLd] <= amp) & (mine[n0.y * kTileLd] <= amp) &
                                (mine[n1.x * kTileLd] <= amp) & (mine[n1.y * kTileLd] <= amp) &
                                (mine[n2.x * kTileLd] <= amp) & (mine[n2.y * kTileLd] <= amp) & (first + k < nv);
            if (is_max) bits |= 1u << (16 * half + k);
        }
        bits |= __shfl_xor_sync(0xffffffffu, bits, 16);
        if (half == 0) mask[voxel * words + w] = live ? bits : 0u;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < here * words; e += kTileThreads) {
        const int row = e / words, w = e % words;
        const unsigned kept = climbs_of(mask + row * words, w, antipodes);
        masks[v0 * words + e] = mask[e];
        if (kept) atomicAdd(count + row, __popc(kept));
    }
    __syncthreads();
    if (threadIdx.x < here) counts[v0 + threadIdx.x] = count[threadIdx.x];
}

size_t tile_bytes(int64_t nv) {
    return size_t(nv) * kTileLd * sizeof(double) + size_t(kTileVoxels) * size_t((nv + 31) / 32) * sizeof(unsigned);
}

// Two tiles in an SM's shared memory, or the warps are too few to hide the gathers.
bool tile_fits(int64_t nv) { return nv > 0 && nv <= 4096 && tile_bytes(nv) <= 110 * 1024; }

// Exclusive prefix sums of counts within blocks of kScanSpan voxels, and each block's sum.
__global__ void __launch_bounds__(kScanBlock) scan_blocks_kernel(const int* __restrict__ counts, int64_t n,
                                                                 int64_t* __restrict__ offsets,
                                                                 int64_t* __restrict__ block_sums) {
    __shared__ int64_t warp_sums[kScanBlock / 32];
    const int64_t first = int64_t(blockIdx.x) * kScanSpan + int64_t(threadIdx.x) * kScanItems;
    int64_t local[kScanItems];
    int64_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        local[k] = sum;
        sum += first + k < n ? counts[first + k] : 0;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    if (w == 0) {
        int64_t ws = warp_sums[lane];
        int64_t wi = ws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t up = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += up;
        }
        warp_sums[lane] = wi - ws;
        if (lane == 31) block_sums[blockIdx.x] = wi;
    }
    __syncthreads();
    const int64_t before = warp_sums[w] + incl - sum;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (first + k < n) offsets[first + k] = before + local[k];
}

// The blocks' sums to exclusive block offsets, in place, and the total; one block.
__global__ void __launch_bounds__(kScanBlock) scan_sums_kernel(int64_t* __restrict__ block_sums, int64_t blocks,
                                                               int64_t* __restrict__ total) {
    __shared__ int64_t warp_sums[kScanBlock / 32];
    __shared__ int64_t carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int64_t b0 = 0; b0 < blocks; b0 += kScanBlock) {
        const int64_t b = b0 + threadIdx.x;
        const int64_t x = b < blocks ? block_sums[b] : 0;
        int64_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) warp_sums[w] = incl;
        __syncthreads();
        if (w == 0) {
            const int64_t ws = warp_sums[lane];
            int64_t wi = ws;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t up = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += up;
            }
            warp_sums[lane] = wi - ws;
        }
        __syncthreads();
        const int64_t base = carry;
        if (b < blocks) block_sums[b] = base + warp_sums[w] + incl - x;
        __syncthreads();
        if (threadIdx.x == kScanBlock - 1) carry = base + warp_sums[w] + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__device__ __forceinline__ int64_t climb_offset(const int64_t* __restrict__ offsets,
                                                const int64_t* __restrict__ block_offsets, int64_t voxel) {
    return offsets[voxel] + block_offsets[voxel / kScanSpan];
}

// The starts from the masks of pass (1), a thread per voxel: (voxel, vertex), or (voxel, ~vertex) where
// the climb stands for the opposite vertex's too.
__global__ void __launch_bounds__(128) peak_fill_kernel(const int* __restrict__ counts,
                                                        const unsigned* __restrict__ masks, int64_t n, int words,
                                                        const int* __restrict__ antipodes,
                                                        const int64_t* __restrict__ offsets,
                                                        const int64_t* __restrict__ block_offsets,
                                                        int2* __restrict__ starts) {
    const int64_t voxel = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (voxel >= n || counts[voxel] == 0) return;  // (the mask of a voxel without maxima may be unwritten)
    int64_t at = climb_offset(offsets, block_offsets, voxel);
    const unsigned* mine = masks + voxel * words;
    for (int w = 0; w < words; ++w)
        for (unsigned b = climbs_of(mine, w, antipodes); b; b &= b - 1u) {
            const int v = 32 * w + __ffs(b) - 1, a = antipodes != nullptr ? antipodes[v] : -1;
            const bool both = a > v && (mine[a >> 5] >> (a & 31) & 1u);
            starts[at++] = make_int2(int(voxel), both ? ~v : v);
        }
}

// Every climb of the list (cpp/src/sh/peaks.cpp:31-78 with the search's settings: 50 steps,
// tolerance 1e-4, steps of at most 0.2): results (total, 4) = the direction and the amplitude,
// the amplitude NaN when the climb has not stopped.
//
// STAGED holds each lane's series in a column of its warp's shared memory, filled when the lane takes a
// climb: every lane reads another voxel's series, so each of a step's 45 loads went to up to 32 lines
// (500,040 voxels: 2.75 ms against 3.21; 5.5 before one climb served both of two opposite maxima). What
// bounds it then: the instructions issued (55% of the slots, 42% of the FP64 pipe's).
// It takes series of up to kStagedDim coefficients (even, to degree 8), four CTAs' columns in an SM.
constexpr int kStagedDim = 45;

template <int LCAP, bool STAGED>
__global__ void __launch_bounds__(128, 4) climb_pool_kernel(const double* __restrict__ coeffs, int64_t ldc, int lmax,
                                                            int full, const double* __restrict__ vertices,
                                                            const int* __restrict__ antipodes,
                                                            const int2* __restrict__ starts, int64_t total,
                                                            double4* __restrict__ results,
                                                            unsigned long long* __restrict__ next) {
    extern __shared__ __align__(16) double columns[];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const bool is_full = full != 0;
    int64_t k = -1;
    int it = 0, opposite = -1;
    bool at_pole = false, second = false;
    double x = 0.0, y = 0.0, z = 0.0;
    const double* sh = coeffs;
    const int dim = n_coeffs(lmax, is_full);
    double* column = columns + (threadIdx.x >> 5) * (kStagedDim * kColumnLd) + lane;
    bool exhausted = false;
    for (;;) {
        // Lanes without a climb take the next ones, one atomic per warp.
        const unsigned want = __ballot_sync(0xffffffffu, k < 0 && !exhausted);
        if (want) {
            unsigned long long base = 0;
            bool taken = false;
            const int leader = __ffs(want) - 1;
            if (lane == leader) base = atomicAdd(next, (unsigned long long)__popc(want));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (base + __popc(want) >= (unsigned long long)total) exhausted = true;
            if (k < 0) {
                const unsigned long long mine = base + __popc(want & below);
                if (mine < (unsigned long long)total) {
                    k = int64_t(mine);
                    const int2 s = starts[k];
                    const int v = s.y < 0 ? ~s.y : s.y;
                    opposite = s.y < 0 ? antipodes[v] : -1;
                    k *= is_full ? 1 : 2;
                    second = false;
                    at_pole = false;
                    x = vertices[3 * v];
                    y = vertices[3 * v + 1];
                    z = vertices[3 * v + 2];
                    sh = coeffs + int64_t(s.x) * ldc;
                    it = 0;
                    taken = true;
                }
            }
            if constexpr (STAGED) {
                __syncwarp();  // the columns' last readings are done
                for (unsigned b = __ballot_sync(0xffffffffu, taken); b; b &= b - 1u) {
                    const int to = __ffs(b) - 1;
                    const double* from = reinterpret_cast<const double*>(
                        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(sh), to));
                    for (int i = lane; i < dim; i += 32) {
                        const unsigned at = unsigned(__cvta_generic_to_shared(column + i * kColumnLd + to - lane));
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(at), "l"(from + i) : "memory");
                    }
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
            }
        }
        if (!__any_sync(0xffffffffu, k >= 0)) break;
        if (k >= 0) {
            double f, step;
            at_pole = at_pole || (1.0 - z) * (1.0 + z) < 1.1e-8;  // sin theta < 1e-4, with room for rounding
            if constexpr (STAGED)
                step = climb_step<LCAP>(ColumnSeries{column}, lmax, is_full, x, y, z, 0.2, &f);
            else
                step = climb_step<LCAP>(GlobalSeries{sh}, lmax, is_full, x, y, z, 0.2, &f);
            const bool found = step < 1e-4;
            if (found || ++it >= 50) {
                results[k + second] = found ? make_double4(x, y, z, f)
                                            : make_double4(CUDART_NAN, CUDART_NAN, CUDART_NAN, CUDART_NAN);
                if (at_pole && opposite >= 0) {
                    x = vertices[3 * opposite];
                    y = vertices[3 * opposite + 1];
                    z = vertices[3 * opposite + 2];
                    opposite = -1;
                    second = true;
                    it = 0;
                } else {
                    if (!is_full && !second) results[k + 1].w = CUDART_NAN;
                    k = -1;
                }
            }
        }
    }
}

__global__ void __launch_bounds__(128) peak_merge_kernel(int64_t n, int full, const int* __restrict__ counts,
                                                         const int64_t* __restrict__ offsets,
                                                         const int64_t* __restrict__ block_offsets,
                                                         double4* __restrict__ results, int n_peaks, double rel,
                                                         double thr, double* __restrict__ dirs,
                                                         double* __restrict__ amps) {
    const int64_t voxel = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (voxel >= n) return;
    double* dv = dirs + voxel * int64_t(n_peaks) * 3;
    double* av = amps + voxel * int64_t(n_peaks);
    for (int k = 0; k < 3 * n_peaks; ++k) dv[k] = CUDART_NAN;
    for (int k = 0; k < n_peaks; ++k) av[k] = CUDART_NAN;
    const int count = counts[voxel];
    if (count == 0) return;
    const bool is_full = full != 0;
    const int slots = is_full ? 1 : 2;  // an even series' climb, and its opposite's where a pole asked for it
    double4* found = results + slots * climb_offset(offsets, block_offsets, voxel);
    int n_found = 0;
    for (int i = 0; i < slots * count; ++i) {
        const double4 c = found[i];
        // Written so that a NaN amplitude is dropped too.
        if (!(c.w > 0.0)) continue;
        int match = -1;
        for (int j = 0; j < n_found; ++j) {
            const double4 o = found[j];
            const double cosine = c.x * o.x + c.y * o.y + c.z * o.z;
            if ((is_full ? cosine : fabs(cosine)) > kSamePeak) {
                match = j;
                break;
            }
        }
        // The found list occupies entries [0, n_found), n_found <= i: entry i is read already.
        if (match < 0)
            found[n_found++] = c;
        else if (c.w > found[match].w)
            found[match] = c;
    }
    if (n_found == 0) return;
    double largest = 0.0;
    const int kept = min(n_peaks, n_found);
    for (int r = 0; r < kept; ++r) {
        int bi = 0;
        double best = -CUDART_INF;
        for (int j = 0; j < n_found; ++j)
            if (found[j].w > best) {
                best = found[j].w;
                bi = j;
            }
        if (r == 0) largest = best;
        if (best < thr || best < rel * largest) break;
        const double4 c = found[bi];
        const bool flip = !is_full && c.z < 0.0;
        dv[3 * r] = flip ? -c.x : c.x;
        dv[3 * r + 1] = flip ? -c.y : c.y;
        dv[3 * r + 2] = flip ? -c.z : c.z;
        av[r] = best;
        found[bi].w = -CUDART_INF;  // taken
    }
}

int lcap_for(int lmax) { return lmax <= 8 ? 8 : (lmax <= 12 ? 12 : 20); }

void check_lmax(int lmax, bool full, int64_t ldc) {
    require(lmax >= 0 && lmax <= kShMaxLmax && (full || lmax % 2 == 0),
            "lmax must be at most 20, and even unless full, got " + std::to_string(lmax));
    require(ldc >= n_coeffs(lmax, full), "ldc must be at least the series' coefficient count");
}

}  // namespace
}  // namespace lar

// A sphere for the peak search: unit vertices and the 6 neighbours of each, on the device.
struct lar_peak_sphere_s {
    int64_t nv = 0;
    lar::DeviceArray<double> vertices;  // (nv, 3)
    lar::DeviceArray<int> neighbours;   // (nv, 6)
    lar::DeviceArray<int> antipodes;    // (nv): the vertex exactly opposite, or -1
};

using namespace lar;

extern "C" {

int lar_peak_sphere_create(const double* vertices, const int64_t* neighbours, int64_t nv, lar_peak_sphere* out) {
    return guarded([&] {
        require(out != nullptr, "out must not be NULL");
        require(nv >= 0 && nv < (int64_t(1) << 31), "nv must be between 0 and 2^31 - 1");
        require(nv == 0 || (vertices != nullptr && neighbours != nullptr), "vertices and neighbours must not be NULL");
        std::vector<int> nb(size_t(nv) * 6);
        for (int64_t k = 0; k < nv * 6; ++k) {
            require(neighbours[k] >= 0 && neighbours[k] < nv, "a neighbour index is outside the sphere");
            nb[size_t(k)] = int(neighbours[k]);
        }
        auto h = std::make_unique<lar_peak_sphere_s>();
        h->nv = nv;
        h->vertices.upload(vertices, size_t(nv) * 3);
        h->neighbours.upload(nb.data(), nb.size());
        // By each vertex's first appearance; + 0.0 so that -0 and 0 are one.
        using Vertex = std::array<double, 3>;
        std::vector<std::pair<Vertex, int>> sorted(static_cast<size_t>(nv));
        for (int64_t k = 0; k < nv; ++k)
            sorted[size_t(k)] = {{vertices[3 * k] + 0.0, vertices[3 * k + 1] + 0.0, vertices[3 * k + 2] + 0.0}, int(k)};
        // A vertex with a NaN has no place in the order: then none has an opposite.
        bool ordered = true;
        for (const auto& s : sorted) ordered = ordered && s.first[0] == s.first[0] && s.first[1] == s.first[1] && s.first[2] == s.first[2];
        std::vector<int> antipodes(size_t(nv), -1);
        if (ordered) {
            std::sort(sorted.begin(), sorted.end());
            for (int64_t k = 0; k < nv; ++k) {
                const Vertex opposite{-vertices[3 * k] + 0.0, -vertices[3 * k + 1] + 0.0, -vertices[3 * k + 2] + 0.0};
                const auto at = std::lower_bound(sorted.begin(), sorted.end(), std::make_pair(opposite, -1));
                if (at != sorted.end() && at->first == opposite) antipodes[size_t(k)] = at->second;
            }
        }
        h->antipodes.upload(antipodes.data(), antipodes.size());
        *out = h.release();
    });
}

void lar_peak_sphere_destroy(lar_peak_sphere sphere) { delete sphere; }

int lar_sh_derivatives(const double* coeffs, int64_t n, int64_t ldc, int lmax, int full, const double* theta,
                       const double* phi, double* out, void* stream) {
    return guarded([&] {
        check_lmax(lmax, full != 0, ldc);
        require(n >= 0, "n must be at least 0");
        if (n == 0) return;
        ensure_constants();
        auto st = static_cast<cudaStream_t>(stream);
        const unsigned blocks = unsigned((n + 127) / 128);
        LaunchScope scope("sh_derivatives_kernel", st);
        switch (lcap_for(lmax)) {
            case 8: sh_derivatives_kernel<8><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, theta, phi, out); break;
            case 12: sh_derivatives_kernel<12><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, theta, phi, out); break;
            default: sh_derivatives_kernel<20><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, theta, phi, out);
        }
        cuda_check(cudaGetLastError(), "sh_derivatives_kernel launch");
    });
}

int lar_climb(const double* coeffs, int64_t n, int64_t ldc, int lmax, int full, const double* starts, int max_iters,
              double tol, double max_step, double* directions, double* amplitudes, void* stream) {
    return guarded([&] {
        check_lmax(lmax, full != 0, ldc);
        require(n >= 0, "n must be at least 0");
        require(max_iters >= 0, "max_iters must be at least 0");
        if (n == 0) return;
        ensure_constants();
        auto st = static_cast<cudaStream_t>(stream);
        const unsigned blocks = unsigned((n + 127) / 128);
        LaunchScope scope("climb_kernel", st);
        switch (lcap_for(lmax)) {
            case 8:
                climb_kernel<8><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, starts, max_iters, tol, max_step,
                                                        directions, amplitudes);
                break;
            case 12:
                climb_kernel<12><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, starts, max_iters, tol, max_step,
                                                         directions, amplitudes);
                break;
            default:
                climb_kernel<20><<<blocks, 128, 0, st>>>(coeffs, n, ldc, lmax, full, starts, max_iters, tol, max_step,
                                                         directions, amplitudes);
        }
        cuda_check(cudaGetLastError(), "climb_kernel launch");
    });
}

int lar_find_peaks(lar_peak_sphere sphere, const double* coeffs, int64_t n, int64_t ldc, int lmax, int full,
                   const double* on_sphere, int64_t lds, int n_peaks, double relative_threshold, double threshold,
                   double* directions, double* amplitudes, void* stream) {
    return guarded([&] {
        require(sphere != nullptr, "sphere must not be NULL");
        check_lmax(lmax, full != 0, ldc);
        require(n >= 0, "n must be at least 0");
        require(n_peaks >= 1, "n_peaks must be at least 1");
        require(lds >= sphere->nv, "lds must be at least the sphere's vertex count");
        require(n < (int64_t(1) << 31), "n must be below 2^31");
        if (n == 0) return;
        ensure_constants();
        auto st = static_cast<cudaStream_t>(stream);
        const int nv = int(sphere->nv);
        const int64_t scan_blocks = (n + kScanSpan - 1) / kScanSpan;
        // Workspace: counts (n), masks (n, words), offsets (n), block offsets, the total and the climbs'
        // counter.
        const int words = (nv + 31) / 32;
        const size_t ws_bytes = size_t(n) * (1 + size_t(words)) * sizeof(int) + (size_t(n) + size_t(scan_blocks) + 2) * sizeof(int64_t) + 64;
        char* ws = nullptr;
        cudaMemPool_t pool = workspace_pool();
        cuda_check(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), ws_bytes, pool, st), "cudaMallocFromPoolAsync");
        auto* offsets = reinterpret_cast<int64_t*>(ws);
        auto* block_offsets = offsets + n;
        auto* total_dev = block_offsets + scan_blocks;
        auto* next = reinterpret_cast<unsigned long long*>(total_dev + 1);
        int* counts = reinterpret_cast<int*>(next + 1);
        auto* masks = reinterpret_cast<unsigned*>(counts + n);
        const unsigned warp_blocks = unsigned((n * 32 + 127) / 128);
        const int* antipodes = full ? nullptr : sphere->antipodes.ptr;
        {
            LaunchScope scope("peak_count_kernel", st);
            if (tile_fits(nv)) {
                const size_t smem = tile_bytes(nv);
                allow_smem(peak_count_tile_kernel, smem);
                peak_count_tile_kernel<<<unsigned((n + kTileVoxels - 1) / kTileVoxels), kTileThreads, smem, st>>>(
                    on_sphere, n, lds, sphere->neighbours.ptr, antipodes, nv, counts, masks);
            } else {
                peak_count_kernel<<<warp_blocks, 128, 0, st>>>(on_sphere, n, lds, sphere->neighbours.ptr, antipodes,
                                                               nv, counts, masks);
            }
            cuda_check(cudaGetLastError(), "peak_count_kernel launch");
        }
        {
            LaunchScope scope("scan_blocks_kernel", st);
            scan_blocks_kernel<<<unsigned(scan_blocks), kScanBlock, 0, st>>>(counts, n, offsets, block_offsets);
            cuda_check(cudaGetLastError(), "scan_blocks_kernel launch");
        }
        {
            LaunchScope scope("scan_sums_kernel", st);
            scan_sums_kernel<<<1, kScanBlock, 0, st>>>(block_offsets, scan_blocks, total_dev);
            cuda_check(cudaGetLastError(), "scan_sums_kernel launch");
        }
        // The climb list's length sizes its buffers: the one wait of the call.
        int64_t total = 0;
        cuda_check(cudaMemcpyAsync(&total, total_dev, sizeof(total), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
        cuda_check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
        char* lists = nullptr;
        if (total > 0) {
            cuda_check(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&lists),
                                               size_t(total) * (sizeof(int2) + (full ? 1 : 2) * sizeof(double4)), pool, st),
                       "cudaMallocFromPoolAsync");
            auto* results = reinterpret_cast<double4*>(lists);
            auto* starts = reinterpret_cast<int2*>(results + (full ? 1 : 2) * total);
            {
                LaunchScope scope("peak_fill_kernel", st);
                peak_fill_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(counts, masks, n, words, antipodes,
                                                                            offsets, block_offsets, starts);
                cuda_check(cudaGetLastError(), "peak_fill_kernel launch");
            }
            cuda_check(cudaMemsetAsync(next, 0, sizeof(*next), st), "cudaMemsetAsync");
            const int lcap = lcap_for(lmax);
            const bool staged = n_coeffs(lmax, full != 0) <= kStagedDim;
            auto climber = staged ? climb_pool_kernel<8, true>
                                  : (lcap == 8 ? climb_pool_kernel<8, false>
                                               : (lcap == 12 ? climb_pool_kernel<12, false> : climb_pool_kernel<20, false>));
            const size_t smem = staged ? size_t(4 * kStagedDim * kColumnLd) * sizeof(double) : 0;
            if (staged)
                allow_smem(climber, smem);
            int per_sm = 0;
            cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, climber, 128, smem),
                       "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
            const int64_t pool_blocks = std::max<int64_t>(
                1, std::min<int64_t>((total + 127) / 128, int64_t(sm_count()) * ctas_per_sm(per_sm, "peaks.ctas_per_sm")));
            {
                LaunchScope scope("climb_pool_kernel", st);
                climber<<<unsigned(pool_blocks), 128, smem, st>>>(coeffs, ldc, lmax, full, sphere->vertices.ptr, antipodes,
                                                               starts, total, results, next);
                cuda_check(cudaGetLastError(), "climb_pool_kernel launch");
            }
        }
        {
            LaunchScope scope("peak_merge_kernel", st);
            peak_merge_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(
                n, full, counts, offsets, block_offsets, reinterpret_cast<double4*>(lists), n_peaks, relative_threshold,
                threshold, directions, amplitudes);
            cuda_check(cudaGetLastError(), "peak_merge_kernel launch");
        }
        if (lists) cuda_check(cudaFreeAsync(lists, st), "cudaFreeAsync");
        cuda_check(cudaFreeAsync(ws, st), "cudaFreeAsync");
    });
}

}  // extern "C"
