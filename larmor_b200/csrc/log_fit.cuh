// Device view of a prepared log-signal design (see log_fit.cu).
#pragma once

#include <cstdint>

#include "common.cuh"

namespace lar {

template <class T>
struct LogDesignDevice {
    int n = 0, p = 0, m = 0;
    const T* x = nullptr;          // (n, p) unit-norm columns
    const T* pinvt = nullptr;      // (n, p) transposed pseudo-inverse
    const T* g = nullptr;          // (m, p) constraints, column-scaled
    const T* gt = nullptr;         // (p, m) the same, transposed (lanes over constraints read it coalesced)
    const T* scales = nullptr;     // (p,) column norms
    const double* scales64 = nullptr;  // (p,) column norms in double, for the outputs
    // The constraints have DKI's form (dki_constraint_bound): rows D, V and bound D - V.
    bool dki = false;
    T bound = T(0);
};

// Whether the constraints g (m, p; host, row-major) have the form DKI's have: 256 rows D on columns
// 1..6, 256 rows V on columns 7..21 and 256 rows b D - V (to rounding), b in *bound.
constexpr int kDkiDirs = 256, kDkiP = 22, kDkiD = 6, kDkiV = 15;
inline bool dki_constraint_bound(const double* g, int64_t m, int64_t p, double* bound) {
    if (p != kDkiP || m != 3 * kDkiDirs) return false;
    double b = 0.0;
    for (int64_t i = 0; i < kDkiDirs && b == 0.0; ++i)
        for (int64_t a = 1; a <= kDkiD && b == 0.0; ++a)
            if (g[i * p + a] != 0.0) b = g[(2 * kDkiDirs + i) * p + a] / g[i * p + a];
    const double eps = 4.0 * 2.220446049250313e-16;
    for (int64_t i = 0; i < kDkiDirs; ++i) {
        const double *d = g + i * p, *v = g + (kDkiDirs + i) * p, *c = g + (2 * kDkiDirs + i) * p;
        for (int64_t a = 0; a < p; ++a) {
            const bool in_d = a >= 1 && a <= kDkiD, in_v = a > kDkiD;
            const double want = in_d ? b * d[a] : in_v ? -v[a] : 0.0;
            const double err = c[a] - want, size = want < 0.0 ? -want : want;
            if ((!in_d && d[a] != 0.0) || (!in_v && v[a] != 0.0)) return false;
            if (!((err < 0.0 ? -err : err) <= eps * size)) return false;
        }
    }
    *bound = b;
    return true;
}

// ---- signal sources ---------------------------------------------------------------------
//
// A CTA owns `count` consecutive voxels, whose rows are contiguous in memory: it copies them
// into shared memory with coalesced loads, then each thread turns its own row into log
// signals (T) in a thread-strided shared array ys[j * BLOCK + tid], computed once per voxel.

// log_s (v, n) double, as larmor._core.fit_log_signal receives it.
struct LogSource {
    const double* log_s;
    int64_t n;
    // Warp-cooperative: ys[j] = y_j of one voxel, lanes over j (coalesced).
    template <class T>
    __device__ __forceinline__ void warp_stage(int64_t voxel, T* ys, int lane) const {
        for (int j = lane; j < n; j += 32) ys[j] = T(log_s[voxel * n + j]);
    }
    // y_i, i counting the (v, n) rows' entries.
    template <class T>
    __device__ __forceinline__ T entry(int64_t, int64_t i) const {
        return T(log_s[i]);
    }
};

// float32 signals (v, n) with a per-voxel floor for samples that are not finite and positive
// (src/larmor/dwi/inputs.py:227-252), logged in T.
struct FlooredSource {
    const float* s;
    const double* floor;
    int64_t n;
    template <class T>
    __device__ __forceinline__ void warp_stage(int64_t voxel, T* ys, int lane) const {
        const T lf = dev_log<T>(T(floor[voxel]));
        for (int j = lane; j < n; j += 32) {
            const float x = s[voxel * n + j];
            ys[j] = (isfinite(x) && x > 0.0f) ? dev_log<T>(T(x)) : lf;
        }
    }
    template <class T>
    __device__ __forceinline__ T entry(int64_t voxel, int64_t i) const {
        const float x = s[i];
        return dev_log<T>((isfinite(x) && x > 0.0f) ? T(x) : T(floor[voxel]));
    }
};

// float32 signals (v, n) prepared as DKIModel.fit does before its log fit
// (src/larmor/dwi/dki.py:243-250): where the voxel's S0 differs from the mean of its own b0s
// (relative 1e-9), the b0 samples become S0; diffusion-weighted samples are capped at S0; then
// samples that are not finite and positive become floor[voxel]. Without S0 (s0 == NULL) only
// the floor applies.
struct CappedSource {
    const float* s;
    const double* s0;      // (v,) or NULL
    const double* floor;   // (v,)
    const uint8_t* is_b0;  // (n,) device
    int64_t n;
    template <class T>
    __device__ __forceinline__ void warp_stage(int64_t voxel, T* ys, int lane) const {
        const T lf = dev_log<T>(T(floor[voxel]));
        if (s0 == nullptr) {
            for (int j = lane; j < n; j += 32) {
                const float x = s[voxel * n + j];
                ys[j] = (isfinite(x) && x > 0.0f) ? dev_log<T>(T(x)) : lf;
            }
            return;
        }
        const double s0v = s0[voxel];
        // The mean of the voxel's own b0s, summed in measurement order as numpy does for short
        // rows.
        double own = 0.0;
        int count = 0;
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + lane;
            const bool b0 = j < n && is_b0[j];
            const double x = b0 ? double(s[voxel * n + j]) : 0.0;
            unsigned set = __ballot_sync(0xffffffffu, b0);
            count += __popc(set);
            for (; set; set &= set - 1u) own += __shfl_sync(0xffffffffu, x, __ffs(set) - 1);
        }
        own = count ? own / count : 0.0;
        const bool repaired = !(fabs(s0v - own) <= 1e-9 * fabs(own));
        for (int j = lane; j < n; j += 32) {
            double x = double(s[voxel * n + j]);
            if (is_b0[j]) {
                if (repaired) x = s0v;
            } else {
                x = isnan(x) ? x : fmin(x, s0v);
            }
            ys[j] = (isfinite(x) && x > 0.0) ? dev_log<T>(T(x)) : lf;
        }
    }
};

}  // namespace lar
