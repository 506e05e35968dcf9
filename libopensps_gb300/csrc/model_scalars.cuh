// Per-model FP64 scalars shared by the batch's, the no-allocation entry point's and the reverse pass's parameter
// kernels. GB300's FP64 pipe takes a warp instruction every 64 cycles per SM sub-partition, whatever the lanes in use,
// so these forms count FP64 instructions: reciprocals of constants from the host, one logarithm of 1 + z for every use
// of it, table searches started from where the table's own form puts the value.
#pragma once
#include <cuda_runtime.h>
#include <cmath>
#include "context.h"

namespace sps {

// The number of leading entries of a strictly monotonic table a[0 .. n) with a[i] <= v (ascending) or a[i] > v
// (descending): the bisection of find_interval0 without its end cases, from a guess (a few dependent loads instead of
// ten to thirteen when the guess is near; right for any guess).
template <bool ASC>
__device__ __forceinline__ int count_from(const double *__restrict__ a, int n, double v, int guess) {
    auto in = [&](int i) { const double x = __ldg(a + i); return ASC ? x <= v : x > v; };
    int g = min(max(guess, 0), n);
    while (g < n && in(g)) ++g;
    while (g > 0 && !in(g - 1)) --g;
    return g;
}

// The first entry of an ascending table that is >= v (n: none), from a guess.
__device__ __forceinline__ int lower_bound_from(const double *__restrict__ a, int n, double v, int guess) {
    int g = min(max(guess, 0), n);
    while (g < n && __ldg(a + g) < v) ++g;
    while (g > 0 && __ldg(a + g - 1) >= v) --g;
    return g;
}

// The cosmology table's interval of redshift z (0 .. 498; the table's redshifts fall with the index, its scale factors
// are evenly spaced from 1 / 1001 to 1).
__device__ __forceinline__ int cosmology_interval(const double *__restrict__ zt, double z) {
    const float a = 1.f / (1.f + (float)z);
    const int guess = (int)((a - 1.f / 1001.f) * (499.f / (1.f - 1.f / 1001.f))) + 1;
    return max(0, min(count_from<false>(zt, 500, z, guess) - 1, 498));
}

// e^x - 1 for 0 <= x <= small steps: the Taylor series to x^8 below 1/32 (x^9 / 9! < 1e-19), expm1 above.
__device__ __forceinline__ double expm1_step(double x) {
    if (!(fabs(x) < 0.03125)) return expm1(x);
    double r = fma(x, 1.0 / 8.0, 1.0);
    r = fma(x * (1.0 / 7.0), r, 1.0);
    r = fma(x * (1.0 / 6.0), r, 1.0);
    r = fma(x * (1.0 / 5.0), r, 1.0);
    r = fma(x * (1.0 / 4.0), r, 1.0);
    r = fma(x * (1.0 / 3.0), r, 1.0);
    r = fma(x * (1.0 / 2.0), r, 1.0);
    return x * r;
}

// Grid constants formed once on the host.
struct GridScalars {
    double dlnl, inv_dlnl, inv_em1;   // step in ln lambda, its inverse, 1 / (e^dlnl - 1)
};
inline GridScalars grid_scalars(double dlnl) { return {dlnl, 1.0 / dlnl, 1.0 / std::expm1(dlnl)}; }

// The observed frame at redshift z (l1z = ln(1 + z)): the shift of lambda / (1 + z) on the log-uniform grid in pixels
// (observed pixel j reads rest pixels j - n0 - 1 and j - n0 at t, the same t for every interior pixel), and the
// magnitudes' distance term (observed_frame_z, distance_term: src/spectra/opensps_batch_photometry.f90:784-903).
__device__ __forceinline__ void observed_frame(double z, double l1z, const GridScalars &g, const double *__restrict__ zt,
                                               const double *__restrict__ dl, float4 &zi, double &dd) {
    zi = make_float4(__int_as_float(0), 0.f, 0.f, 0.f);
    dd = 0.0;
    if (!(fabs(z) > SAFE_FLOOR)) return;
    const double s = l1z * g.inv_dlnl;
    const double n0 = floor(s), phi = s - n0;
    zi.x = __int_as_float((int)n0);
    zi.y = phi > 0.0 ? (float)(expm1_step((1.0 - phi) * g.dlnl) * g.inv_em1) : 0.f;
    zi.z = (float)s;
    zi.w = 1.f;
    const int i = cosmology_interval(zt, z);
    const double z0 = __ldg(zt + i), d0 = __ldg(dl + i);
    const double dm = fma((__ldg(dl + i + 1) - d0) / (__ldg(zt + i + 1) - z0), z - z0, d0);
    // 5 log10(dm / 10) - 2.5 log10(1 + z)
    if (dm == dm && dm > SAFE_FLOOR) dd = (5.0 * log(dm * 0.1) - 2.5 * l1z) * 0.43429448190325182765;
}

}  // namespace sps
