// Reciprocal and square root of positive doubles for the diagnostics' FP64 terms.
#pragma once

#include <cuda_runtime.h>

namespace axs {

// A positive double within float range cut to float, and a normal float
// widened, both by integer operations.
__device__ __forceinline__ bool float_sized(double d)
{
    const int h = __double2hiint(d);
    return h > 0x39b00000 && h < 0x46300000;  // about 2^-100 to 2^100
}
__device__ __forceinline__ float cut_to_float(double d)
{
    return __int_as_float(__funnelshift_l(__double2loint(d), __double2hiint(d) - 0x38000000, 3));
}
__device__ __forceinline__ double widen_normal(float x)
{
    const int u = __float_as_int(x);
    return __hiloint2double((u >> 3) + 0x38000000, u << 29);
}

// 1/d and sqrt(d) of d > 0 in FP64 from a float estimate, for the few FP64
// operations they take (3 and 5): 1/d by one step of third order, r (1 + e + e^2)
// with e = 1 - d r (the truncated geometric series; e^3 < 2^-60), sqrt(d) by two
// Newton steps on the residual d - s^2. Correctly rounded for all but 2 and 1 values in
// a million (next to a tie; 1.3 10^9 tried), an ulp off for those.
__device__ __forceinline__ double recip_pos(double d)
{
    if (!float_sized(d)) return 1.0 / d;
    const double r = widen_normal(__fdividef(1.f, cut_to_float(d)));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double sqrt_pos(double d)
{
    if (!float_sized(d)) return sqrt(d);
    const float y = rsqrtf(cut_to_float(d));
    const double h = widen_normal(0.5f * y);
    double s = d * widen_normal(y);
    s = fma(fma(-s, s, d), h, s);
    return fma(fma(-s, s, d), h, s);
}
// Whether a sum of squares is above zero, by its bits (a comparison is an FP64 operation).
// A NaN's sign bit decides; the terms made with either answer are NaN.
__device__ __forceinline__ bool positive(double d)
{
    return (__double2hiint(d) | __double2loint(d)) != 0 && __double2hiint(d) <= 0x7ff00000;
}

// sqrt(d) scale >= threshold as the correctly rounded sqrt decides it: sqrt is asked within
// 2^-19 of the threshold (by the high words: no FP64 operation for the cells further off).
__device__ __forceinline__ bool root_reaches(double d, double scale, double threshold)
{
    double r = sqrt_pos(d) * scale;
    if ((unsigned)__double2hiint(r) - (unsigned)__double2hiint(threshold) + 1u <= 2u) r = sqrt(d) * scale;
    return r >= threshold;
}

}  // namespace axs
