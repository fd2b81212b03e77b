// FP32 values times FP64 probe scales without the FP64 conversion unit (16
// conversions per clock and SM).  Nothing from CUDA but the casts of bits, so
// that tests compile it for the host.

#ifndef SLQ_SCALE_CUH_
#define SLQ_SCALE_CUH_

#include <cfloat>
#include <cmath>

namespace slq {

// s as an FP32 pair hi + lo (48 bits), for 0 and 2^-100 <= |s| <= 2^126; other
// scales, for which a pair holds fewer bits, become a NaN.
__device__ __forceinline__ void scale_pair(double s, float& hi, float& lo)
{
    const double a = fabs(s);
    const bool fits = a == 0.0 || (a >= 0x1p-100 && a <= 0x1p126);
    hi = fits ? static_cast<float>(s) : __int_as_float(0x7fc00000);
    lo = fits ? static_cast<float>(s - static_cast<double>(hi)) : 0.0f;
}

// x s rounded to FP32 for the pair of s: the FP32 product and its exact
// remainder, which is the double product rounded to FP32 up to ties (relative
// error before the rounding 2^-48).  Not finite, whatever the double product
// is, where that does not hold: results next to FP32's largest value or past
// it, results below 2^-100 (whose remainder may be below the subnormals), an x
// that is not finite and a scale without a pair.  The caller looks for these
// and computes them in FP64.  A zero product is taken as it is: of an x or of
// the scale of a stopped probe that is zero, or below 2^-150.
__device__ __forceinline__ float y_scaled(float x, float hi, float lo)
{
    const float p = x * hi;
    const float y = p + fmaf(x, lo, fmaf(x, hi, -p));
    // 0 < |p| < 2^-100, from the bits without the sign; a zero passes
    constexpr unsigned SMALL = 2u * 0x0d800000u;
    const bool small = 2u * static_cast<unsigned>(__float_as_int(p)) - 1u < SMALL - 1u;
    return small ? __int_as_float(0x7fc00000) : y;
}

// 2^-896 x as a double, from the bits of x: exact for every finite x, zeros
// and subnormals included (the FP32 exponent is read with the FP64 bias).
__device__ __forceinline__ double f64_of_finite(float x)
{
    const int b = __float_as_int(x);
    return __hiloint2double((b >> 3) & static_cast<int>(0x8fffffffu), b << 29);
}
constexpr double TWO_896 = 0x1p896;

// y for a finite x, NaN for an x that is not (the same bits but for the sign
// of a zero): makes a sum of f64_of_finite(x) y show such an x.
__device__ __forceinline__ float with_nan_of(float x, float y) { return fmaf(x, 0.0f, y); }

}  // namespace slq

#endif  // SLQ_SCALE_CUH_
