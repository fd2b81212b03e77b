#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline

static int __float_as_int(float x) { int i; std::memcpy(&i, &x, 4); return i; }
static float __int_as_float(int i) { float x; std::memcpy(&x, &i, 4); return x; }
static double __hiloint2double(int hi, int lo)
{
    const uint64_t b = (static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32) |
                       static_cast<uint32_t>(lo);
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}

#include "slq_scale.cuh"

// y[i] = x[i] * s[i] as a product's epilogue computes it (the double product
// where y_scaled gives none), wide[i] = whether it did, 2^896 f64_of_finite(x[i])
// and y[i] with the NaN of x[i]
extern "C" void scale(int n, const float* x, const double* s, float* y, int* wide, double* back,
                      float* shown)
{
    for (int i = 0; i < n; ++i)
    {
        float hi, lo;
        slq::scale_pair(s[i], hi, lo);
        y[i] = slq::y_scaled(x[i], hi, lo);
        wide[i] = !std::isfinite(y[i]);
        if (wide[i]) y[i] = static_cast<float>(static_cast<double>(x[i]) * s[i]);
        back[i] = slq::f64_of_finite(x[i]) * slq::TWO_896;
        shown[i] = slq::with_nan_of(x[i], y[i]);
    }
}
