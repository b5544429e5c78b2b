// e^-x of the delta weights (k_v4tc.cu).  Compiles as plain C++ too, with the same roundings.
#pragma once
#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define SPRING_HD __host__ __device__ __forceinline__
#else
#define SPRING_HD inline
#endif

namespace spring {

// e^-x for 0 <= x <= 40 (relative error below 2.3e-16), without branches so that several run side by side: Cody and
// Waite's two-step reduction by ln 2, the Taylor polynomial to r^13 (remainder below 5e-18 for |r| <= ln 2 / 2)
// in Estrin's order.
SPRING_HD double exp_neg(double x) {
    constexpr double SHIFT = 6755399441055744.0;  // 1.5 2^52: the sum's low word is the rounded integer
    const double t = fma(-x, 1.4426950408889634, SHIFT), k = t - SHIFT;
    const double r = fma(-k, 2.3190468138462996e-17, fma(-k, 0.6931471805599453, -x));
    const double r2 = r * r, r4 = r2 * r2;
    const double a = fma(r, 1.0 / 6, 1.0 / 2), b = fma(r, 1.0 / 120, 1.0 / 24), c = fma(r, 1.0 / 5040, 1.0 / 720);
    const double d = fma(r, 1.0 / 362880, 1.0 / 40320), e = fma(r, 1.0 / 39916800, 1.0 / 3628800);
    const double f = fma(r, 1.0 / 6227020800.0, 1.0 / 479001600);
    const double lo = fma(r2, b, a), mid = fma(r2, d, c), hi = fma(r2, f, e);
    const double y = 1.0 + fma(r2, fma(r4, fma(r4, hi, mid), lo), r);
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(y) + __double2loint(t) * (1 << 20), __double2loint(y));
#else
    long long bt, by;  // the low word of t is the exponent to add
    memcpy(&bt, &t, 8);
    memcpy(&by, &y, 8);
    by += (long long)((unsigned long long)(long long)(int)bt << 52);
    double v;
    memcpy(&v, &by, 8);
    return v;
#endif
}

}  // namespace spring
