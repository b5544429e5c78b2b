// Linear-tetrahedron helpers shared by the 3-phonon, isotope, iterative-BTE,
// 4-phonon and path-mode kernels.
//
// FindgAndIver (src/Kappa/Src/TetrahedronIntegration_m.f90:93-218): the
// weight g and vertex weights I of a tetrahedron whose sorted vertex energies
// are M[0..3], at the energy Mqs.  kappa.x takes the cases with >= / <= bounds;
// LineWidth.x (src/LineWidth/Src/TetrahedronIntegration_m.f90:113-169) and
// kappa_iter.x use strict bounds.  my_sort (:18-90) is an ascending sort of the
// four vertices.
#pragma once

namespace spring {
namespace tet {

// Weights in the form the sums use them, A[v] = g I[v] / 6 of sorted energies M[0..3], and g (FindgAndIver).
// Its vertex weights of the middle case divide by g; in the product with g that division cancels, so
// four reciprocals of energy differences replace its 14 divisions (every remaining term of one weight has
// the same sign, so the result is as accurate as the differences).  Undefined weights stay NaN: the middle
// case at M0 = M1 = Mqs and the upper corner at M2 = M3 = Mqs, where FindgAndIver forms 0/0.  False (and
// nothing written) when Mqs lies outside.
template <bool STRICT>
static __device__ __forceinline__ bool g_weights(double x, const double* M, double& g, double* A) {
    const double t0 = x - M[0], t1 = x - M[1], t2 = x - M[2], t3 = x - M[3];
    const bool c1 = STRICT ? (x > M[0]) && (x < M[1]) : (x >= M[0]) && (x < M[1]);
    const bool c2 = STRICT ? (x > M[1]) && (x < M[2]) : (x >= M[1]) && (x < M[2]);
    const bool c3 = STRICT ? (x > M[2]) && (x < M[3]) : (x >= M[2]) && (x <= M[3]);
    if (!(c1 || c2 || c3)) return false;
    // reciprocals: r30 always; ra = 1/(M1-M0), 1/(M2-M1), 1/(M3-M2); rb = 1/(M2-M0) or, upper corner,
    // 1/(M3-M1); rc = 1/(M3-M1), middle case only
    const double r30 = 1.0 / (M[3] - M[0]);
    const double ra = 1.0 / (c1 ? M[1] - M[0] : (c2 ? M[2] - M[1] : M[3] - M[2]));
    const double rb = 1.0 / (c3 ? M[3] - M[1] : M[2] - M[0]);
    if (c2) {
        const double rc = 1.0 / (M[3] - M[1]);
        const double u = t0 * rb, w = t2 * rb, y = t1 * rc, z = t3 * rc;
        const double h = -(u * t2 + y * t3);
        const double f = ra * r30;
        g = 3.0 * f * h;
        const double hr = h * r30, ha = h * ra;
        double k = f * ONEBYSIX;
        if (t0 == 0.0) k = __longlong_as_double(0x7ff8000000000000LL);
        A[0] = k * (t0 * (w * w) - t3 * hr);
        A[1] = k * (t1 * (z * z) - t2 * ha);
        A[2] = k * (t1 * ha - t2 * (u * u));
        A[3] = k * (t0 * hr - t3 * (y * y));
    } else {
        const double t = c1 ? t0 : t3;
        const double f = (t * t) * (ra * rb * r30);  // g / 3
        g = 3.0 * f;
        const double k = f * ONEBYSIX;
        const double e30 = (c1 ? t3 : t0) * r30;
        if (c1) {
            const double kt = k * t;
            A[0] = -k * (t1 * ra + t2 * rb + e30);
            A[1] = kt * ra;
            A[2] = kt * rb;
            A[3] = kt * r30;
        } else {
            const double kt = -k * t;
            A[0] = kt * r30;
            A[1] = kt * rb;
            A[2] = kt * ra;
            A[3] = k * (e30 + t1 * rb + t2 * ra);
        }
    }
    return true;
}

// Ascending order of four keys with two integers carried along (equal keys: any order; their weights
// are equal).
static __device__ __forceinline__ void sort4_carry(double* M, int* a, int* b) {
#define SPRING_CE(i, j)                                          \
    {                                                            \
        const bool sw_ = M[j] < M[i];                            \
        const double m_ = M[i];                                  \
        M[i] = sw_ ? M[j] : m_;                                  \
        M[j] = sw_ ? m_ : M[j];                                  \
        const int a_ = a[i], b_ = b[i];                          \
        a[i] = sw_ ? a[j] : a_;                                  \
        a[j] = sw_ ? a_ : a[j];                                  \
        b[i] = sw_ ? b[j] : b_;                                  \
        b[j] = sw_ ? b_ : b[j];                                  \
    }
    SPRING_CE(0, 1) SPRING_CE(2, 3) SPRING_CE(0, 2) SPRING_CE(1, 3) SPRING_CE(1, 2)
#undef SPRING_CE
}

static __device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace tet
}  // namespace spring
