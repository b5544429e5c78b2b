// Shapes and the operator entry of the two-atom V3 kernel (k_v3s.cu), shared with the tensor-core operator
// pass (k_v3tc.cu) and the iterative kappa (k_bte.cu).
#pragma once
#include "spring_internal.cuh"

namespace spring {
namespace {
namespace s3 {

constexpr int NB = 2, N = 6, NA = 7;
constexpr int MAXT = 9;

// One entry of the Gaussian BTE scattering operator: row r0 = q0 slot * 6 + s0, grid modes
// k1 = g1 * 6 + s1 and k2 = g2 * 6 + s2 of an enumerated pair, and the temperature-free parts of
// its coefficient c = (n1 - n2) P + (1 + n1 + n2) Q: P = 4 W (d(w0 + w1 - w2) - d(w0 + w2 - w1)),
// Q = 4 W d(w0 - w1 - w2) (halved, and the second delta of P absent, when q1 = q2).
struct BteEntry {
    int r0, k1, k2, pad;
    double P, Q;
};
static_assert(sizeof(BteEntry) == 32, "BTE entry");
constexpr double EXP_CUT_BTE = 40.0;  // exp(-40) = 4e-18 of a delta's peak: terms below are dropped

}  // namespace s3
}  // namespace
}  // namespace spring
