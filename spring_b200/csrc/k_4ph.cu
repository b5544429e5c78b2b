// Four-phonon scattering on the device.
//
//  - Enumeration, MomentumConsrv4th + Permutation4th
//    (src/Kappa/Src/QuasiMomentumConsrv4th_m.f90:32-312).  The sequential covering loop
//    has a closed form: (q1,q2) is visited in grid order and the first ordering of a
//    grid multiset {q1,q2,q3} met by the loop covers every other ordering, so (q1,q2)
//    is a representative iff its key q1*Nq+q2 is the smallest of the orderings of its
//    multiset; quartet numbers come from a scan.  Each representative then writes its
//    Allq1q2q3 cells in the reference's order (direct entry, then the five
//    permutations with the reference's "no new permutation" test on the integer
//    vectors), so the arrays are bit-identical to the reference algorithm's.
//  - V4 -> W4, ScatterMatEl4 / ScatterProbability4 (src/Kappa/Src/FourthOrder_m.f90:286-473),
//    regrouped like V3: D_mu[a][nu b][eta c][ro d] = sum over slots of each basis block of
//    FC4 e^{i q1.R1} e^{i q2.R2} e^{i q3.R3} m^-1/2 m^-1/2 m^-1/2, then four Ndof^5
//    contractions with e3, e2, e1, e0.  FP64.  Two-atom cells (Ndof 6).
//  - Rates.  Tetrahedron: TetrahedronIntegration4th / SumOverPolarization /
//    FindFandOmegaVer_4th (src/Kappa/Src/Tetrahedron4th_sep.f90:37-425), with the
//    reference's reading of the stored quartet W through `per` for every permutation
//    type; Gaussian: the same three channels with delta(w0 - M) (build-side form),
//    summed over every ordered grid (q1, q2) - each distinct ordering of a quartet's
//    grid points once - with W taken from the quartet's own W4.
// Roofline: FP64 FMA for V4 (222 kflop phase-folded FC4 + 249 kflop contractions per
// quartet); FP64 ALU for the tetrahedron sums.
#include <algorithm>
#include <cub/cub.cuh>

#include "spring_internal.cuh"
#include "tetra.cuh"

namespace spring {
namespace {

constexpr int NB = 2, N = 6, NA_MAX = 8, QB = 2;
constexpr double EXP_CUT = 40.0;  // exp(-40) = 4e-18 of a delta's peak: terms below it are dropped

__device__ __forceinline__ int imod(int a, int n) {
    int r = a % n;
    return r < 0 ? r + n : r;
}

// q3 = G - (q0 + q1 + q2) with the first G of (0,+1,-1)^3 inside [-N/2, N/2]^3 (componentwise).
__device__ __forceinline__ int partner4(const int* q0, const int* q1, const int* q2, const int* nn, int* q3) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int b = nn[d] / 2;
        const int v = -(q0[d] + q1[d] + q2[d]);
        int w = v;
        if (w > b || w < -b) {
            w = v + nn[d];
            if (w > b || w < -b) w = v - nn[d];
        }
        q3[d] = w;
    }
    return imod(q3[0], nn[0]) + nn[0] * (imod(q3[1], nn[1]) + nn[1] * imod(q3[2], nn[2]));
}

struct Mesh3 {
    int n[3];
};

__global__ void k_enum4_flags(int nq, Mesh3 m, const int* __restrict__ q0, const int* __restrict__ qint,
                              int* __restrict__ g3o, int* __restrict__ rep) {
    const long long total = (long long)nq * nq;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int g1 = (int)(i / nq), g2 = (int)(i % nq);
        int q3[3];
        const int g3 = partner4(q0, qint + 3 * g1, qint + 3 * g2, m.n, q3);
        g3o[i] = g3;
        const long long k = i, L = nq;
        const long long o[5] = {g1 * L + g3, g2 * L + g1, g2 * L + g3, g3 * L + g1, g3 * L + g2};
        bool r = true;
#pragma unroll
        for (int j = 0; j < 5; ++j) r = r && (k <= o[j]);
        rep[i] = r ? 1 : 0;
    }
}

__global__ void k_enum4_write(int nq, Mesh3 m, const int* __restrict__ q0, const int* __restrict__ qint,
                              const int* __restrict__ g3a, const int* __restrict__ rep, const int* __restrict__ pos,
                              int* __restrict__ all, int* __restrict__ perm, long long cap, int4* __restrict__ quart,
                              unsigned long long* __restrict__ total) {
    const int per[5][3] = {{0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    const long long tot = (long long)nq * nq;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
        if (!rep[i]) continue;
        const int g1 = (int)(i / nq), g2 = (int)(i % nq), g3 = g3a[i];
        const int cnt = pos[i] + 1;
        if (quart) quart[cnt - 1] = make_int4(g1, g2, g3, 0);
        if (perm && cnt <= cap) {
            perm[3 * (size_t)(cnt - 1)] = g1 + 1;
            perm[3 * (size_t)(cnt - 1) + 1] = g2 + 1;
            perm[3 * (size_t)(cnt - 1) + 2] = g3 + 1;
        }
        int Q[3][3];
        partner4(q0, qint + 3 * g1, qint + 3 * g2, m.n, Q[2]);
        for (int d = 0; d < 3; ++d) {
            Q[0][d] = qint[3 * g1 + d];
            Q[1][d] = qint[3 * g2 + d];
        }
        const int G[3] = {g1, g2, g3};
        if (all) {
            int* e = all + 3 * ((size_t)g1 * nq + g2);
            e[0] = 0; e[1] = cnt; e[2] = g3 + 1;
        }
        int pg[5][3];
        unsigned long long newc = 0;
        for (int pp = 0; pp < 5; ++pp) {
            for (int k = 0; k < 3; ++k) pg[pp][k] = G[per[pp][k]];
            bool nonew = true;
            for (int k = 0; k < 3; ++k)
                for (int d = 0; d < 3; ++d)
                    if (Q[per[pp][k]][d] != Q[k][d]) nonew = false;
            for (int qq = 0; qq < pp; ++qq)
                nonew = nonew || (pg[pp][0] == pg[qq][0] && pg[pp][1] == pg[qq][1] && pg[pp][2] == pg[qq][2]);
            if (!nonew) {
                ++newc;
                if (all) {
                    int* e = all + 3 * ((size_t)pg[pp][0] * nq + pg[pp][1]);
                    e[0] = pp + 1; e[1] = cnt; e[2] = pg[pp][2] + 1;
                }
            }
        }
        atomicAdd(total, 1ull + newc);
    }
}

// ------------------------------------------------------------------------- V4
struct V4Args {
    int nq, nT, nq0, q0, na, nquart;
    double mfac, onebysigma, onebysigma2;
    int pol_lo[4], pol_hi[4];
};

struct V4Smem {
    double2 e[QB][4][36];          // e0 (times m_mu^-1/2 by row), e1, e2, e3: [s][row]
    double2 ppp[QB][NA_MAX * NA_MAX * NA_MAX];
    double2 A[QB][648];            // D4 [a][nb][ec][rd], then T2 [a nb][s2][s3]
    double2 B[QB][648];            // T1 [a nb ec][s3], then T3 [a][s1][s2 s3]
    double2 phi[QB][1296];         // Phi, then W (as doubles in .x)
    double lw[MAX_NDOF][10];       // [s0][T] rate accumulators (T <= 9), last column unused
    double ph[QB][3][NA_MAX][2];
    double wq[QB][3][N];           // omega of the quartet's three grid points
    double nq[QB][9][3][N];        // their occupations per temperature
    int g[QB][4];                  // g1 g2 g3 valid
    unsigned short slot[NA_MAX * NA_MAX * NA_MAX];  // (n1 na + n2) na + n3 by block of basis atoms
};

// One CTA works off groups of QB quartets.  Most of the work is D4: FC4, 444 KB out of L2, against the triple
// phase products.  The neighbour triples are put in the order of their (nu, eta, ro) blocks, so that a block is
// one loop with its loads in flight ahead; a warp reads 32 consecutive entries abcd of a triple, each for QB
// quartets, and two warps share their sums.  Bound by the L2 reads and their latency.  5^3, ten q0 (26 700
// quartets): 4.45 -> 2.75 ms against one thread per (quartet, entry) with a loop nest over the blocks' neighbours
// (3.27 with four lanes per entry: 64-byte pieces of unaligned rows).
constexpr int V4T = 256;
template <int EPI>
__global__ void __launch_bounds__(V4T, 2)
k_v4(V4Args a, const int4* __restrict__ quart, const double* __restrict__ fc4, const double* __restrict__ posr,
     const int* __restrict__ btyp, const int* __restrict__ off, const double* __restrict__ mrs,
     const double* __restrict__ qpnt, const int* __restrict__ q0int, const double2* __restrict__ ev0,
     const double* __restrict__ om0, const double* __restrict__ ob0, const double* __restrict__ nbe0,
     const double2* __restrict__ evg, const double* __restrict__ omg, const double* __restrict__ obg,
     const double* __restrict__ nbeg, double* __restrict__ out_rate, double* __restrict__ out_w) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V4Smem& S = *reinterpret_cast<V4Smem*>(smem_raw);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int na = a.na;
    const bool gq0 = q0int[0] == 0 && q0int[1] == 0 && q0int[2] == 0;
    if (EPI == 0)
        for (int i = tid; i < MAX_NDOF * 10; i += nt) (&S.lw[0][0])[i] = 0.0;
    for (int grp = blockIdx.x; grp * QB < a.nquart; grp += gridDim.x) {
        __syncthreads();
        if (tid < QB) {
            const int k = grp * QB + tid;
            const bool v = k < a.nquart;
            const int4 q = v ? quart[k] : make_int4(0, 0, 0, 0);
            S.g[tid][0] = q.x; S.g[tid][1] = q.y; S.g[tid][2] = q.z; S.g[tid][3] = v;
        }
        __syncthreads();
        for (int i = tid; i < QB * 4 * 36; i += nt) {
            const int p = i / 144, w = (i / 36) % 4, k = i % 36;
            double2 v = w == 0 ? ev0[k] : evg[(size_t)S.g[p][w - 1] * 36 + k];
            if (w == 0) {
                const double mm = mrs[(k % 6) / 3];
                v.x *= mm;
                v.y *= mm;
            }
            S.e[p][w][k] = v;
        }
        for (int i = tid; i < QB * 1296; i += nt) S.phi[i / 1296][i % 1296] = make_double2(0.0, 0.0);
        for (int mu = 0; mu < NB; ++mu) {
            const int* o = off + mu * (NB + 1);
            for (int i = tid; i < QB * 3 * na; i += nt) {
                const int p = i / (3 * na), k = (i / na) % 3, Nn = i % na;
                const int gg = S.g[p][k];
                const double* R = posr + ((size_t)mu * na + Nn) * 3;
                const double qr = qpnt[3 * gg] * R[0] + qpnt[3 * gg + 1] * R[1] + qpnt[3 * gg + 2] * R[2];
                double sn, cs;
                sincos(qr, &sn, &cs);
                const double mm = mrs[btyp[mu * na + Nn]];
                S.ph[p][k][Nn][0] = mm * cs;
                S.ph[p][k][Nn][1] = mm * sn;
            }
            __syncthreads();
            for (int i = tid; i < QB * na * na * na; i += nt) {
                const int p = i / (na * na * na), n1 = (i / (na * na)) % na, n2 = (i / na) % na, n3 = i % na;
                const double* x = S.ph[p][0][n1];
                const double* y = S.ph[p][1][n2];
                const double* z = S.ph[p][2][n3];
                const double xr = x[0] * y[0] - x[1] * y[1], xi = x[0] * y[1] + x[1] * y[0];
                // slots are sorted by basis atom: place among the (nu, eta, ro) blocks
                const int h = o[1], c[2] = {h, na - h};
                const int nu = n1 >= h, eta = n2 >= h, ro = n3 >= h;
                const int m1 = n1 - nu * h, m2 = n2 - eta * h, m3 = n3 - ro * h;
                const int k = nu * h * na * na + c[nu] * (eta * h * na + c[eta] * ro * h) + (m1 * c[eta] + m2) * c[ro] + m3;
                S.ppp[p][k] = make_double2(xr * z[0] - xi * z[1], xr * z[1] + xi * z[0]);
                if (p == 0) S.slot[k] = (unsigned short)((n1 * na + n2) * na + n3);
            }
            __syncthreads();
            // D4: the eight (nu, eta, ro) blocks in turn, both quartets; even triples into A, odd ones into B
            if (tid < 6 * 32) {
                const int j = tid / 96, r = tid % 96, rc = min(r, 80);
                const int al = rc / 27, be = (rc / 9) % 3, ga = (rc / 3) % 3, de = rc % 3;
                const double* f = fc4 + (size_t)mu * na * na * na * 81 + rc;
                const int c[2] = {o[1], na - o[1]};
                int k0 = 0;
#pragma unroll 1
                for (int b = 0; b < 8; ++b) {
                    const int nu = b >> 2, eta = (b >> 1) & 1, ro = b & 1;
                    const int k1 = k0 + (nu ? c[1] : c[0]) * (eta ? c[1] : c[0]) * (ro ? c[1] : c[0]);
                    double2 acc[QB];
#pragma unroll
                    for (int p = 0; p < QB; ++p) acc[p] = make_double2(0.0, 0.0);
#pragma unroll 12
                    for (int k = k0 + j; k < k1; k += 2) {
                        const double fv = __ldg(f + (size_t)S.slot[k] * 81);
#pragma unroll
                        for (int p = 0; p < QB; ++p) {
                            const double2 q = S.ppp[p][k];
                            acc[p].x = fma(fv, q.x, acc[p].x);
                            acc[p].y = fma(fv, q.y, acc[p].y);
                        }
                    }
                    k0 = k1;
                    if (r < 81)
#pragma unroll
                        for (int p = 0; p < QB; ++p)
                            (j ? S.B : S.A)[p][((al * 6 + nu * 3 + be) * 6 + eta * 3 + ga) * 6 + ro * 3 + de] = acc[p];
                }
            }
            __syncthreads();
            for (int i = tid; i < QB * 648; i += nt) {
                const double2 x = S.B[i / 648][i % 648];
                double2& y = S.A[i / 648][i % 648];
                y.x += x.x;
                y.y += x.y;
            }
            __syncthreads();
            // T1[a nb ec][s3] = sum_rd D4[a nb ec][rd] e3(rd, s3)
            for (int u = tid; u < QB * 108; u += nt) {
                const int p = u / 108, row = u % 108;
                double2 acc[N];
#pragma unroll
                for (int s = 0; s < N; ++s) acc[s] = make_double2(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const double2 d = S.A[p][row * 6 + k];
#pragma unroll
                    for (int s = 0; s < N; ++s) {
                        const double2 e = S.e[p][3][s * 6 + k];
                        acc[s].x = fma(d.x, e.x, fma(-d.y, e.y, acc[s].x));
                        acc[s].y = fma(d.x, e.y, fma(d.y, e.x, acc[s].y));
                    }
                }
#pragma unroll
                for (int s = 0; s < N; ++s) S.B[p][row * 6 + s] = acc[s];
            }
            __syncthreads();
            // T2[a nb][s2][s3] = sum_ec e2(ec, s2) T1[a nb ec][s3]
            for (int u = tid; u < QB * 108; u += nt) {
                const int p = u / 108, ab = (u % 108) / 6, s2 = u % 6;
                double2 acc[N];
#pragma unroll
                for (int s = 0; s < N; ++s) acc[s] = make_double2(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const double2 e = S.e[p][2][s2 * 6 + k];
#pragma unroll
                    for (int s = 0; s < N; ++s) {
                        const double2 t = S.B[p][(ab * 6 + k) * 6 + s];
                        acc[s].x = fma(e.x, t.x, fma(-e.y, t.y, acc[s].x));
                        acc[s].y = fma(e.x, t.y, fma(e.y, t.x, acc[s].y));
                    }
                }
#pragma unroll
                for (int s = 0; s < N; ++s) S.A[p][(ab * 6 + s2) * 6 + s] = acc[s];
            }
            __syncthreads();
            // T3[a][s1][s2 s3] = sum_nb e1(nb, s1) T2[a nb][s2 s3]
            for (int u = tid; u < QB * 108; u += nt) {
                const int p = u / 108, al = (u % 108) / 36, s1 = (u % 36) / 6, s2 = u % 6;
                double2 acc[N];
#pragma unroll
                for (int s = 0; s < N; ++s) acc[s] = make_double2(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const double2 e = S.e[p][1][s1 * 6 + k];
#pragma unroll
                    for (int s = 0; s < N; ++s) {
                        const double2 t = S.A[p][((al * 6 + k) * 6 + s2) * 6 + s];
                        acc[s].x = fma(e.x, t.x, fma(-e.y, t.y, acc[s].x));
                        acc[s].y = fma(e.x, t.y, fma(e.y, t.x, acc[s].y));
                    }
                }
#pragma unroll
                for (int s = 0; s < N; ++s) S.B[p][((al * 6 + s1) * 6 + s2) * 6 + s] = acc[s];
            }
            __syncthreads();
            // Phi[s0][s1 s2 s3] += sum_a e0'(mu a, s0) T3[a][s1 s2 s3]
            for (int u = tid; u < QB * 216; u += nt) {
                const int p = u / 216, s0 = (u % 216) / 36, s12 = u % 36;
#pragma unroll
                for (int s = 0; s < N; ++s) {
                    double2 acc = S.phi[p][(s0 * 36 + s12) * 6 + s];
#pragma unroll
                    for (int al = 0; al < 3; ++al) {
                        const double2 e = S.e[p][0][s0 * 6 + mu * 3 + al];
                        const double2 t = S.B[p][(al * 36 + s12) * 6 + s];
                        acc.x = fma(e.x, t.x, fma(-e.y, t.y, acc.x));
                        acc.y = fma(e.x, t.y, fma(e.y, t.x, acc.y));
                    }
                    S.phi[p][(s0 * 36 + s12) * 6 + s] = acc;
                }
            }
            __syncthreads();
        }
        // W4 = |Phi|^2 (1/w0)(1/w1)(1/w2)(1/w3) Sctr4THz2/Nq^2, zero for Gamma acoustic modes
        for (int i = tid; i < QB * 1296; i += nt) {
            const int p = i / 1296, k = i % 1296;
            const int s0 = k / 216, s1 = (k / 36) % 6, s2 = (k / 6) % 6, s3 = k % 6;
            const int g1 = S.g[p][0], g2 = S.g[p][1], g3 = S.g[p][2];
            const bool z = (gq0 && s0 < 3) || (g1 == 0 && s1 < 3) || (g2 == 0 && s2 < 3) || (g3 == 0 && s3 < 3);
            const double2 v = S.phi[p][k];
            const double a2 = v.x * v.x + v.y * v.y;
            const double W = z ? 0.0 : (a2 * (ob0[s0] * obg[(size_t)g1 * N + s1] * obg[(size_t)g2 * N + s2] *
                                              obg[(size_t)g3 * N + s3])) * a.mfac;
            S.phi[p][k].x = W;
            if (EPI == 1 && S.g[p][3]) out_w[(size_t)(grp * QB + p) * 1296 + k] = W;
        }
        if (EPI == 0) {
            __syncthreads();
            // Gaussian: every distinct ordering (qa, qb, qc) of the quartet's grid points.  The
            // frequencies and occupations of the three points are staged; each (mode quad, ordering)
            // is screened in FP32 against the window where a delta weight exceeds exp(-40) of its
            // peak, and only the rest is evaluated in FP64.
            for (int i = tid; i < QB * 3 * N; i += nt) {
                const int p = i / (3 * N), k = (i / N) % 3, sx = i % N;
                const int gg = S.g[p][k];
                S.wq[p][k][sx] = omg[(size_t)gg * N + sx];
                for (int t = 0; t < a.nT; ++t) S.nq[p][t][k][sx] = nbeg[(size_t)t * a.nq * N + (size_t)gg * N + sx];
            }
            __syncthreads();
            const int perms[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
            const double pre = a.onebysigma * ONEBYSQRT2PI;
            const float Rf = (float)(sqrt(2.0 * EXP_CUT) / a.onebysigma * 1.0001 + 1e-3);
            for (int i = tid; i < QB * 1296; i += nt) {
                const int p = i / 1296, k = i % 1296;
                if (!S.g[p][3]) continue;
                const int s0 = k / 216, sa = (k / 36) % 6, sb = (k / 6) % 6, sc = k % 6;
                if (s0 < (gq0 ? 3 : a.pol_lo[0]) || s0 > a.pol_hi[0]) continue;  // SumOverPolarization s0Strt
                if (sa < a.pol_lo[1] || sa > a.pol_hi[1] || sb < a.pol_lo[2] || sb > a.pol_hi[2] ||
                    sc < a.pol_lo[3] || sc > a.pol_hi[3])
                    continue;
                const int* G = S.g[p];
                const double w0 = om0[s0];
                const float f0 = (float)w0;
                for (int pi = 0; pi < 6; ++pi) {
                    const int ia = perms[pi][0], ib = perms[pi][1], ic = perms[pi][2];
                    const int ga = G[ia], gb = G[ib];
                    bool dup = false;
                    for (int pj = 0; pj < pi; ++pj)
                        dup = dup || (G[perms[pj][0]] == ga && G[perms[pj][1]] == gb);
                    if (dup) continue;
                    const double wa = S.wq[p][ia][sa], wb = S.wq[p][ib][sb], wc = S.wq[p][ic][sc];
                    const float fa = (float)wa, fb = (float)wb, fc = (float)wc;
                    if (fabsf(f0 - (fa + fb + fc)) >= Rf && fabsf(f0 - (fb + fc - fa)) >= Rf &&
                        fabsf(f0 - (fc - fa - fb)) >= Rf)
                        continue;
                    int m[3];
                    m[ia] = sa;
                    m[ib] = sb;
                    m[ic] = sc;
                    const double Wv = S.phi[p][((s0 * 6 + m[0]) * 6 + m[1]) * 6 + m[2]].x;
                    if (Wv == 0.0) continue;
                    const double d1 = w0 - (wa + wb + wc), d2 = w0 - (wb + wc - wa), d3 = w0 - (wc - wa - wb);
                    const double x1 = 0.5 * a.onebysigma2 * (d1 * d1), x2 = 0.5 * a.onebysigma2 * (d2 * d2),
                                 x3 = 0.5 * a.onebysigma2 * (d3 * d3);
                    const double e1 = x1 < EXP_CUT ? pre * exp(-x1) : 0.0;
                    const double e2 = x2 < EXP_CUT ? pre * exp(-x2) : 0.0;
                    const double e3 = x3 < EXP_CUT ? pre * exp(-x3) : 0.0;
                    if (e1 == 0.0 && e2 == 0.0 && e3 == 0.0) continue;
                    for (int t = 0; t < a.nT; ++t) {
                        const double na_ = S.nq[p][t][ia][sa], nbb = S.nq[p][t][ib][sb], nc = S.nq[p][t][ic][sc];
                        const double n0 = nbe0[(size_t)t * a.nq0 * N + s0];
                        const double v = ONEBYSIX * (Wv * (na_ * nbb * nc / n0)) * e1 +
                                         0.5 * (Wv * ((1.0 + na_) * nbb * nc / n0)) * e2 +
                                         0.5 * (Wv * ((1.0 + na_) * (1.0 + nbb) * nc / n0)) * e3;
                        atomicAdd(&S.lw[s0][t], v);
                    }
                }
            }
        }
    }
    if (EPI == 0) {
        __syncthreads();
        for (int i = tid; i < N * a.nT; i += nt) {
            const int s0 = i / a.nT, t = i % a.nT;
            if (S.lw[s0][t] != 0.0) atomicAdd(&out_rate[((size_t)t * a.nq0 + a.q0) * N + s0], S.lw[s0][t]);
        }
    }
}

// ------------------------------------------------------------------------- tetrahedron
struct T4Args {
    int nq, nT, nq0, q0, ntet, nquart;
    int pol_lo[4], pol_hi[4];
};

// One lane per tetrahedron over q2, one q1 per block.  The channels' energies are w1 + p, p - w1 and m - w1 with
// p = w2 + w3 and m = w3 - w2, so for every (s2, s3) the lane sorts p and m once, screens the 18 (s0, channel)
// of every s1 in FP32 against their ranges (widened by far more than the rounding) into a mask of up to 108
// bits, and, when the warp has a hit, forms the six reciprocals of each set once: about 7 % of the checks hit
// (6^3), 7 per (tetrahedron, s2, s3), all of which use them.  The hits of the 32 tetrahedra are queued and
// evaluated 32 at a time (each lane working off its own mask instead idles behind the busiest one: 16.6 ms);
// what an evaluation reads of its tetrahedron (sorted energies, reciprocals, occupation products, W offsets)
// lies in that lane's shared-memory column.
// Vertex energies closer than 1e-5 of their magnitude (a tetrahedron that holds both legs of a pair, the
// resonances w0 + w1 -> w0 + w1) are the exception: there the rounding of (w1 + w2) + w3 decides between the
// cases, so such hits form, sort and weight the channel's own energies.
// The legs are not folded: the reference's reading of the stored W is not symmetric in them.
// One temperature: 5^3, ten q0 116.6 -> 5.8 ms, 6^3, sixteen 546 -> 25 ms against one thread per (q1, tetrahedron,
// s1, s2, s3) that ran every formula any lane of its warp needed; 15.3 and 45 ms with each hit sorting its own
// energies and taking its own reciprocals.  Bound by issue (IPC 1.75) and the latency of the W reads.
constexpr int T4W = 4;  // warps per block
// n1 / n0 overflows by itself for n0 near the smallest double, where n2 n3 makes up for it: a power of two moves
// between the two factors, which changes no bit of their product elsewhere.
constexpr double T4UP = 18446744073709551616.0;  // 2^64

template <int NT>
struct T4Smem {
    double acc[T4W][N * NT][32];        // per-lane sums [s0][T]
    double val[T4W][2][10][32];         // p, m sets: sorted energies; 1/(30), (10), (21), (32), (20), (31)
    double nf[T4W][2][NT][4][32];       // n2 n3 and (1 + n2) n3 by vertex, times T4UP
    int off[T4W][4][32];                // by vertex: W offset of (s2, s3) | stride of s1 << 8
    int pos[T4W][4][32], v2[T4W][4][32], v3[T4W][4][32];  // quartet and points of each vertex
    int rank[T4W][2][32];               // vertices by rank, two bits each; 256: well separated
    unsigned short queue[T4W][32 * 6 * 3 * N];  // lane | check << 5
    double w0m[N][N], w0p[N][N];        // w0 - w1, w0 + w1 [s1][s0]
    float f0m[N][8], f0p[N][8];         // the same in FP32 (two values of padding)
    double fac[NT][2][N][N];            // n1 / n0 / 6, (1 + n1) / n0 / 2 [T][.][s1][s0], over T4UP
    double w0[N];
};

template <int NT>
__global__ void __launch_bounds__(32 * T4W, 3) k_tetra4(T4Args a, int per2, int nb2, const int4* __restrict__ tet,
                                                        const int* __restrict__ all, const double* __restrict__ Wq,
                                                        const int* __restrict__ q0int, const double* __restrict__ om0,
                                                        const double* __restrict__ nbe0, const double* __restrict__ omg,
                                                        const double* __restrict__ nbeg, double* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T4Smem<NT>& S = *reinterpret_cast<T4Smem<NT>*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool gq0 = q0int[0] == 0 && q0int[1] == 0 && q0int[2] == 0;
    const int s0a = gq0 ? 3 : a.pol_lo[0], s0e = a.pol_hi[0];
    for (int i = lane; i < N * NT * 32; i += 32) (&S.acc[warp][0][0])[i] = 0.0;
    if (threadIdx.x < N) S.w0[threadIdx.x] = om0[threadIdx.x];
    unsigned live = 0;
#pragma unroll
    for (int k = 0; k < 3 * N; ++k)
        if (k % N >= s0a && k % N <= s0e) live |= 1u << (3 * N - 1 - k);
    const int groups = (a.ntet + 31) / 32;
    double(*acc)[32] = S.acc[warp];
    for (int q1 = blockIdx.y; q1 < a.nq; q1 += gridDim.y) {
        __syncthreads();
        for (int i = threadIdx.x; i < N * N; i += blockDim.x) {
            const int s1 = i / N, s0 = i % N;
            const double w0 = S.w0[s0], w1 = omg[(size_t)q1 * N + s1];
            S.w0m[s1][s0] = w0 - w1;
            S.w0p[s1][s0] = w0 + w1;
            S.f0m[s1][s0] = (float)(w0 - w1);
            S.f0p[s1][s0] = (float)(w0 + w1);
            for (int T = 0; T < a.nT; ++T) {
                const double n1 = nbeg[((size_t)T * a.nq + q1) * N + s1], n0 = nbe0[(size_t)T * a.nq0 * N + s0];
                S.fac[T][0][s1][s0] = ONEBYSIX * (n1 / (n0 * T4UP));
                S.fac[T][1][s1][s0] = 0.5 * ((1.0 + n1) / (n0 * T4UP));
            }
        }
        __syncthreads();
        for (int u = blockIdx.x * T4W + warp; u < groups * nb2; u += gridDim.x * T4W) {
            const int t = u / nb2 * 32 + lane;
            const int s2a = a.pol_lo[2] + u % nb2 * per2, s2e = min(s2a + per2 - 1, a.pol_hi[2]);
            bool on = t < a.ntet;
            const int4 tv = on ? tet[t] : make_int4(0, 0, 0, 0);
            const int v2[4] = {tv.x, tv.y, tv.z, tv.w};
            int v3[4], cst[4];  // cst: strides of s1, s2, s3 in W
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int* e = all + 3 * ((size_t)q1 * a.nq + v2[v]);
                const int ty = on ? e[0] : 0, ps = on ? e[1] - 1 : 0;
                v3[v] = on ? e[2] - 1 : 0;
                // every cell is written by the enumeration; an unwritten one is skipped, not read
                const bool ok = ty >= 0 && ty <= 5 && ps >= 0 && ps < a.nquart && v3[v] >= 0 && v3[v] < a.nq;
                on = on && ok;
                if (!ok) v3[v] = 0;
                S.pos[warp][v][lane] = ps;
                S.v2[warp][v][lane] = v2[v];
                S.v3[warp][v][lane] = v3[v];
                // modes of the stored quartet read through the reference's permutation
                // 0: 123, 1: 132, 2: 213, 3: 231, 4: 312, 5: 321
                const int c1 = ty < 2 ? 36 : (ty == 2 || ty == 4 ? 6 : 1);
                const int c2 = ty == 2 || ty == 3 ? 36 : (ty == 0 || ty == 5 ? 6 : 1);
                cst[v] = c1 | c2 << 8 | (43 - c1 - c2) << 16;
            }
            for (int s2 = s2a; s2 <= s2e; ++s2) {
                double w2[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) w2[v] = omg[(size_t)v2[v] * N + s2];
                for (int s3 = a.pol_lo[3]; s3 <= a.pol_hi[3]; ++s3) {
                    double p[4], m[4];
                    int ip[4] = {0, 1, 2, 3}, im[4] = {0, 1, 2, 3}, unused[4] = {0, 0, 0, 0};
                    float mag = 0.0f;
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        const double w3 = omg[(size_t)v3[v] * N + s3];
                        p[v] = w2[v] + w3;
                        m[v] = w3 - w2[v];
                        mag += (float)fmax(fabs(p[v]), fabs(m[v]));
                    }
                    tet::sort4_carry(p, ip, unused);
                    tet::sort4_carry(m, im, unused);
                    // screen: one bit per check, set outside
                    const float pl = (float)p[0], ph = (float)p[3], ml = (float)m[0], mh = (float)m[3];
                    const float pm = 0.5f * (pl + ph), mm = 0.5f * (ml + mh);
                    const float pr = 0.5f * (ph - pl), mr = 0.5f * (mh - ml);
                    unsigned long long hit[2] = {0, 0};
#pragma unroll
                    for (int s1 = 0; s1 < N; ++s1) {
                        if (s1 < a.pol_lo[1] || s1 > a.pol_hi[1]) continue;
                        unsigned o = 0;
                        // FP32 rounding of the energies is below 4e-7 of the sum of magnitudes
                        // (|w1| and |w0| are at most |w0 - w1| + |w0 + w1|; a NaN leaves every check open)
                        const float marg = 1e-6f * (mag + fabsf(S.f0m[s1][0]) + fabsf(S.f0p[s1][0]));
                        const float hp = pr + marg, hm = mr + marg;
                        float wm[N], wp[N];
#pragma unroll
                        for (int i = 0; i < N; ++i) {
                            wm[i] = S.f0m[s1][i];
                            wp[i] = S.f0p[s1][i];
                        }
#pragma unroll
                        for (int i = 0; i < N; ++i) o = __funnelshift_l(__float_as_uint(hp - fabsf(wm[i] - pm)), o, 1);
#pragma unroll
                        for (int i = 0; i < N; ++i) o = __funnelshift_l(__float_as_uint(hp - fabsf(wp[i] - pm)), o, 1);
#pragma unroll
                        for (int i = 0; i < N; ++i) o = __funnelshift_l(__float_as_uint(hm - fabsf(wp[i] - mm)), o, 1);
                        if (on) hit[s1 / 3] |= (unsigned long long)(~o & live) << (18 * (s1 % 3));
                    }
                    if (!__any_sync(0xffffffffu, (hit[0] | hit[1]) != 0)) continue;
                    const double gap = 1e-5 * (double)mag;  // false for a NaN too
                    const bool sp = p[1] - p[0] > gap && p[2] - p[1] > gap && p[3] - p[2] > gap;
                    const bool sm = m[1] - m[0] > gap && m[2] - m[1] > gap && m[3] - m[2] > gap;
                    S.rank[warp][0][lane] = ip[0] | ip[1] << 2 | ip[2] << 4 | ip[3] << 6 | sp << 8;
                    S.rank[warp][1][lane] = im[0] | im[1] << 2 | im[2] << 4 | im[3] << 6 | sm << 8;
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        S.off[warp][v][lane] = (s2 * (cst[v] >> 8 & 255) + s3 * (cst[v] >> 16)) | (cst[v] & 255) << 8;
#pragma unroll
                    for (int set = 0; set < 2; ++set) {
                        const double* e = set ? m : p;
                        double(*V)[32] = S.val[warp][set];
#pragma unroll
                        for (int k = 0; k < 4; ++k) V[k][lane] = e[k];
                        V[4][lane] = 1.0 / (e[3] - e[0]);
                        V[5][lane] = 1.0 / (e[1] - e[0]);
                        V[6][lane] = 1.0 / (e[2] - e[1]);
                        V[7][lane] = 1.0 / (e[3] - e[2]);
                        V[8][lane] = 1.0 / (e[2] - e[0]);
                        V[9][lane] = 1.0 / (e[3] - e[1]);
                    }
#pragma unroll 1
                    for (int T = 0; T < a.nT; ++T) {
                        const double* nb = nbeg + (size_t)T * a.nq * N;
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            const double n2 = nb[(size_t)v2[v] * N + s2], n3 = nb[(size_t)v3[v] * N + s3];
                            const double u3 = n3 * T4UP;
                            S.nf[warp][0][T][v][lane] = n2 * u3;
                            S.nf[warp][1][T][v][lane] = (1.0 + n2) * u3;
                        }
                    }
                    const int c = __popcll(hit[0]) + __popcll(hit[1]);
                    int before = 0, tot = 0;
                    const unsigned lt = (1u << lane) - 1;
#pragma unroll
                    for (int b = 0; b < 7; ++b) {
                        const unsigned bal = __ballot_sync(0xffffffffu, (c >> b) & 1);
                        before += __popc(bal & lt) << b;
                        tot += __popc(bal) << b;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        for (unsigned long long in = hit[h]; in; in &= in - 1)
                            S.queue[warp][before++] = (unsigned short)(lane | (54 * h + __ffsll((long long)in) - 1) << 5);
                    __syncwarp();
                    for (int i = lane; i < tot; i += 32) {
                        const unsigned code = S.queue[warp][i];
                        const int tl = code & 31, bit = code >> 5, s1 = bit / 18, k = 17 - (bit - 18 * s1);
                        const int ch = k >= 12 ? 2 : (k >= 6 ? 1 : 0), s0 = k - 6 * ch, set = ch >> 1;
                        const int rk = S.rank[warp][set][tl];
                        double A[4];
                        int vs[4];  // vertex of each weight
                        if (!(rk & 256)) {
                            double M[4];
                            const double w1 = omg[(size_t)q1 * N + s1];
                            int none[4] = {0, 0, 0, 0};
#pragma unroll
                            for (int v = 0; v < 4; ++v) {
                                const double y = omg[(size_t)S.v2[warp][v][tl] * N + s2], w3 = omg[(size_t)S.v3[warp][v][tl] * N + s3];
                                M[v] = ch == 0 ? w1 + y + w3 : (ch == 1 ? y + w3 - w1 : w3 - w1 - y);
                                vs[v] = v;
                            }
                            tet::sort4_carry(M, vs, none);
                            double gw;
                            if (!tet::g_weights<false>(S.w0[s0], M, gw, A)) continue;
                        } else {
                            const double(*V)[32] = S.val[warp][set];
                            const double x = ch == 0 ? S.w0m[s1][s0] : S.w0p[s1][s0];
                            const double e0 = V[0][tl], e1 = V[1][tl], e2 = V[2][tl], e3 = V[3][tl];
                            const double t0 = x - e0, t1 = x - e1, t2 = x - e2, t3 = x - e3;
                            const bool c1 = x >= e0 && x < e1, c2 = x >= e1 && x < e2, c3 = x >= e2 && x <= e3;
                            if (!(c1 || c2 || c3)) continue;
                            // the weights of tet::g_weights from the set's reciprocals
                            const double r30 = V[4][tl], ra = V[c1 ? 5 : (c2 ? 6 : 7)][tl], rb = V[c3 ? 9 : 8][tl];
                            if (c2) {
                                const double rc = V[9][tl];
                                const double uu = t0 * rb, ww = t2 * rb, y = t1 * rc, z = t3 * rc;
                                const double hh = -(uu * t2 + y * t3), hr = hh * r30, ha = hh * ra;
                                const double kf = ra * r30 * ONEBYSIX;
                                A[0] = kf * (t0 * (ww * ww) - t3 * hr);
                                A[1] = kf * (t1 * (z * z) - t2 * ha);
                                A[2] = kf * (t1 * ha - t2 * (uu * uu));
                                A[3] = kf * (t0 * hr - t3 * (y * y));
                            } else {
                                const double tt = c1 ? t0 : t3;
                                const double kf = (tt * tt) * (ra * rb * r30) * ONEBYSIX;
                                const double far = (c1 ? t3 : t0) * r30;
                                const double kt = c1 ? kf * tt : -kf * tt;
                                const double near = c1 ? -kf * (t1 * ra + t2 * rb + far) : kf * (far + t1 * rb + t2 * ra);
                                A[0] = c1 ? near : kt * r30;
                                A[1] = c1 ? kt * ra : kt * rb;
                                A[2] = c1 ? kt * rb : kt * ra;
                                A[3] = c1 ? kt * r30 : near;
                            }
#pragma unroll
                            for (int r = 0; r < 4; ++r) vs[r] = rk >> (2 * r) & 3;
                        }
                        const double* Ws = Wq + s0 * 216;
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const int o = S.off[warp][vs[r]][tl];
                            const double W = Ws[(size_t)S.pos[warp][vs[r]][tl] * 1296 + (o & 255) + s1 * (o >> 8)];
                            A[r] = isnan(A[r]) ? 0.0 : A[r] * W;  // undefined weights count as zero
                        }
#pragma unroll
                        for (int T = 0; T < NT; ++T) {
                            if (T >= a.nT) break;
                            double sum = 0.0;
#pragma unroll
                            for (int r = 0; r < 4; ++r) sum = fma(A[r], S.nf[warp][set][T][vs[r]][tl], sum);
                            acc[s0 * NT + T][lane] += sum * S.fac[T][ch ? 1 : 0][s1][s0];
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    __syncthreads();
    for (int i = warp; i < N * NT; i += T4W) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < T4W; ++w) v += S.acc[w][i][lane];
        v = tet::warp_sum(v);
        const int s0 = i / NT, T = i % NT;
        if (lane == 0 && T < a.nT && v != 0.0) atomicAdd(&out[((size_t)T * a.nq0 + a.q0) * N + s0], v);
    }
}

template <int NT>
int launch_tetra4(spring_ctx* c, const T4Args& t, const int* all, const double* wq, const int* q0i, const double* om0,
                  const double* nbe0, double* d_rate) {
    const int n2 = t.pol_hi[2] - t.pol_lo[2] + 1, groups = (t.ntet + 31) / 32;
    int per2 = 6;  // shorter units (of s2) while the chip is not full
    while (per2 > 1 && (long long)t.nq * groups * ((n2 + per2 - 1) / per2) < 148LL * 192) --per2;
    const int nb2 = (n2 + per2 - 1) / per2;
    // one unit a warp: the blocks of a q1 end together and the scheduler evens out the rest
    const int gy = std::min(t.nq, 65535), gx = (groups * nb2 + T4W - 1) / T4W;
    const size_t smem = sizeof(T4Smem<NT>);
    cudaFuncSetAttribute(k_tetra4<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "tetra4: injected launch failure");
    k_tetra4<NT><<<dim3(gx, gy), 32 * T4W, smem, c->stream>>>(t, per2, nb2, reinterpret_cast<const int4*>(c->d_tetra.p), all,
                                                              wq, q0i, om0, nbe0, c->ph_grid.omega.p, c->ph_grid.nbe.p,
                                                              d_rate);
    return launch_check(c, "k_tetra4");
}

// Enumerate the quartets of q0 into device buffers (grid-pair scratch owned by the caller).
struct Enum4Bufs {
    DBuf<int> g3, rep, pos, all;
    DBuf<int4> quart;
    DBuf<unsigned long long> total;
};

int enumerate4(spring_ctx* c, int q0, Enum4Bufs& b, bool want_all, int* d_perm, long long cap, long long* h_counts) {
    const long long tot = (long long)c->nq * c->nq;
    if (tot > 0x7fffffffLL) return fail(c, SPRING_ERR_UNSUPPORTED, "Nq^2 exceeds 2^31");
    SPRING_CHECK(dalloc(c, b.g3, tot, "quartet scratch"));
    SPRING_CHECK(dalloc(c, b.rep, tot, "quartet scratch"));
    SPRING_CHECK(dalloc(c, b.pos, tot, "quartet scratch"));
    SPRING_CHECK(dalloc(c, b.total, 1, "quartet scratch"));
    if (want_all) SPRING_CHECK(dalloc(c, b.all, tot * 3, "Allq1q2q3"));
    Mesh3 m{{c->mesh[0], c->mesh[1], c->mesh[2]}};
    const int* q0v = c->d_irr_int.p + 3 * q0;
    const int threads = 256, blocks = (int)std::min<long long>((tot + threads - 1) / threads, 148LL * 32);
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "enumerate4: injected launch failure");
    k_enum4_flags<<<blocks, threads, 0, c->stream>>>(c->nq, m, q0v, c->d_qint.p, b.g3.p, b.rep.p);
    SPRING_CHECK(launch_check(c, "k_enum4_flags"));
    SPRING_CHECK(run_exclusive_scan(c, b.rep.p, b.pos.p, (int)tot));
    int last = 0;
    SPRING_CHECK(d2h_sum2(c, b.pos.p + tot - 1, b.rep.p + tot - 1, &last, "quartet count"));
    const long long nquart = last;
    SPRING_CHECK(dalloc(c, b.quart, std::max<long long>(nquart, 1), "quartet list"));
    SPRING_CHECK(zero(c, b.total.p, sizeof(unsigned long long), "quartet count"));
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "enumerate4: injected launch failure");
    k_enum4_write<<<blocks, threads, 0, c->stream>>>(c->nq, m, q0v, c->d_qint.p, b.g3.p, b.rep.p, b.pos.p,
                                                     want_all ? b.all.p : nullptr, d_perm, cap, b.quart.p, b.total.p);
    SPRING_CHECK(launch_check(c, "k_enum4_write"));
    h_counts[0] = nquart;
    return SPRING_OK;
}

size_t bytes4(const Enum4Bufs& b) {
    return sizeof(int) * (b.g3.n + b.rep.n + b.pos.n + b.all.n) + sizeof(int4) * b.quart.n;
}

void free4(Enum4Bufs& b) {
    dfree(b.g3); dfree(b.rep); dfree(b.pos); dfree(b.all); dfree(b.quart); dfree(b.total);
}

}  // namespace

int run_enumerate4_fortran(spring_ctx* c, int q0, int* d_all, int* d_perm, long long cap, long long* h_counts) {
    Enum4Bufs b;
    int rc = enumerate4(c, q0, b, d_all != nullptr, d_perm, cap, h_counts);
    unsigned long long total = 0;
    if (rc == SPRING_OK) rc = d2h(c, &total, b.total.p, sizeof total, "quartet total");
    h_counts[1] = (long long)total;
    if (rc == SPRING_OK && d_all) {
        const size_t bytes = sizeof(int) * 3 * (size_t)c->nq * c->nq;
        cudaError_t e = cudaMemcpyAsync(d_all, b.all.p, bytes, cudaMemcpyDeviceToDevice, c->stream);
        if (e != cudaSuccess) rc = cuda_fail(c, e, "Allq1q2q3 copy");
    }
    cudaStreamSynchronize(c->stream);
    free4(b);
    return rc;
}

// Quartet list of q0 (0-based) in buffers kept by the context: (g1, g2, g3, 0) sorted by (g1, g2).
int run_enum4_list(spring_ctx* c, int q0, const int4** d_quart, long long* nquart) {
    if (!c->e4) c->e4 = new Enum4Bufs();
    Enum4Bufs& b = *static_cast<Enum4Bufs*>(c->e4);
    long long cnt[2] = {0, 0};
    SPRING_CHECK(enumerate4(c, q0, b, false, nullptr, 0, cnt));
    *d_quart = b.quart.p;
    *nquart = cnt[0];
    return SPRING_OK;
}

void free_enum4(spring_ctx* c) {
    if (!c->e4) return;
    Enum4Bufs* b = static_cast<Enum4Bufs*>(c->e4);
    free4(*b);
    delete b;
    c->e4 = nullptr;
}

int run_lw4(spring_ctx* c, int q0_first, int n_q0, int delta_mode, double sigma, const int* pol4, double* d_rate) {
    if (c->nb != NB || c->na4 > NA_MAX || c->nT > 9)
        return fail(c, SPRING_ERR_UNSUPPORTED, "four-phonon path handles two-atom cells, Na4 <= %d, <= 9 temperatures",
                    NA_MAX);
    V4Args a{};
    a.nq = c->nq;
    a.nT = c->nT;
    a.nq0 = c->nq0;
    a.na = c->na4;
    a.mfac = host_constants().Sctr4THz2 / (double(c->nq) * double(c->nq));
    a.onebysigma = delta_mode == SPRING_DELTA_GAUSS ? 1.0 / sigma : 0.0;
    a.onebysigma2 = a.onebysigma * a.onebysigma;
    for (int k = 0; k < 4; ++k) {
        a.pol_lo[k] = pol4 ? pol4[2 * k] - 1 : 0;
        a.pol_hi[k] = pol4 ? pol4[2 * k + 1] - 1 : N - 1;
    }
    const size_t smem = sizeof(V4Smem);
    cudaFuncSetAttribute(k_v4<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_v4<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    // quartet lists (up to 256 MB) and their W (up to 512 MB) stay with the context
    if (!c->e4) c->e4 = new Enum4Bufs();
    Enum4Bufs& b = *static_cast<Enum4Bufs*>(c->e4);
    DBuf<double>& wq = c->d_w4;
    int rc = SPRING_OK;
    for (int q0 = q0_first; rc == SPRING_OK && q0 < q0_first + n_q0; ++q0) {
        long long cnt[2];
        rc = enumerate4(c, q0, b, delta_mode == SPRING_DELTA_TETRA, nullptr, 0, cnt);
        if (rc != SPRING_OK) break;
        a.q0 = q0;
        a.nquart = (int)cnt[0];
        const int groups = (a.nquart + QB - 1) / QB;
        const int grid = std::max(1, std::min(groups, 148 * 2));
        const double2* ev0 = c->ph_irr.evec.p + (size_t)q0 * 36;
        const double* om0 = c->ph_irr.omega.p + (size_t)q0 * N;
        const double* ob0 = c->ph_irr.oneby.p + (size_t)q0 * N;
        const double* nbe0 = c->ph_irr.nbe.p + (size_t)q0 * N;
        const int* q0i = c->d_irr_int.p + 3 * q0;
        if (delta_mode == SPRING_DELTA_GAUSS) {
            if (launch_injected(c)) { rc = fail(c, SPRING_ERR_INJECTED, "v4: injected launch failure"); break; }
            k_v4<0><<<grid, V4T, smem, c->stream>>>(a, b.quart.p, c->d_fc4.p, c->d_fc4_posr.p, c->d_fc4_btyp.p,
                                                    c->d_fc4_off.p, c->d_mass_rs.p, c->d_qpnt.p, q0i, ev0, om0, ob0,
                                                    nbe0, c->ph_grid.evec.p, c->ph_grid.omega.p, c->ph_grid.oneby.p,
                                                    c->ph_grid.nbe.p, d_rate, nullptr);
            rc = launch_check(c, "k_v4<gauss>");
        } else {
            // asking for the free memory takes up to milliseconds on a busy host: only to grow the buffer
            const size_t need = (size_t)a.nquart * 1296 * sizeof(double);
            size_t free_b = 0, total_b = 0;
            if (need > wq.n * sizeof(double)) cudaMemGetInfo(&free_b, &total_b);
            if (need > wq.n * sizeof(double) && need > (free_b + wq.n * sizeof(double)) / 2) {
                rc = fail(c, SPRING_ERR_UNSUPPORTED, "tetrahedron four-phonon W of one q0 needs %zu bytes", need);
                break;
            }
            if ((rc = dalloc(c, wq, (size_t)a.nquart * 1296, "quartet W")) != SPRING_OK) break;
            if (launch_injected(c)) { rc = fail(c, SPRING_ERR_INJECTED, "v4: injected launch failure"); break; }
            k_v4<1><<<grid, V4T, smem, c->stream>>>(a, b.quart.p, c->d_fc4.p, c->d_fc4_posr.p, c->d_fc4_btyp.p,
                                                    c->d_fc4_off.p, c->d_mass_rs.p, c->d_qpnt.p, q0i, ev0, om0, ob0,
                                                    nbe0, c->ph_grid.evec.p, c->ph_grid.omega.p, c->ph_grid.oneby.p,
                                                    c->ph_grid.nbe.p, nullptr, wq.p);
            if ((rc = launch_check(c, "k_v4<wstore>")) != SPRING_OK) break;
            T4Args t{};
            t.nq = c->nq;
            t.nT = c->nT;
            t.nq0 = c->nq0;
            t.q0 = q0;
            t.ntet = 6 * c->nq;
            t.nquart = a.nquart;
            for (int k = 0; k < 4; ++k) {
                t.pol_lo[k] = a.pol_lo[k];
                t.pol_hi[k] = a.pol_hi[k];
            }
            rc = c->nT == 1 ? launch_tetra4<1>(c, t, b.all.p, wq.p, q0i, om0, nbe0, d_rate)
                 : c->nT <= 3 ? launch_tetra4<3>(c, t, b.all.p, wq.p, q0i, om0, nbe0, d_rate)
                              : launch_tetra4<9>(c, t, b.all.p, wq.p, q0i, om0, nbe0, d_rate);
        }
    }
    cudaStreamSynchronize(c->stream);
    if (wq.n * sizeof(double) > ((size_t)512 << 20)) dfree(wq);
    if (bytes4(b) > ((size_t)256 << 20)) free4(b);
    return rc;
}

}  // namespace spring
