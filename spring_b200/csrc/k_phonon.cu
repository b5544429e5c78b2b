// Harmonic phonons on the device: get_phonon (src/Kappa/Src/DynaMat_mod.f90:486-709)
// for a batch of q-points, one CTA per q-point (two-atom cells: a part of a warp).
//   1. D(q) and dD/dq_k from FC2 (DynMatgv_SR, DynaMat_mod.f90:98-190).
//   2. Hermitian eigensolve in FP64 by cyclic complex Jacobi with round-robin
//      (parallel) pair ordering: n/2 disjoint rotations per step, column
//      updates then row updates, until the off-diagonal mass is below 1e-30 of
//      the diagonal's or a sweep finds no element above 1e-16 sqrt|a_pp a_qq|
//      (threshold Jacobi).  Eigenvalues ascending like LAPACK zheevd.  The
//      eigenvector phase (gauge) is the eigensolver's own: only gauge-invariant
//      quantities are comparable with LAPACK's.
//   3. omega = sqrt|lambda| (negative for imaginary modes), v = Re(e^H dD e)/(2 omega),
//      nBE for every temperature, 1/(omega wTHz); Gamma acoustic modes zeroed.
//   4. On a Gamma-centred mesh only one point of each (q, -q) pair is solved: the
//      other gets e(-q) = conj(e(q)) (D(-q) = D(q)* for real force constants),
//      the same omega, 1/omega and nBE, and v(-q) = -v(q).  The irreducible
//      points run in the same launch.
// Latency bound: the FLOPs (~10 n^3 per sweep) are few, the rotation rounds a serial chain.
#include <algorithm>
#include <vector>

#include "spring_internal.cuh"

namespace spring {
namespace {

struct PhArgs {
    int nb, n, na2;
    double latvec[9];
    double wTHz, vg_ms, BEConv;
    int nT;
    const double2* dd;  // dipole-dipole D and dD/dq per work item ([4][n][n]), or null
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }

// (x, y) <- (c x - s e y, s x + c e y), its roundings written out: eigenvectors of a degenerate branch
// depend on the last bit, and should not on how a caller is compiled
__device__ __forceinline__ void rot_ey(double c, double s, double2 ey, double2& x, double2& y) {
    y = make_double2(__fma_rn(s, x.x, __dmul_rn(c, ey.x)), __fma_rn(s, x.y, __dmul_rn(c, ey.y)));
    x = make_double2(__fma_rn(c, x.x, -__dmul_rn(s, ey.x)), __fma_rn(c, x.y, -__dmul_rn(s, ey.y)));
}
__device__ __forceinline__ void rot_col(double c, double s, double2 e, double2& x, double2& y) {
    rot_ey(c, s, make_double2(__fma_rn(e.x, y.x, -__dmul_rn(e.y, y.y)), __fma_rn(e.x, y.y, __dmul_rn(e.y, y.x))), x, y);
}
__device__ __forceinline__ void rot_row(double c, double s, double2 e, double2& x, double2& y) {
    rot_ey(c, s, make_double2(__fma_rn(e.x, y.x, -__dmul_rn(e.y, y.y)), __fma_rn(e.y, y.x, __dmul_rn(e.x, y.y))), x, y);
}

constexpr int MAX_SWEEPS = 30;

// Outputs of one set of q-points: [q][s][row] eigenvectors, [q][s] scalars, [T][nq][s] nBE,
// [q][s][3] velocities; q vectors qpts[q][3].
struct PhSet {
    const double* qpts;
    double2* evec;
    double* omega;
    double* oneby;
    double* nbe;
    double* vel;
    int nq;
};

// Work item i < n_a: point list_a[i] (or i when list_a is null) of set SA; else point i - n_a of set SB.
// NN: the branches.  Bound by the chain of rotation rounds (about 160 at 24 branches), and a round
// by its rotation's dependent FP64 divisions and square roots (2460 cycles when one thread does them all
// against 1900 for the two update passes).  So three warps share a rotation (angle, threshold, phase), and
// one pass updates A on both sides by 2x2 blocks, each from and to registers; V follows one round behind,
// in the warps that have no rotations.  Rows are padded to an odd length.  24 branches, 295 points: 741 -> 259 us against one
// thread per rotation, passes of their own for columns, rows and V, and serial sums.  Every branch count has its
// own instance: with n at run time the index arithmetic makes 3, 9, 12, 15, 18 and 21 branches 50, 169, 202, 294,
// 489 and 664 us at 8^3, against 42, 138, 160, 231, 394 and 548 (the same bits).
constexpr int PHT = 384;
template <int NN>
__global__ void __launch_bounds__(PHT, 2) k_phonons(PhArgs a, PhSet SA, const int* __restrict__ list_a, int n_a, PhSet SB,
                                                    int n_b, const double* __restrict__ fc2, const int* __restrict__ idx,
                                                    const int* __restrict__ num, const double* __restrict__ mrs,
                                                    const double* __restrict__ temps) {
    extern __shared__ double2 sm[];
    constexpr int n = NN;
    const int m = n + (n & 1), mh = m / 2;  // even size for round-robin pairing (index n is a dummy)
    const int ld = n | 1;        // row stride of A and V
    double2* A = sm;             // [n][ld]
    double2* V = A + n * ld;     // [n][ld]
    double2* dD = V + n * ld;    // [3][n][n]
    double2* rotE2 = dD + 3 * n * n;                       // [2][m/2] e^{i phi}; the current rotations and the ones before
    double* rotC2 = reinterpret_cast<double*>(rotE2 + m);  // [2][m/2]
    double* rotS2 = rotC2 + m;                             // [2][m/2]
    double* lam = rotS2 + m;                               // [m]
    int* rotP2 = reinterpret_cast<int*>(lam + m);          // [2][m/2]
    int* rotQ2 = rotP2 + m;                                // [2][m/2]
    int* rotV2 = rotQ2 + m;                                // [2][m/2] the rotation is applied
    int* rank = rotV2 + m;                                 // [n]
    __shared__ int nrot;                                  // rotations applied in this sweep
    __shared__ double part[2][PHT / 32];                  // off-diagonal and diagonal sums by warp

    const int tid = threadIdx.x, nt = blockDim.x, warp = tid / 32, lane = tid % 32;
    for (int item = blockIdx.x; item < n_a + n_b; item += gridDim.x) {
        const bool in_a = item < n_a;
        const PhSet& P = in_a ? SA : SB;
        const int q = in_a ? (list_a ? list_a[item] : item) : item - n_a;
        const int nq = P.nq;
        double2* __restrict__ evec = P.evec;
        double* __restrict__ omega = P.omega;
        double* __restrict__ oneby = P.oneby;
        double* __restrict__ nbe = P.nbe;
        double* __restrict__ vel = P.vel;
        const double qx = P.qpts[3 * q], qy = P.qpts[3 * q + 1], qz = P.qpts[3 * q + 2];
        for (int i = tid; i < 2 * n * ld + 3 * n * n; i += nt) A[i] = make_double2(0.0, 0.0);  // A, V, dD
        __syncthreads();
        // --- phases e^{iq.R} per (mu, N), in V's place until it is set
        const bool pre = a.nb * a.na2 <= n * ld;
        for (int w = tid; pre && w < a.nb * a.na2; w += nt) {
            const int mu = w / a.na2, N = w % a.na2;
            if (N >= num[mu]) continue;
            const int* e = idx + 4 * w;
            double R[3];
            for (int r = 0; r < 3; ++r) R[r] = a.latvec[r] * e[0] + a.latvec[r + 3] * e[1] + a.latvec[r + 6] * e[2];
            const double qr = qx * R[0] + qy * R[1] + qz * R[2];
            double sn, cs;
            sincos(qr, &sn, &cs);
            V[w] = make_double2(cs, sn);
        }
        __syncthreads();
        // --- D(q), dD/dq: thread per (mu, alpha, beta); neighbours in reference order
        for (int w = tid; w < a.nb * 9; w += nt) {
            const int mu = w / 9, al = (w / 3) % 3, be = w % 3;
            const int row = 3 * mu + al;
            for (int N = 0; N < num[mu]; ++N) {
                const int* e = idx + 4 * (N + a.na2 * mu);
                const int nu = e[3] - 1;
                double R[3];
                for (int r = 0; r < 3; ++r)
                    R[r] = a.latvec[r] * e[0] + a.latvec[r + 3] * e[1] + a.latvec[r + 6] * e[2];
                double sn, cs;
                if (pre) {
                    cs = V[mu * a.na2 + N].x;
                    sn = V[mu * a.na2 + N].y;
                } else {
                    const double qr = qx * R[0] + qy * R[1] + qz * R[2];
                    sincos(qr, &sn, &cs);
                }
                const double f = fc2[((mu * a.na2 + N) * 3 + al) * 3 + be];  // fC(1,be,al,N,mu)
                const double mf = mrs[mu] * mrs[nu];
                const int col = 3 * nu + be;
                double2 t = make_double2(f * cs * mf, f * sn * mf);
                A[row * ld + col] = cadd(A[row * ld + col], t);
                for (int k = 0; k < 3; ++k)  // (i R_k) * t
                    dD[(k * n + row) * n + col] = cadd(dD[(k * n + row) * n + col], make_double2(-t.y * R[k], t.x * R[k]));
            }
        }
        __syncthreads();
        if (a.dd) {  // + DynEw, dDynEw/dq (LongEw); then the lower triangle from the upper one, as zheevd('U')
            const double2* d = a.dd + (size_t)item * 4 * n * n;
            for (int i = tid; i < 4 * n * n; i += nt) {
                double2& t = i < n * n ? A[i / n * ld + i % n] : dD[i - n * n];
                t = cadd(t, d[i]);
            }
            __syncthreads();
            for (int i = tid; i < n * n; i += nt) {
                const int r = i / n, cc = i % n;
                if (r > cc) A[r * ld + cc] = conj2(A[cc * ld + r]);
                else if (r == cc) A[r * ld + cc].y = 0.0;
            }
        }
        for (int i = tid; i < n * ld; i += nt) V[i] = make_double2(i / ld == i % ld ? 1.0 : 0.0, 0.0);
        __syncthreads();

        // --- cyclic complex Jacobi
        // V <- V U (columns p, q of every row) for the round whose rotations are in half h
        auto update_v = [&](int h, int first, int step) {
            for (int w = first; w < n * mh; w += step) {
                const int k = h * mh + w % mh;
                if (!rotV2[k]) continue;
                double2* row = V + w / mh * ld;
                const int p = rotP2[k], qq = rotQ2[k];
                double2 x = row[p], y = row[qq];
                rot_col(rotC2[k], rotS2[k], conj2(rotE2[k]), x, y);
                row[p] = x;
                row[qq] = y;
            }
        };
        int round = 0;
        for (int sweep = 0; sweep < MAX_SWEEPS; ++sweep) {
            double off = 0.0, dg = 0.0;
            for (int w = tid; w < n * n; w += nt) {
                const int i = w / n, j = w % n;
                const double2 z = A[i * ld + j];
                if (j > i) off += z.x * z.x + z.y * z.y;
                else if (j == i) dg += z.x * z.x;
            }
            for (int d = 16; d; d /= 2) {
                off += __shfl_xor_sync(~0u, off, d);
                dg += __shfl_xor_sync(~0u, dg, d);
            }
            if (lane == 0) {
                part[0][warp] = off;
                part[1][warp] = dg;
            }
            if (tid == 0) nrot = 0;
            __syncthreads();
            off = dg = 0.0;
            for (int i = 0; i < nt / 32; ++i) {
                off += part[0][i];
                dg += part[1][i];
            }
            if (off <= 1e-30 * dg || off == 0.0) break;  // the same in every thread
            for (int r = 0; r < m - 1; ++r, ++round) {
                const int half = (round & 1) * mh;
                double2* rotE = rotE2 + half;
                double *rotC = rotC2 + half, *rotS = rotS2 + half;
                int *rotP = rotP2 + half, *rotQ = rotQ2 + half, *rotV = rotV2 + half;
                // rotations of the round's pairs: warp 0 the angle, 1 whether it is applied, 2 the phase;
                // the others take V through the round before
                if (warp >= 3 && round > 0) update_v((round - 1) & 1, tid - 96, nt - 96);
                for (int k = lane; warp < 3 && k < mh; k += 32) {
                    int p, qq;
                    if (k == 0) { p = r; qq = m - 1; }
                    else { p = (r + k) % (m - 1); qq = (r - k + (m - 1)) % (m - 1); }
                    if (p > qq) { int t = p; p = qq; qq = t; }
                    if (qq >= n) {  // the dummy's partner sits out
                        if (warp == 1) {
                            rotP[k] = p;
                            rotQ[k] = qq;
                            rotV[k] = 0;
                        }
                        continue;
                    }
                    const double2 z = A[p * ld + qq];
                    const double app = A[p * ld + p].x, aqq = A[qq * ld + qq].x;
                    const double rr = hypot(z.x, z.y);
                    if (warp == 0) {
                        const double tau = (aqq - app) / (2.0 * rr);
                        const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                        const double c = 1.0 / sqrt(1.0 + t * t);
                        rotC[k] = c;
                        rotS[k] = t * c;
                    } else if (warp == 1) {
                        const bool valid = rr > 1e-300 && rr > 1e-16 * sqrt(fabs(app * aqq));
                        if (valid) atomicAdd(&nrot, 1);
                        rotP[k] = p;
                        rotQ[k] = qq;
                        rotV[k] = valid;
                    } else {
                        rotE[k] = make_double2(z.x / rr, z.y / rr);
                    }
                }
                __syncthreads();
                // A <- U^H A U by blocks {p1, q1} x {p2, q2}: its columns, then its rows; the rotated pair
                // becomes zero, its diagonal real
                for (int w = tid; w < mh * mh; w += nt) {
                    const int k2 = w % mh, p2 = rotP[k2], q2 = rotQ[k2], v2 = rotV[k2];
                    const double c2 = rotC[k2], s2 = rotS[k2];
                    const double2 eb = conj2(rotE[k2]);
                    const int k1 = w / mh, p1 = rotP[k1], q1 = rotQ[k1], v1 = rotV[k1];
                    if (!v1 && !v2) continue;
                    const double c1 = rotC[k1], s1 = rotS[k1];
                    const double2 e = rotE[k1], zero = make_double2(0.0, 0.0);
                    double2 b00 = A[p1 * ld + p2], b01 = q2 < n ? A[p1 * ld + q2] : zero;
                    double2 b10 = q1 < n ? A[q1 * ld + p2] : zero, b11 = q1 < n && q2 < n ? A[q1 * ld + q2] : zero;
                    if (v2) {
                        rot_col(c2, s2, eb, b00, b01);
                        rot_col(c2, s2, eb, b10, b11);
                    }
                    if (v1) {
                        rot_row(c1, s1, e, b00, b10);
                        rot_row(c1, s1, e, b01, b11);
                        if (k1 == k2) {
                            b00.y = b11.y = 0.0;
                            b01 = b10 = zero;
                        }
                    }
                    A[p1 * ld + p2] = b00;
                    if (q2 < n) A[p1 * ld + q2] = b01;
                    if (q1 < n) A[q1 * ld + p2] = b10;
                    if (q1 < n && q2 < n) A[q1 * ld + q2] = b11;
                }
                __syncthreads();
            }
            if (nrot == 0) break;  // nothing above the threshold: converged (nrot read after the last barrier)
            __syncthreads();
        }
        if (round > 0) update_v((round - 1) & 1, tid, nt);
        // --- ascending order (stable): rank of each eigenvalue
        for (int i = tid; i < n; i += nt) {
            const double li = A[i * ld + i].x;
            int rk = 0;
            for (int j = 0; j < n; ++j) {
                const double lj = A[j * ld + j].x;
                rk += (lj < li) || (lj == li && j < i);
            }
            rank[i] = rk;
            lam[i] = li;
        }
        __syncthreads();
        const bool gamma = fabs(qx) < CMP_PREC && fabs(qy) < CMP_PREC && fabs(qz) < CMP_PREC;
        // eigenvectors: evec[q][s][row] = V[row][col with rank s]
        for (int w = tid; w < n * n; w += nt) {
            const int col = w / n, row = w % n;
            evec[((size_t)q * n + rank[col]) * n + row] = V[row * ld + col];
        }
        // per-mode quantities; the velocities' inner sums (dD e)_i go through A
        double2* T = A;
        for (int k = 0; k < 3; ++k) {
            for (int w = tid; w < n * n; w += nt) {
                const int i = w / n, col = w % n;
                double2 t = make_double2(0.0, 0.0);
                for (int j = 0; j < n; ++j) t = cadd(t, cmul(dD[(k * n + i) * n + j], V[j * ld + col]));
                T[w] = t;
            }
            __syncthreads();
            for (int col = tid; col < n; col += nt) {
                const int s = rank[col];
                const double lv = lam[col];
                double W = sqrt(fabs(lv));
                if (fabs(lv) > EPS_F32 && lv < 0.0) W = -W;
                const bool zero_mode = gamma && s < 3;
                double2 acc = make_double2(0.0, 0.0);
                for (int i = 0; i < n; ++i) acc = cadd(acc, cmul(conj2(V[i * ld + col]), T[i * n + col]));
                vel[((size_t)q * n + s) * 3 + k] = zero_mode ? 0.0 : acc.x / (2.0 * W) * a.vg_ms;
                if (k > 0) continue;
                omega[(size_t)q * n + s] = W * a.wTHz;
                oneby[(size_t)q * n + s] = zero_mode ? 0.0 : 1.0 / (W * a.wTHz);
            }
            __syncthreads();
        }
        for (int w = tid; w < a.nT * n; w += nt) {
            const int t = w / n, col = w % n, s = rank[col];
            const double lv = lam[col];
            const double W = sqrt(fabs(lv));
            nbe[((size_t)t * nq + q) * n + s] = gamma && s < 3 ? 0.0 : 1.0 / (exp(a.BEConv * W / temps[t]) - 1.0);
        }
        __syncthreads();
    }
}

// Two-atom cells (n = 6): L lanes per q-point, 32 / L points per one-warp block, each group with its own
// shared-memory state (4 KB per point).  The same steps as k_phonons (phases once per (mu, N), then D and
// dD/dq in reference neighbour order; the same round-robin Jacobi rotations and stopping rules; ordering,
// velocities, nBE), with every control decision warp-uniform: the groups synchronise with full-warp
// barriers, a converged or idle group only skips work, and the sweep loop ends when every group of the
// warp has converged.  Bound by the dependent divisions and square roots of about 25 rotation rounds: 87 -> 49 us
// at 8^3 points (32 lanes), 89 -> 62 at 16^3 (32), 98 -> 81 at 20^3 (16), 123 -> 104 at 24^3 (8), against
// eight lanes with one lane per rotation and passes of their own for columns and rows.
constexpr int PH6_NA2 = 32;
struct Ph6 {
    double2 A[36], V[36], dD[3 * 36];
    double2 ph[2 * PH6_NA2];  // e^{i q.R} per (mu, N)
    double2 rotE[3];
    double rotC[3], rotS[3], lam[6];
    int rotP[3], rotQ[3], rotV[3], rank[6], nrot;
};

template <int L>
__global__ void __launch_bounds__(32) k_phonons_n6(PhArgs a, PhSet SA, const int* __restrict__ list_a, int n_a,
                                                  PhSet SB, int n_b, const double* __restrict__ fc2,
                                                  const int* __restrict__ idx, const int* __restrict__ num,
                                                  const double* __restrict__ mrs, const double* __restrict__ temps) {
    constexpr int n = 6, m = 6, PH6_PTS = 32 / L;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ Ph6 sh[PH6_PTS];
    const int gi = threadIdx.x / L, gl = threadIdx.x % L;
    Ph6& S = sh[gi];
    const int total = n_a + n_b;
    for (int base = blockIdx.x * PH6_PTS; base < total; base += gridDim.x * PH6_PTS) {
        const int item = base + gi;
        const bool act = item < total;
        const bool in_a = item < n_a;
        const PhSet& P = in_a ? SA : SB;
        const int q = act ? (in_a ? (list_a ? list_a[item] : item) : item - n_a) : 0;
        double qx = 0.0, qy = 0.0, qz = 0.0;
        if (act) {
            qx = P.qpts[3 * q];
            qy = P.qpts[3 * q + 1];
            qz = P.qpts[3 * q + 2];
            for (int w = gl; w < 36; w += L) S.V[w] = make_double2(w % 7 == 0 ? 1.0 : 0.0, 0.0);
            for (int w = gl; w < 2 * a.na2; w += L) {
                const int mu = w / a.na2, N = w % a.na2;
                if (N < num[mu]) {
                    const int* e = idx + 4 * (N + a.na2 * mu);
                    double R[3];
                    for (int r = 0; r < 3; ++r)
                        R[r] = a.latvec[r] * e[0] + a.latvec[r + 3] * e[1] + a.latvec[r + 6] * e[2];
                    const double qr = qx * R[0] + qy * R[1] + qz * R[2];
                    double sn, cs;
                    sincos(qr, &sn, &cs);
                    S.ph[mu * PH6_NA2 + N] = make_double2(cs, sn);
                }
            }
        }
        __syncwarp();
        // D(q), dD/dq: lane per (mu, alpha, beta), both columns in registers; neighbours in reference order
        if (act)
            for (int w = gl; w < 18; w += L) {
                const int mu = w / 9, al = (w / 3) % 3, be = w % 3;
                const int row = 3 * mu + al, nn = num[mu];
                double2 acc[2][4];
                for (int i = 0; i < 8; ++i) acc[i / 4][i % 4] = make_double2(0.0, 0.0);
#pragma unroll 2
                for (int N = 0; N < nn; ++N) {
                    const int4 e = reinterpret_cast<const int4*>(idx)[N + a.na2 * mu];
                    const int nu = e.w - 1;
                    double R[3];
                    for (int r = 0; r < 3; ++r) R[r] = a.latvec[r] * e.x + a.latvec[r + 3] * e.y + a.latvec[r + 6] * e.z;
                    const double2 pe = S.ph[mu * PH6_NA2 + N];
                    const double f = fc2[((mu * a.na2 + N) * 3 + al) * 3 + be];  // fC(1,be,al,N,mu)
                    const double mf = mrs[mu] * mrs[nu];
                    const double2 t = make_double2(f * pe.x * mf, f * pe.y * mf);
                    double2 u[4];
                    for (int k = 0; k < 4; ++k) {  // t, (i R_k) t
                        u[k] = nu ? acc[1][k] : acc[0][k];
                        u[k] = k ? cadd(u[k], make_double2(-t.y * R[k - 1], t.x * R[k - 1])) : cadd(u[k], t);
                        if (nu) acc[1][k] = u[k];
                        else acc[0][k] = u[k];
                    }
                }
                for (int nu = 0; nu < 2; ++nu) {
                    const int e = row * n + 3 * nu + be;
                    S.A[e] = acc[nu][0];
                    for (int k = 0; k < 3; ++k) S.dD[k * 36 + e] = acc[nu][1 + k];
                }
            }
        __syncwarp();
        if (act && a.dd) {  // + DynEw, dDynEw/dq (LongEw)
            const double2* d = a.dd + (size_t)item * 4 * 36;
            for (int w = gl; w < 4 * 36; w += L) {
                double2& t = w < 36 ? S.A[w] : S.dD[w - 36];
                t = cadd(t, d[w]);
            }
        }
        __syncwarp();
        if (act && a.dd)  // the lower triangle from the upper one, as zheevd('U') reads it
            for (int w = gl; w < 36; w += L) {
                const int r = w / n, cc = w % n;
                if (r > cc) S.A[w] = conj2(S.A[cc * n + r]);
                else if (r == cc) S.A[w].y = 0.0;
            }
        __syncwarp();

        // --- cyclic complex Jacobi, one group per point
        bool gdone = !act;
        for (int sweep = 0; sweep < MAX_SWEEPS; ++sweep) {
            double off = 0.0, dg = 0.0;
            if (!gdone)
                for (int w = gl; w < 36; w += L) {
                    const int i = w / n, j = w % n;
                    const double2 z = S.A[w];
                    if (i == j) dg += z.x * z.x;
                    else if (j > i) off += z.x * z.x + z.y * z.y;
                }
            for (int o = L / 2; o > 0; o >>= 1) {  // within the group; every lane gets the same sums
                off += __shfl_xor_sync(FULL, off, o);
                dg += __shfl_xor_sync(FULL, dg, o);
            }
            if (!gdone && (off <= 1e-30 * dg || off == 0.0)) gdone = true;
            if (__all_sync(FULL, gdone)) break;
            if (gl == 0) S.nrot = 0;
            __syncwarp();
            for (int r = 0; r < m - 1; ++r) {
                // lanes 0..2 the rotations' angles, 3..5 their threshold and phase, by the same instructions: a
                // division or square root of one role runs along with one of the other
                if (!gdone && gl < m) {
                    const int k = gl % 3;
                    const bool angle = gl < 3;
                    int p, qq;
                    if (k == 0) { p = r; qq = m - 1; }
                    else { p = (r + k) % (m - 1); qq = (r - k + (m - 1)) % (m - 1); }
                    if (p > qq) { const int t = p; p = qq; qq = t; }
                    const double2 z = S.A[p * n + qq];
                    const double app = S.A[p * n + p].x, aqq = S.A[qq * n + qq].x;
                    const double rr = hypot(z.x, z.y);
                    const double tau = (angle ? aqq - app : z.x) / (angle ? 2.0 * rr : rr);
                    const double sq = sqrt(angle ? 1.0 + tau * tau : fabs(app * aqq));
                    const double t = (angle ? (tau >= 0.0 ? 1.0 : -1.0) : z.y) / (angle ? fabs(tau) + sq : rr);
                    if (angle) {
                        const double c = 1.0 / sqrt(1.0 + t * t);
                        S.rotC[k] = c;
                        S.rotS[k] = t * c;
                    } else {
                        const bool valid = rr > 1e-300 && rr > 1e-16 * sq;
                        if (valid) atomicAdd(&S.nrot, 1);
                        S.rotP[k] = p;
                        S.rotQ[k] = qq;
                        S.rotV[k] = valid;
                        S.rotE[k] = make_double2(tau, t);
                    }
                }
                __syncwarp();
                if (!gdone)  // A <- U^H A U by 2x2 blocks (its columns, then its rows), V <- V U
                    for (int w = gl; w < 27; w += L) {
                        const int k2 = w % 3, p2 = S.rotP[k2], q2 = S.rotQ[k2], v2 = S.rotV[k2];
                        const double c2 = S.rotC[k2], s2 = S.rotS[k2];
                        const double2 eb = conj2(S.rotE[k2]);
                        if (w >= 9) {
                            if (!v2) continue;
                            double2* row = S.V + (w - 9) / 3 * n;
                            double2 x = row[p2], y = row[q2];
                            rot_col(c2, s2, eb, x, y);
                            row[p2] = x;
                            row[q2] = y;
                            continue;
                        }
                        const int k1 = w / 3, p1 = S.rotP[k1], q1 = S.rotQ[k1], v1 = S.rotV[k1];
                        double2 b00 = S.A[p1 * n + p2], b01 = S.A[p1 * n + q2];
                        double2 b10 = S.A[q1 * n + p2], b11 = S.A[q1 * n + q2];
                        if (v2) {
                            rot_col(c2, s2, eb, b00, b01);
                            rot_col(c2, s2, eb, b10, b11);
                        }
                        if (v1) {
                            const double c1 = S.rotC[k1], s1 = S.rotS[k1];
                            const double2 e = S.rotE[k1];
                            rot_row(c1, s1, e, b00, b10);
                            rot_row(c1, s1, e, b01, b11);
                            if (k1 == k2) {
                                b00.y = b11.y = 0.0;
                                b01 = b10 = make_double2(0.0, 0.0);
                            }
                        }
                        S.A[p1 * n + p2] = b00;
                        S.A[p1 * n + q2] = b01;
                        S.A[q1 * n + p2] = b10;
                        S.A[q1 * n + q2] = b11;
                    }
                __syncwarp();
            }
            if (!gdone && S.nrot == 0) gdone = true;  // nothing above the threshold: converged
            __syncwarp();
        }
        // --- ascending order (stable): rank of each eigenvalue
        if (act && gl < n) {
            const double li = S.A[gl * n + gl].x;
            int rk = 0;
            for (int j = 0; j < n; ++j) {
                const double lj = S.A[j * n + j].x;
                rk += (lj < li) || (lj == li && j < gl);
            }
            S.rank[gl] = rk;
            S.lam[rk] = li;
        }
        __syncwarp();
        if (act) {
            const int nq = P.nq;
            const bool gamma = fabs(qx) < CMP_PREC && fabs(qy) < CMP_PREC && fabs(qz) < CMP_PREC;
            for (int w = gl; w < 36; w += L) {
                const int col = w / n, row = w % n;
                P.evec[((size_t)q * n + S.rank[col]) * n + row] = S.V[row * n + col];
            }
            for (int w = gl; w < 3 * n; w += L) {
                const int k = w / n, col = w % n, s = S.rank[col];
                const double lv = S.A[col * n + col].x;
                double W = sqrt(fabs(lv));
                if (fabs(lv) > EPS_F32 && lv < 0.0) W = -W;
                const bool zero_mode = gamma && s < 3;
                double2 acc = make_double2(0.0, 0.0);
                for (int i = 0; i < n; ++i) {
                    double2 t = make_double2(0.0, 0.0);
                    for (int j = 0; j < n; ++j) t = cadd(t, cmul(S.dD[(k * n + i) * n + j], S.V[j * n + col]));
                    acc = cadd(acc, cmul(conj2(S.V[i * n + col]), t));
                }
                P.vel[((size_t)q * n + s) * 3 + k] = zero_mode ? 0.0 : acc.x / (2.0 * W) * a.vg_ms;
                if (k > 0) continue;
                P.omega[(size_t)q * n + s] = W * a.wTHz;
                P.oneby[(size_t)q * n + s] = zero_mode ? 0.0 : 1.0 / (W * a.wTHz);
                for (int t = 0; t < a.nT; ++t)
                    P.nbe[((size_t)t * nq + q) * n + s] =
                        zero_mode ? 0.0 : 1.0 / (exp(a.BEConv * fabs(W) / temps[t]) - 1.0);
            }
        }
        __syncwarp();
    }
}

// Points of the other half of the (q, -q) pairs: copies of their partner with conjugate
// eigenvectors and reversed velocities.
__global__ void k_phonons_tr(int n, int nT, int nq, const int* __restrict__ fill, const int* __restrict__ partner,
                             double2* __restrict__ evec, double* __restrict__ omega, double* __restrict__ oneby,
                             double* __restrict__ nbe, double* __restrict__ vel, int n_fill) {
    const int per = n * n + n * (3 + nT + 2);
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < (long long)n_fill * per;
         w += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(w / per), k = (int)(w % per);
        const int g = fill[i], p = partner[g];
        if (k < n * n) {
            const double2 e = evec[(size_t)p * n * n + k];
            evec[(size_t)g * n * n + k] = make_double2(e.x, -e.y);
        } else {
            const int r = k - n * n, s = r % n, what = r / n;  // 0..2 velocity, 3 omega, 4 1/omega, 5.. nBE
            if (what < 3) vel[((size_t)g * n + s) * 3 + what] = -vel[((size_t)p * n + s) * 3 + what];
            else if (what == 3) omega[(size_t)g * n + s] = omega[(size_t)p * n + s];
            else if (what == 4) oneby[(size_t)g * n + s] = oneby[(size_t)p * n + s];
            else {
                const int t = what - 5;
                nbe[((size_t)t * nq + g) * n + s] = nbe[((size_t)t * nq + p) * n + s];
            }
        }
    }
}

PhArgs ph_args(spring_ctx* c) {
    PhArgs a;
    a.nb = c->nb;
    a.n = c->ndof;
    a.na2 = c->na2;
    for (int i = 0; i < 9; ++i) a.latvec[i] = c->latvec[i];
    HostConst k = host_constants();
    a.wTHz = k.wTHz;
    a.vg_ms = k.vg_ms;
    a.BEConv = k.BEConv;
    a.nT = c->nT;
    a.dd = nullptr;
    return a;
}

size_t ph_smem(int n) {
    const int m = n + (n & 1);
    return sizeof(double2) * (2 * n * (n | 1) + 3 * n * n + m) + sizeof(double) * 3 * m + sizeof(int) * (3 * m + n) + 16;
}

int launch_phonons(spring_ctx* c, const PhSet& A, const int* list_a, int n_a, const PhSet& B, int n_b,
                   int gamma_mode = 0) {
    PhArgs a = ph_args(c);
    SPRING_CHECK(launch_ewald(c, A.qpts, A.nq, list_a, n_a, B.qpts, B.nq, n_b, gamma_mode, &a.dd));
    const int n = c->ndof;
    const size_t smem = ph_smem(n);
    const int items = n_a + n_b;
    if (items == 0) return SPRING_OK;
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "phonons: injected launch failure");
    if (n == 6 && a.nb == 2 && a.na2 <= PH6_NA2) {
#define SPRING_PH6(L)                                                                                              \
    k_phonons_n6<L><<<std::min((items + 32 / L - 1) / (32 / L), 148 * 13 * L / 8), 32, 0, c->stream>>>(              \
        a, A, list_a, n_a, B, n_b, c->d_fc2.p, c->d_fc2_idx.p, c->d_fc2_num.p, c->d_mass_rs.p, c->d_temps.p)
        // 32, 16, 8 lanes: 49, 58, 76 us up to 1000 points, 62, 65, 77 at 2200, 100, 81, 85 at 4300, 145, 124, 104
        // at 7300
        if (items <= 148 * 16) SPRING_PH6(32);
        else if (items <= 148 * 32) SPRING_PH6(16);
        else SPRING_PH6(8);
#undef SPRING_PH6
        return launch_check(c, "k_phonons_n6");
    }
    const int blocks = items < 148 * 32 ? items : 148 * 32;
    // the rotations' three warps and a thread per V update
    const int threads = std::min(PHT, 96 + (n * ((n + 1) / 2) + 31) / 32 * 32);
#define SPRING_PH(NN)                                                                                              \
    case NN:                                                                                                       \
        if (smem > 48 * 1024)                                                                                      \
            cudaFuncSetAttribute(k_phonons<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);           \
        k_phonons<NN><<<blocks, threads, smem, c->stream>>>(a, A, list_a, n_a, B, n_b, c->d_fc2.p, c->d_fc2_idx.p, \
                                                            c->d_fc2_num.p, c->d_mass_rs.p, c->d_temps.p);         \
        break
    switch (n) {
        SPRING_PH(3);
        SPRING_PH(6);
        SPRING_PH(9);
        SPRING_PH(12);
        SPRING_PH(15);
        SPRING_PH(18);
        SPRING_PH(21);
        SPRING_PH(24);
    }
#undef SPRING_PH
    return launch_check(c, "k_phonons");
}

PhSet ph_set(Phonons& ph, const double* q, int nq) {
    return PhSet{q, ph.evec.p, ph.omega.p, ph.oneby.p, ph.nbe.p, ph.vel.p, nq};
}

}  // namespace

int run_phonons(spring_ctx* c, Phonons& ph, const double* d_q, int nq, int gamma_mode) {
    const PhSet A = ph_set(ph, d_q, nq);
    return launch_phonons(c, A, nullptr, nq, A, 0, gamma_mode);
}

// Grid and irreducible phonons in one launch; on a Gamma-centred mesh only one point of each
// (q, -q) pair of the grid is solved and the other filled by time reversal.
int run_phonons_mesh(spring_ctx* c) {
    const int nq = c->nq;
    const PhSet G = ph_set(c->ph_grid, c->d_qpnt.p, nq), I = ph_set(c->ph_irr, c->d_irr_q.p, c->nq0);
    const bool tr = c->mesh_shift[0] == 0 && c->mesh_shift[1] == 0 && c->mesh_shift[2] == 0 &&
                    !(c->ew.on && c->ew.even);
    if (!tr) {
        SPRING_CHECK(launch_phonons(c, G, nullptr, nq, G, 0));
        return launch_phonons(c, I, nullptr, c->nq0, I, 0);
    }
    if (c->tr_nq != nq) {  // partner of every grid point and the two lists (built once per mesh)
        std::vector<int> partner(nq), solve, fill;
        for (int g = 0; g < nq; ++g) {
            const int x = g % c->mesh[0], y = (g / c->mesh[0]) % c->mesh[1], z = g / (c->mesh[0] * c->mesh[1]);
            const int xm = (c->mesh[0] - x) % c->mesh[0], ym = (c->mesh[1] - y) % c->mesh[1],
                      zm = (c->mesh[2] - z) % c->mesh[2];
            const int p = xm + c->mesh[0] * (ym + c->mesh[1] * zm);
            partner[g] = p;
            (g <= p ? solve : fill).push_back(g);
        }
        SPRING_CHECK(dalloc(c, c->d_tr_partner, nq, "time-reversal partners"));
        SPRING_CHECK(dalloc(c, c->d_tr_solve, std::max<size_t>(solve.size(), 1), "time-reversal lists"));
        SPRING_CHECK(dalloc(c, c->d_tr_fill, std::max<size_t>(fill.size(), 1), "time-reversal lists"));
        SPRING_CHECK(h2d(c, c->d_tr_partner.p, partner.data(), sizeof(int) * nq, "time-reversal partners"));
        SPRING_CHECK(h2d(c, c->d_tr_solve.p, solve.data(), sizeof(int) * solve.size(), "time-reversal lists"));
        SPRING_CHECK(h2d(c, c->d_tr_fill.p, fill.data(), sizeof(int) * fill.size(), "time-reversal lists"));
        c->tr_nsolve = (int)solve.size();
        c->tr_nfill = (int)fill.size();
        c->tr_nq = nq;
    }
    SPRING_CHECK(launch_phonons(c, G, c->d_tr_solve.p, c->tr_nsolve, I, c->nq0));
    if (c->tr_nfill == 0) return SPRING_OK;
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "phonons: injected launch failure");
    const int n = c->ndof;
    const long long work = (long long)c->tr_nfill * (n * n + n * (5 + c->nT));
    k_phonons_tr<<<(int)std::min<long long>((work + 255) / 256, 148LL * 16), 256, 0, c->stream>>>(
        n, c->nT, nq, c->d_tr_fill.p, c->d_tr_partner.p, G.evec, G.omega, G.oneby, G.nbe, G.vel, c->tr_nfill);
    return launch_check(c, "k_phonons_tr");
}

}  // namespace spring
