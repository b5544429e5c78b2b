// V3 -> W for cells with many branches: FP64 matrix instructions (mma.sync m8n8k4.f64, the only FP64 matrix
// form of sm_100).  Same quantity and epilogues as k_v3.cu (see there for the reference citations), another
// grouping of the sums.  Per pair (q0, q1, q2):
//   D_mu[a][nu b][eta c]  as in k_v3.cu, kept only for the basis types nu, eta among mu's neighbours
//   T1_mu[a][nu b][s2]  = sum_{eta c} D_mu[a][nu b][eta c] e2(eta c, s2)
//   H[s0][nu b][s2]     = sum_{mu a}  m_mu^-1/2 e0(mu a, s0) T1_mu[a][nu b][s2]   (mu with nu among its types)
//   Phi[s0][s1][s2]     = sum_{nu b}  e1(nu b, s1) H[s0][nu b][s2]
// Contracting e0 before e1 leaves a last step that is complete per s0, so a block of eight s0 needs only its
// own H in shared memory and no Phi accumulator outlives a step; nothing is computed twice.  In the 8-atom
// rocksalt cell an atom has four neighbour types of eight: 4.7 Mflop per pair, where the kernel in k_v3.cu
// does 24 Mflop (all types, and T1 and T2 again for every block of six s0) from shared memory at three
// complex products per load.
// One CTA of 12 warps per SM: T1 of every mu, one H block, e0 and e1 fill the 227 KB.  Complex products are
// four real ones.  Row strides are 4 (A operands) or 2 (B operands) complex modulo 8, so a fragment's 8 x 4
// lanes read distinct banks.
// Gaussian epilogue: W of the block goes to shared memory; warps screen (s1, s2, channel) of one s0 against
// the underflow point of exp and evaluate 32 hits at a time, one accumulator per temperature.
// 8-atom cell: 6^3, nine temperatures 12.7 -> 0.85 ms, 8^3, three 52.1 -> 3.1 ms (14 TFLOP/s); W grids of
// 6^3 12.6 -> 0.75 ms.  Bound: of the 100k cycles a pair takes, 37k are the FP64 tensor pipe (9216 m8n8k4;
// Phi, H and T1 take 23k, 16k and 9k), 31k the latency of the Gaussian epilogue and 15k that of the inputs
// and D, which three warps per scheduler do not hide.
#include <algorithm>

#include "v3item.cuh"
#include "tetra.cuh"

namespace spring {
namespace {

constexpr int MW = 12, MT_ = 9;  // warps per CTA; temperatures per epilogue pass
constexpr int QCAP = 576;        // hits of one epilogue unit: 8 x 24 (s1, s2), three channels

// Shared-memory layout (in double2 unless noted) and sizes of one launch.
struct V3mLayout {
    int KT;            // rows of T1 per (mu, a): 3 x most neighbour types of an atom, padded to 4
    int RS, S2, DS;    // row strides: e0 / e1, e2 / T1 / H, D
    int TB, HS;        // strides of a T1 block (mu, a) and of one s0 of H
    int NR;            // H rows: n padded to 4
    int GM;            // mu per D group
    int oE1, oT1, oX;  // e0 at 0; X: H and W, or e2 | phases | phase products | D
    int oPh, oPP, oD;  // within X
    int oQ;            // hit queues, within X behind W
    int oI;            // byte offset of the scalars and tables
    int bytes;
};

__device__ __forceinline__ void dmma(double* c, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// c (re, im pairs of one 8 x 8 tile) += a b, complex, K = 4
__device__ __forceinline__ void cmma(double (*c)[2], double2 a, double2 b) {
    dmma(c[0], a.x, b.x);
    dmma(c[1], a.x, b.y);
    dmma(c[0], -a.y, b.y);
    dmma(c[1], a.y, b.x);
}
__device__ __forceinline__ void put2(double2* o, const double (*c)[2]) {
    o[0] = make_double2(c[0][0], c[1][0]);
    o[1] = make_double2(c[0][1], c[1][1]);
}

// NT: 8-wide tiles of the branches (n <= 8 NT).
template <int NT, int EPI>
__global__ void __launch_bounds__(32 * MW, 1) k_v3m(V3Args a_, V3mLayout L, V3Ptrs P, const int* __restrict__ off,
                                                    const int* __restrict__ range, int n_q0, int cap, int npairs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V3Args a = a_;
    const int n = a.n, na = a.na, nb = a.nb, NP = 8 * NT;
    double2* sm = reinterpret_cast<double2*>(smem_raw);
    double2 *sE0 = sm, *sE1 = sm + L.oE1, *sT1 = sm + L.oT1, *sX = sm + L.oX;
    double2 *sE2 = sX, *sPh = sX + L.oPh, *sPP = sX + L.oPP, *sD = sX + L.oD, *sH = sX;
    double* sW = reinterpret_cast<double*>(sX);           // [8][n][n + 1]
    double* sc = reinterpret_cast<double*>(smem_raw + L.oI);  // w0, w1, w2, 1/w0, 1/w1, 1/w2: [6][24]
    double* sN = sc + 6 * MAX_NDOF;                       // n(T) of q1 and q2: [2][MT_][24]
    int* sTy = reinterpret_cast<int*>(sN + 2 * MT_ * MAX_NDOF);  // [mu][8] neighbour types
    int* sNt = sTy + MAX_NB * MAX_NB;                     // [mu] their number
    int* sKh = sNt + MAX_NB;                              // [nu] rows (mu, a) of H's sum, a multiple of 4
    int* sKo = sKh + MAX_NB;                              // [nu][24] T1 offset of row (mu, a), nu b = 0
    int* sKr = sKo + MAX_NB * MAX_NDOF;                   // [nu][24] row of e0 (n: a zero column)
    int* sKe = sKr + MAX_NB * MAX_NDOF;                   // [mu][24] e2 offset of D's columns (0 beyond them: D is zero)
    unsigned short* sQ = reinterpret_cast<unsigned short*>(sX + L.oQ);  // [MW][QCAP] hit queues, behind W
    int* sSl = sKe + MAX_NB * MAX_NDOF;                   // [mu][8] first slot | slots << 8 of each type
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    constexpr int TH = 32 * MW;

    if (tid < nb) {  // the types of mu = tid
        int cnt = 0;
        for (int nu = 0; nu < nb; ++nu)
            if (off[tid * (nb + 1) + nu + 1] > off[tid * (nb + 1) + nu]) {
                sSl[tid * MAX_NB + cnt] = off[tid * (nb + 1) + nu] | (off[tid * (nb + 1) + nu + 1] - off[tid * (nb + 1) + nu]) << 8;
                sTy[tid * MAX_NB + cnt++] = nu;
            }
        sNt[tid] = cnt;
        for (int k = 0; k < MAX_NDOF; ++k)
            sKe[tid * MAX_NDOF + k] = k < 3 * cnt ? (3 * sTy[tid * MAX_NB + k / 3] + k % 3) * L.S2 : 0;
    }
    __syncthreads();
    if (tid < nb) {  // the mu that have type nu = tid
        int k = 0;
        for (int mu = 0; mu < nb; ++mu)
            for (int p = 0; p < sNt[mu]; ++p)
                if (sTy[mu * MAX_NB + p] == tid)
                    for (int al = 0; al < 3; ++al, ++k) {
                        sKo[tid * MAX_NDOF + k] = (mu * 3 + al) * L.TB + 3 * p * L.S2;
                        sKr[tid * MAX_NDOF + k] = 3 * mu + al;
                    }
        for (; k & 3; ++k) {  // times zero: any block of T1 that is written (the first is not where atom 0 has no slots)
            sKo[tid * MAX_NDOF + k] = sKo[tid * MAX_NDOF + k - 1];
            sKr[tid * MAX_NDOF + k] = n;
        }
        sKh[tid] = k;
    }
    int first = a.pair_first, count = npairs;
    if (range) {
        first = min(range[0], cap);
        count = min(range[n_q0], cap) - first;
    }
    for (int it = blockIdx.x; it < count; it += gridDim.x) {
        const int pr = first + it;
        const int2 pq = P.pairs[pr];
        const int g1 = pq.x, g2 = pq.y, q0 = P.pair_q0[pr], p0 = P.q0_grid ? P.q0_grid[q0] : q0;
        __syncthreads();  // the previous pair's epilogue is done
        // eigenvectors (zero beyond n), scalars, neighbour phases
        for (int i = tid; i < NP * L.RS; i += TH) {
            const int s = i / L.RS, row = i % L.RS;
            double2 x = make_double2(0.0, 0.0), y = x;
            if (s < n && row < n) {
                x = P.ev0[((size_t)p0 * n + s) * n + row];
                const double m = P.mrs[row / 3];
                x.x *= m;
                x.y *= m;
                y = P.evg[((size_t)g1 * n + s) * n + row];
            }
            sE0[i] = x;
            sE1[i] = y;
        }
        for (int i = tid; i < NP * n; i += TH) {
            const int s = i / n, row = i % n;
            sE2[row * L.S2 + s] = s < n ? P.evg[((size_t)g2 * n + s) * n + row] : make_double2(0.0, 0.0);
        }
        for (int i = tid; i < 6 * n; i += TH) {
            const int w = i / n, s = i % n;
            const double* src = w == 0 ? P.om0 : (w == 3 ? P.ob0 : (w < 3 ? P.omg : P.obg));
            sc[w * MAX_NDOF + s] = src[(size_t)(w % 3 == 0 ? p0 : (w % 3 == 1 ? g1 : g2)) * n + s];
        }
        if (EPI == 0 && a.nT <= MT_)
            for (int i = tid; i < 2 * a.nT * n; i += TH) {
                const int s = i % n, t = i / n % a.nT, w = i / (n * a.nT);
                sN[(w * MT_ + t) * MAX_NDOF + s] = P.nbeg[((size_t)t * a.nq + (w ? g2 : g1)) * n + s];
            }
        for (int i = tid; i < nb * 2 * na; i += TH) {
            const int N = i % na, w = i / na % 2, mu = i / (2 * na), g = w ? g2 : g1;
            const double* Rv = P.posr + ((size_t)mu * na + N) * 3;
            const double qr = P.qpnt[3 * g] * Rv[0] + P.qpnt[3 * g + 1] * Rv[1] + P.qpnt[3 * g + 2] * Rv[2];
            double sn, cs;
            sincos(qr, &sn, &cs);
            sPh[i] = make_double2(cs, sn);
        }
        __syncthreads();
        for (int mg = 0; mg < nb; mg += L.GM) {
            const int gm = min(L.GM, nb - mg);
            for (int i = tid; i < gm * na * na; i += TH) {
                const int N2 = i % na, N1 = i / na % na, mu = mg + i / (na * na);
                const double2 p1 = sPh[(2 * mu) * na + N1], p2 = sPh[(2 * mu + 1) * na + N2];
                const double m = P.mrs[P.btyp[mu * na + N1]] * P.mrs[P.btyp[mu * na + N2]];
                sPP[i] = make_double2(m * (p1.x * p2.x - p1.y * p2.y), m * (p1.x * p2.y + p1.y * p2.x));
            }
            __syncthreads();
            // D: one thread per (mu, a, row, eta), three columns each (their FC3 values are adjacent); the
            // terms are independent loads
            const int kt = L.KT / 3 + (L.KT % 3 != 0);  // column triples, the last possibly cut
            for (int i = tid; i < gm * 3 * L.KT * kt; i += TH) {
                const int kp = i % kt, j = i / kt, r = j % L.KT, ma = j / L.KT, ml = ma / 3, mu = mg + ml;
                double2 acc[3];
#pragma unroll
                for (int g = 0; g < 3; ++g) acc[g] = make_double2(0.0, 0.0);
                if (r < 3 * sNt[mu] && kp < sNt[mu]) {
                    const int l1 = sSl[mu * MAX_NB + r / 3], l2 = sSl[mu * MAX_NB + kp];
                    const int a1 = l1 & 255, a2 = l2 & 255, c1 = l1 >> 8, cnt = c1 * (l2 >> 8);
                    const double* f = P.fc3 + (size_t)mu * na * na * 27 + (ma % 3 * 3 + r % 3) * 3;
#pragma unroll 4
                    for (int t = 0, N1 = a1, N2 = a2; t < cnt; ++t) {
                        const double* fv = f + (N1 * na + N2) * 27;
                        const double2 pp = sPP[(ml * na + N1) * na + N2];
#pragma unroll
                        for (int g = 0; g < 3; ++g) {
                            acc[g].x = fma(fv[g], pp.x, acc[g].x);
                            acc[g].y = fma(fv[g], pp.y, acc[g].y);
                        }
                        if (++N1 == a1 + c1) {
                            N1 = a1;
                            ++N2;
                        }
                    }
                }
#pragma unroll
                for (int g = 0; g < 3; ++g)
                    if (3 * kp + g < L.KT) sD[j * L.DS + 3 * kp + g] = acc[g];
            }
            __syncthreads();
            // T1 of (mu, a): one warp each
            for (int u = warp; u < gm * 3; u += MW) {
                const int mu = mg + u / 3, K = 3 * sNt[mu];
                const double2* D = sD + u * L.KT * L.DS;
                double2* T1 = sT1 + (mu * 3 + u % 3) * L.TB;
                for (int mt = 0; mt * 8 < K; ++mt) {
                    const double2* A = D + min(mt * 8 + lr, L.KT - 1) * L.DS + lc;
                    double c[NT][2][2];
#pragma unroll
                    for (int t = 0; t < NT; ++t) c[t][0][0] = c[t][0][1] = c[t][1][0] = c[t][1][1] = 0.0;
                    for (int k0 = 0; k0 < K; k0 += 4) {
                        const double2 av = A[k0];
                        const double2* B = sE2 + sKe[mu * MAX_NDOF + k0 + lc] + lr;
#pragma unroll
                        for (int t = 0; t < NT; ++t) cmma(c[t], av, B[8 * t]);
                    }
                    if (mt * 8 + lr < L.KT)
#pragma unroll
                        for (int t = 0; t < NT; ++t) put2(T1 + (mt * 8 + lr) * L.S2 + 8 * t + 2 * lc, c[t]);
                }
            }
            __syncthreads();
        }
        const bool gq0 = P.irr_int[3 * q0] == 0 && P.irr_int[3 * q0 + 1] == 0 && P.irr_int[3 * q0 + 2] == 0;
        const bool gq1 = g1 == 0, gq2 = g2 == 0;
        for (int sb = 0; sb < n; sb += 8) {
            // H of s0 = sb .. sb + 7
            for (int r = warp; r < L.NR; r += MW) {
                double c[NT][2][2];
#pragma unroll
                for (int t = 0; t < NT; ++t) c[t][0][0] = c[t][0][1] = c[t][1][0] = c[t][1][1] = 0.0;
                if (r < n) {
                    const int nu = r / 3, K = sKh[nu];
                    const double2* A = sE0 + (sb + lr) * L.RS;
                    const double2* B = sT1 + (r % 3) * L.S2 + lr;
                    for (int k0 = 0; k0 < K; k0 += 4) {
                        const double2 av = A[sKr[nu * MAX_NDOF + k0 + lc]];
                        const double2* Bk = B + sKo[nu * MAX_NDOF + k0 + lc];
#pragma unroll
                        for (int t = 0; t < NT; ++t) cmma(c[t], av, Bk[8 * t]);
                    }
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) put2(sH + lr * L.HS + r * L.S2 + 8 * t + 2 * lc, c[t]);
            }
            __syncthreads();
            // Phi of (s0, eight s1): up to two units per warp, written once every warp has read its H
            double c[2][NT][2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int u = warp + h * MW, s0l = u & 7, mt = u >> 3;
#pragma unroll
                for (int t = 0; t < NT; ++t) c[h][t][0][0] = c[h][t][0][1] = c[h][t][1][0] = c[h][t][1][1] = 0.0;
                if (u >= 8 * NT || sb + s0l >= n) continue;
                const double2* A = sE1 + (mt * 8 + lr) * L.RS + lc;
                const double2* B = sH + s0l * L.HS + lc * L.S2 + lr;
                for (int k0 = 0; k0 < L.NR; k0 += 4) {
                    const double2 av = A[k0];
#pragma unroll
                    for (int t = 0; t < NT; ++t) cmma(c[h][t], av, B[k0 * L.S2 + 8 * t]);
                }
            }
            __syncthreads();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int u = warp + h * MW, s0l = u & 7, s0 = sb + s0l, s1 = (u >> 3) * 8 + lr;
                if (u >= 8 * NT || s0 >= n || s1 >= n) continue;
                const double o01 = sc[3 * MAX_NDOF + s0] * sc[4 * MAX_NDOF + s1];
#pragma unroll
                for (int t = 0; t < NT; ++t)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int s2 = 8 * t + 2 * lc + j;
                        if (s2 >= n) continue;
                        const bool zero = (gq0 && s0 < 3) || (gq1 && s1 < 3) || (gq2 && s2 < 3);
                        const double re = c[h][t][0][j], im = c[h][t][1][j];
                        sW[(s0l * n + s1) * (n + 1) + s2] =
                            zero ? 0.0 : (re * re + im * im) * (o01 * sc[5 * MAX_NDOF + s2]) * a.mfac;
                    }
            }
            __syncthreads();
            if (EPI == 1) {
                const size_t n3 = (size_t)n * n * n;
                const int slot = q0 - a.q0_first, len = min(8, n - sb) * n * n;
                double* w1 = P.out_w + ((size_t)slot * a.nq + g1) * n3 + (size_t)sb * n * n;
                for (int i = tid; i < len; i += TH) w1[i] = sW[i / n * (n + 1) + i % n];
                if (g1 != g2) {
                    double* w2 = P.out_w + ((size_t)slot * a.nq + g2) * n3 + (size_t)sb * n * n;
                    for (int i = tid; i < len; i += TH)
                        w2[i] = sW[(i / (n * n) * n + i % n) * (n + 1) + i / n % n];
                }
            } else {
                const double pre = a.onebysigma * ONEBYSQRT2PI, mult = g1 != g2 ? 2.0 : 1.0;
                unsigned short* queue = sQ + warp * QCAP;
                for (int t0 = 0; t0 < a.nT; t0 += MT_) {
                    const int nt = min(MT_, a.nT - t0);
                    if (a.nT > MT_) {
                        __syncthreads();
                        for (int i = tid; i < 2 * nt * n; i += TH) {
                            const int s = i % n, t = i / n % nt, w = i / (n * nt);
                            sN[(w * MT_ + t) * MAX_NDOF + s] = P.nbeg[((size_t)(t0 + t) * a.nq + (w ? g2 : g1)) * n + s];
                        }
                        __syncthreads();
                    }
                    // (s0, a third of the s1): two units per warp at 24 branches; a step takes rp rows of s1
                    const int rp = 32 / n, lrow = lane / n, s2 = lane % n;
                    const bool lane_on = lrow < rp && s2 >= a.pol_lo[2] && s2 <= a.pol_hi[2] && !(gq2 && s2 < 3);
                    const double w2 = sc[2 * MAX_NDOF + s2];
                    for (int u = warp; u < 24; u += MW) {
                        const int s0l = u & 7, s0 = sb + s0l;
                        if (s0 >= n || s0 < a.pol_lo[0] || s0 > a.pol_hi[0]) continue;
                        const double w0 = sc[s0];
                        const int step = (n + 2) / 3, i0 = (u >> 3) * step, i1 = min(i0 + step, n);
                        double acc[MT_], accp = 0.0;
#pragma unroll
                        for (int t = 0; t < MT_; ++t) acc[t] = 0.0;
                        int qn = 0;
#pragma unroll 4
                        for (int ib = i0; ib < i1; ib += rp) {
                            const int s1 = ib + lrow;
                            unsigned in = 0;
                            if (lane_on && s1 < i1 && s1 >= a.pol_lo[1] && s1 <= a.pol_hi[1] && !(gq1 && s1 < 3)) {
                                const double w1 = sc[MAX_NDOF + s1];
                                const double d1 = w0 - w1 - w2, d2 = w0 + w1 - w2, d3 = w0 - w1 + w2;
                                in = (0.5 * a.onebysigma2 * (d1 * d1) < EXP_UNDERFLOW ? 1 : 0) |
                                     (0.5 * a.onebysigma2 * (d2 * d2) < EXP_UNDERFLOW ? 2 : 0) |
                                     (0.5 * a.onebysigma2 * (d3 * d3) < EXP_UNDERFLOW ? 4 : 0);
                            }
                            const unsigned code = s1 | s2 << 5, lt = (1u << lane) - 1;
#pragma unroll
                            for (int ch = 0; ch < 3; ++ch) {
                                const unsigned m = __ballot_sync(0xffffffffu, in >> ch & 1);
                                if (in >> ch & 1) queue[qn + __popc(m & lt)] = code | ch << 10;
                                qn += __popc(m);
                            }
                        }
                        __syncwarp();
                        // two hits per lane at a time: their exponentials overlap
                        for (int i = lane; i < qn; i += 64) {
                            double v[2];
                            const double *n1[2], *n2[2];
                            bool sum[2];
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const bool have = i + 32 * h < qn;
                                const unsigned code = have ? queue[i + 32 * h] : 0;
                                const int t1 = code & 31, t2 = code >> 5 & 31, ch = code >> 10;
                                const double v1 = sc[MAX_NDOF + t1], v2 = sc[2 * MAX_NDOF + t2];
                                const double d = ch == 0 ? w0 - v1 - v2 : (ch == 1 ? w0 + v1 - v2 : w0 - v1 + v2);
                                const double e = have ? pre * exp(-(0.5 * a.onebysigma2 * (d * d))) : 0.0;
                                accp += e;
                                v[h] = sW[(s0l * n + t1) * (n + 1) + t2] * (ch == 2 ? -e : e);
                                if (!have) v[h] = 0.0;
                                n1[h] = sN + t1;
                                n2[h] = sN + MT_ * MAX_NDOF + t2;
                                sum[h] = ch == 0;
                            }
#pragma unroll
                            for (int t = 0; t < MT_; ++t) {
                                if (t >= nt) break;
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const double x = n1[h][t * MAX_NDOF], y = n2[h][t * MAX_NDOF];
                                    acc[t] = fma(v[h], sum[h] ? x + y + 1.0 : x - y, acc[t]);
                                }
                            }
                        }
                        __syncwarp();
                        // the sums of three temperatures and the phase space run side by side
#pragma unroll
                        for (int t = 0; t < MT_; t += 3) {
                            if (t >= nt) break;
                            double x[4] = {acc[t], acc[t + 1], acc[t + 2], accp};
                            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                                for (int h = 0; h < 4; ++h) x[h] += __shfl_down_sync(0xffffffffu, x[h], o);
                            if (lane != 0) continue;
#pragma unroll
                            for (int h = 0; h < 3; ++h)
                                if (t + h < nt && x[h] != 0.0)
                                    atomicAdd(&P.out_lw[((size_t)(t0 + t + h) * a.nq0 + q0) * n + s0], mult * x[h]);
                            if (t == 0 && t0 == 0 && x[3] != 0.0) atomicAdd(&P.out_p3[(size_t)q0 * n + s0], mult * x[3]);
                        }
                    }
                }
            }
            __syncthreads();  // W has been read: H of the next block takes its place
        }
    }
}

// The layout for a cell of n branches, na slots and at most `types` neighbour types per atom; bytes is above
// the limit of a CTA when it does not fit.
V3mLayout v3m_layout(int nb, int n, int na, int types) {
    auto up = [](int x, int m, int r) { return x + ((r - x) % m + m) % m; };  // least y >= x with y = r mod m
    V3mLayout L{};
    const int NP = (n + 7) / 8 * 8;
    L.KT = (3 * types + 3) / 4 * 4;
    L.NR = (n + 3) / 4 * 4;
    L.RS = up(std::max(n + 1, L.NR), 8, 4);
    L.S2 = NP + 2;
    L.DS = up(L.KT, 8, 4);
    L.TB = up(L.KT * L.S2, 8, 2);
    L.HS = up(L.NR * L.S2, 8, 1);
    L.oE1 = NP * L.RS;
    L.oT1 = 2 * NP * L.RS;
    L.oX = L.oT1 + nb * 3 * L.TB;
    L.oPh = n * L.S2;
    L.oPP = L.oPh + nb * 2 * na;
    L.oQ = (8 * n * (n + 1) + 1) / 2;
    const int h = std::max(8 * L.HS, L.oQ + MW * QCAP * (int)sizeof(unsigned short) / (int)sizeof(double2));
    const auto x_of = [&](int gm) { return L.oPP + gm * na * na + gm * 3 * L.KT * L.DS; };
    L.GM = nb;  // as many mu per group as H's place holds, at least one
    while (L.GM > 1 && x_of(L.GM) > h) --L.GM;
    L.oD = L.oPP + L.GM * na * na;
    L.oI = (L.oX + std::max(h, x_of(L.GM))) * (int)sizeof(double2);
    L.bytes = L.oI + (6 + 2 * MT_) * MAX_NDOF * (int)sizeof(double) +
              (2 * MAX_NB * MAX_NB + 2 * MAX_NB + 3 * MAX_NB * MAX_NDOF) * (int)sizeof(int);
    return L;
}

}  // namespace

// Whether launch_v3m takes the context's cell.  Fewer branches leave the 8-wide tiles half empty and a step
// too short for its barriers: at 3 to 9 branches the kernel in k_v3.cu takes 0.24 - 0.33 ms where this one
// takes 0.50 - 1.3; from 12 on this one is ahead (12: 0.93 -> 0.50 ms, 15: 3.0 -> 0.36, 18: 2.2 -> 0.40,
// 24: 10.1 -> 0.55; W grids of 16 q0).  SPRING_OPT_GENERIC_V3 leaves every cell to k_v3.cu.
bool v3m_takes(const spring_ctx* c) {
    return !c->force_generic_v3 && c->ndof >= 12 && v3m_layout(c->nb, c->ndof, c->na3, c->fc3_types).bytes <= 227 * 1024;
}

// Launch for pair set ps, q0 block [q0_first, +n_q0); *handled is false when the layout does not fit.
int launch_v3m(spring_ctx* c, const PairSet& ps, const Q0View& v, int q0_first, int n_q0, int epi, double sigma,
               const Pol* pol, double* lw, double* p3, double* w, bool* handled) {
    *handled = false;
    if (!v3m_takes(c)) return SPRING_OK;
    const V3mLayout L = v3m_layout(c->nb, c->ndof, c->na3, c->fc3_types);
    *handled = true;
    V3Args a{};
    a.nb = c->nb;
    a.n = c->ndof;
    a.na = c->na3;
    a.nq = c->nq;
    a.nq0 = ps.n0;
    a.nT = c->nT;
    a.q0_first = q0_first;
    a.mfac = host_constants().Sctr3THz2 / double(c->nq);
    if (epi == 0) {
        a.onebysigma = 1.0 / sigma;
        a.onebysigma2 = a.onebysigma * a.onebysigma;
        for (int k = 0; k < 3; ++k) {
            a.pol_lo[k] = pol->lo[k];
            a.pol_hi[k] = pol->hi[k];
        }
    }
    // as launch_v3: the pair range from the host's offsets, or read on the device
    const int* range = nullptr;
    long long npairs;
    if (ps.h_ok) {
        a.pair_first = ps.h_pairoff[q0_first];
        npairs = ps.h_pairoff[q0_first + n_q0] - a.pair_first;
    } else {
        range = ps.pairoff.p + q0_first;
        npairs = std::min<long long>((long long)n_q0 * (c->nq / 2 + 8), ps.cap);
    }
    if (npairs == 0) return SPRING_OK;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    const int resident = std::max(1, 227 * 1024 / (L.bytes + 1024));
    const int grid = (int)std::min<long long>(npairs, (long long)sms * resident);
    const V3Ptrs P{ps.pairs.p, ps.pair_q0.p, c->d_fc3.p, c->d_fc3_posr.p, c->d_fc3_btyp.p, c->d_mass_rs.p,
                   c->d_qpnt.p, v.q0_int, v.q0_grid, v.evec, v.omega, v.oneby, c->ph_grid.evec.p,
                   c->ph_grid.omega.p, c->ph_grid.oneby.p, c->ph_grid.nbe.p, lw, p3, w};
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "v3: injected launch failure");
#define SPRING_V3M(NT, EPI)                                                                                    \
    do {                                                                                                       \
        allow_smem(k_v3m<NT, EPI>);                                                                            \
        k_v3m<NT, EPI><<<grid, 32 * MW, L.bytes, c->stream>>>(a, L, P, c->d_fc3_off.p, range, n_q0, ps.cap,    \
                                                              (int)npairs);                                    \
    } while (0)
    const int nt = (c->ndof + 7) / 8;  // 2 or 3: at least 12 branches
    if (epi == 0) {
        if (nt == 2) SPRING_V3M(2, 0);
        else SPRING_V3M(3, 0);
    } else {
        if (nt == 2) SPRING_V3M(2, 1);
        else SPRING_V3M(3, 1);
    }
#undef SPRING_V3M
    return launch_check(c, epi == 0 ? "k_v3<gauss>" : "k_v3<wgrid>");
}

}  // namespace spring
