// V3 -> W for two-atom cells (Ndof = 6) with 7-slot neighbour clusters: the shapes of the rocksalt benchmark
// crystal, on the FP64 matrix instructions (mma.sync m8n8k4.f64).  Same mathematics and epilogues as k_v3.cu
// (see there for the reference citations).
//
// Two warps take four pairs at a time through every step; they meet at one barrier of their own, eight such
// teams per SM.
//   fold   D[eta c][mu a, nu b] of the four pairs: FC3 (27 abc rows of one mu, constant in shared memory)
//          times the phase products (four pairs x re/im = 8 columns), K the slot pairs of one basis block;
//          one mu per warp
//   T1     T1[s2][mu a, nu b]  = e2 D,  T2[s1][mu a, s2] = e1 T1,  Phi[s0][s1, s2] = e0' T2, pair by pair,
//          two pairs per warp
// Each contraction is one 8 x 72 real product with K = 12: complex numbers enter as
//   [Ar | Ai] [[Br, Bi], [-Bi, Br]],
// so the six rows fill 6 of 8, the 36 complex columns 9 tiles exactly and K three steps exactly; a lane ends up
// with whole complex numbers.  Results overwrite their input in place (a row stride of 38 complex keeps the
// 8 x 4 lanes of a fragment on distinct banks); e0, e1 and e2 go from global memory straight into fragments.
// Gaussian epilogue: W replaces Phi in shared memory; every (s1, s2, channel) is screened in FP32 against the
// underflow point of exp, hits are queued per s0, and the warp evaluates one s0 at a time, two hits per lane.
// 109 m8n8k4 per pair (436 cycles of an SM's FP64 pipe; the 20.8 k FMA of the pair are 325).  The former kernel
// (8 pairs per 288-thread CTA, FMA from shared memory) spent 2500 cycles a pair, this one 1150 (Gaussian) and
// 1000 (W grids): 24^3, three temperatures 25.4 -> 11.7 ms, 20^3, nine 10.3 -> 5.25 ms; W grids of 16^3 2.6 ->
// 1.13 ms; 630 pairs (5^3) 24 -> 26 us and 24 -> 18 us.  What is left beside the FP64 pipe is the latency of the
// loads and of the evaluations with four warps per scheduler.
#include <algorithm>

#include "v3s.cuh"

namespace spring {
namespace {

using namespace s3;

constexpr int TEAMS = 8;           // teams of two warps per CTA (one CTA per SM)
constexpr int GP = 4, WP = 2;      // pairs per group, per warp
constexpr int ST = 38, DP = 6 * ST;  // row stride and size of a pair's D / T1 / T2, complex
constexpr int KMAX = 64, FS = 36;  // slot pairs of one mu, each basis block padded to 4; row stride of FC3
constexpr int QC = WP * 108;       // queue entries of one s0: 36 (s1, s2) x 3 channels per pair
constexpr double EXP_UNDERFLOW = 745.2;

struct S3Args {
    int nq, nT, nq0, q0_first, pair_first, pair_end;
    const int* plist;  // null: pairs pair_first .. pair_end - 1; else the pairs plist[pair_first .. pair_end - 1]
    double mfac, onebysigma, onebysigma2;
    int pol_lo[3], pol_hi[3];
};

// Inputs and outputs of one launch.
struct S3Ptrs {
    const int2* pairs;
    const int* pair_q0;
    const double* fc3;
    const double* posr;
    const int* off;
    const double* mrs;
    const double* qpnt;
    const int* q0_int;
    const int* q0_grid;
    const double2* ev0;
    const double* om0;
    const double* ob0;
    const double2* evg;
    const double* omg;
    const double* obg;
    const double* nbeg;
    double* out_lw;
    double* out_p3;
    double* out_w;
    // EPI 2 (the Gaussian BTE operator): entries appended at *item_ctr (those past item_cap are
    // counted, not written)
    void* out_items;
    unsigned long long* item_ctr;
    long long item_cap;
};

struct TeamMem {
    double2 D[GP][DP];  // D, T1, T2; then W (216 doubles [s0][s1][s2]) and n (doubles [leg][s][T]) of the pair
    union {
        double2 ph[GP][2][NB * NA];            // neighbour phases [pair][leg][mu][N], until the fold is done
        unsigned short queue[2][N][QC];        // hits by warp and s0
    };
    double w[GP][3][N], ob[GP][3][N];
    float wf[GP][3][N];
    int g1[GP], g2[GP], q0[GP], p0[GP], gam[GP];  // gam: bits q0, q1, q2 is Gamma; -1 beyond the last pair
};
static_assert(sizeof(double2) * DP >= sizeof(double) * (216 + 2 * N * MAXT), "W and n fit a pair's place");

struct Smem {
    double fc[NB][KMAX][FS];       // FC3 times its neighbour masses [k][abc], zero on padding
    TeamMem tm[TEAMS];
    double posr[NB * NA * 3], mrs[NB];
    int ksrc[NB][KMAX];            // N1 | N2 << 8 of row k (0 on padding)
    int kb[NB][NB * NB + 1];       // first row of each (nu, eta) block
    int off[NB * (NB + 1)];        // first slot of each basis atom
};

__device__ __forceinline__ void team_sync(int team) { asm volatile("bar.sync %0, 64;" ::"r"(team + 1) : "memory"); }

__device__ __forceinline__ void dmma(double* c, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// c[t] = (row lane / 4, complex column 4 t + lane % 4) of the 6 x 36 product of A (three K steps in a lane's
// fragments) and the 6 x 36 complex matrix at B.
__device__ __forceinline__ void product(double (*c)[2], const double* A, const double2* B, const int* boff,
                                        const unsigned* neg) {
    const double* b = reinterpret_cast<const double*>(B);
#pragma unroll
    for (int t = 0; t < 9; ++t) c[t][0] = c[t][1] = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const double v = b[boff[k] + 8 * t];
            dmma(c[t], A[k], __hiloint2double(__double2hiint(v) ^ (int)neg[k], __double2loint(v)));
        }
}

// A fragment of a 6 x 6 eigenvector block e[s][row]: row of the product s, K = (row, re / im).
__device__ __forceinline__ void efrag(double* A, const double2* __restrict__ e, int lr, int lc) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int kk = 4 * k + lc, im = kk >= 6, row = kk - 6 * im;
        A[k] = lr < 6 ? reinterpret_cast<const double*>(e)[(lr * 6 + row) * 2 + im] : 0.0;
    }
}

// range != null: the pair range is read on the device, pairs range[0] .. range[n_q0] (the pair
// offsets of the enumeration, clamped to the list's capacity), instead of a.pair_first/pair_end.
// EPI 0: Gaussian sums of up to NT temperatures; 1: W grids; 2: operator entries.
template <int EPI, int NT>
__global__ void __launch_bounds__(64 * TEAMS, 1) k_v3s(S3Args a_, S3Ptrs P, const int* __restrict__ range, int n_q0, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    S3Args a = a_;
    constexpr int TH = 64 * TEAMS;
    const int tid = threadIdx.x, lane = tid & 31, half = tid >> 5 & 1, team = tid >> 6, t64 = tid & 63;
    const int lr = lane >> 2, lc = lane & 3;
    TeamMem& M = S.tm[team];
    if (range) {
        a.pair_first = min(range[0], cap);
        a.pair_end = min(range[n_q0], cap);
    }
    // the cell: slot pairs (N1, N2) of each basis block as rows k, each block padded to four
    for (int i = tid; i < NB * KMAX * FS; i += TH) (&S.fc[0][0][0])[i] = 0.0;
    for (int i = tid; i < NB * KMAX; i += TH) (&S.ksrc[0][0])[i] = 0;
    for (int i = tid; i < NB * NA * 3; i += TH) S.posr[i] = P.posr[i];
    if (tid < NB * (NB + 1)) S.off[tid] = P.off[tid];
    if (tid < NB) S.mrs[tid] = P.mrs[tid];
    __syncthreads();
    if (tid < NB) {
        const int* o = S.off + tid * (NB + 1);
        int k = 0;
        for (int b = 0; b < NB * NB; ++b) {
            S.kb[tid][b] = k;
            k += ((o[b / NB + 1] - o[b / NB]) * (o[b % NB + 1] - o[b % NB]) + 3) & ~3;
        }
        S.kb[tid][NB * NB] = k;
    }
    __syncthreads();
    for (int i = tid; i < NB * NA * NA * 27; i += TH) {
        const int abc = i % 27, n2 = i / 27 % NA, n1 = i / (27 * NA) % NA, mu = i / (27 * NA * NA);
        const int* o = S.off + mu * (NB + 1);
        if (n1 >= o[NB] || n2 >= o[NB]) continue;  // beyond the atom's slots
        const int nu = n1 >= o[1], eta = n2 >= o[1];
        const int k = S.kb[mu][nu * NB + eta] + (n1 - o[nu]) * (o[eta + 1] - o[eta]) + n2 - o[eta];
        S.fc[mu][k][abc] = P.fc3[i] * (S.mrs[nu] * S.mrs[eta]);
        if (abc == 0) S.ksrc[mu][k] = n1 | n2 << 8;
    }
    __syncthreads();

    // lane constants: B fragments of a product, D positions of the fold's rows
    int boff[3], dpos[4];
    unsigned neg[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int kk = 4 * k + lc, im = kk >= 6, row = kk - 6 * im;
        boff[k] = (row * ST + (lr >> 1)) * 2 + ((lr & 1) ^ im);
        neg[k] = im && !(lr & 1) ? 0x80000000u : 0u;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int abc = 8 * m + lr;
        dpos[m] = (abc % 3) * ST + abc / 9 * 6 + abc / 3 % 3;
    }
    const int ngroups = max(0, (a.pair_end - a.pair_first + GP - 1) / GP);
    // contiguous groups per team, spread over the SMs first
    const int teams = TEAMS * gridDim.x, wid = team * gridDim.x + blockIdx.x;
    const int per = (ngroups + teams - 1) / teams;
    const int gb = min(wid * per, ngroups), ge = min(gb + per, ngroups);

    for (int grp = gb; grp < ge; ++grp) {
        team_sync(team);
        if (t64 < GP) {
            const int idx = a.pair_first + grp * GP + t64;
            const bool have = idx < a.pair_end;
            const int pr = have ? (a.plist ? a.plist[idx] : idx) : (a.plist ? a.plist[a.pair_first] : a.pair_first);
            const int2 g = P.pairs[pr];
            const int q = P.pair_q0[pr];
            M.g1[t64] = g.x;
            M.g2[t64] = g.y;
            M.q0[t64] = q;
            M.p0[t64] = P.q0_grid ? P.q0_grid[q] : q;
            const bool gq0 = P.q0_int[3 * q] == 0 && P.q0_int[3 * q + 1] == 0 && P.q0_int[3 * q + 2] == 0;
            M.gam[t64] = have ? (gq0 ? 1 : 0) | (g.x == 0 ? 2 : 0) | (g.y == 0 ? 4 : 0) : -1;
        }
        team_sync(team);
        double xw[2], xo[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = t64 + 64 * h, p = i / (3 * N), k = i / N % 3, s = i % N;
            if (i < GP * 3 * N) {
                const size_t q = (size_t)(k == 0 ? M.p0[p] : (k == 1 ? M.g1[p] : M.g2[p])) * N + s;
                xw[h] = (k == 0 ? P.om0 : P.omg)[q];
                xo[h] = (k == 0 ? P.ob0 : P.obg)[q];
            }
        }
        for (int i = t64; i < GP * 2 * NB * NA; i += 64) {
            const int p = i / (2 * NB * NA), leg = i / (NB * NA) % 2, j = i % (NB * NA);
            const int g = leg ? M.g2[p] : M.g1[p];
            const double* R = S.posr + j * 3;
            const double qr = P.qpnt[3 * g] * R[0] + P.qpnt[3 * g + 1] * R[1] + P.qpnt[3 * g + 2] * R[2];
            double sn, cs;
            sincos(qr, &sn, &cs);
            M.ph[p][leg][j] = make_double2(cs, sn);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = t64 + 64 * h;
            if (i < GP * 3 * N) {
                (&M.w[0][0][0])[i] = xw[h];
                (&M.ob[0][0][0])[i] = xo[h];
                (&M.wf[0][0][0])[i] = (float)xw[h];
            }
        }
        team_sync(team);
        {
            // fold, mu = half: column 2 pair + re/im; a lane ends with D of pair lc at rows abc = 8 m + lr
            const double2* x = M.ph[lr >> 1][0] + half * NA;
            const double2* y = M.ph[lr >> 1][1] + half * NA;
            const bool im = lr & 1;
#pragma unroll 1
            for (int blk = 0; blk < NB * NB; ++blk) {
                double c[4][2];
#pragma unroll
                for (int m = 0; m < 4; ++m) c[m][0] = c[m][1] = 0.0;
                for (int k = S.kb[half][blk] + lc; k < S.kb[half][blk + 1]; k += 4) {
                    const int src = S.ksrc[half][k];
                    const double2 u = x[src & 255], v = y[src >> 8];
                    const double b = im ? u.x * v.y + u.y * v.x : u.x * v.x - u.y * v.y;
                    const double* f = &S.fc[half][k][lr];
#pragma unroll
                    for (int m = 0; m < 4; ++m) dmma(c[m], f[8 * m], b);
                }
                double2* D = &M.D[lc][(blk % NB) * 3 * ST + half * 18 + blk / NB * 3];
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (8 * m + lr < 27) D[dpos[m]] = make_double2(c[m][0], c[m][1]);
            }
        }
        team_sync(team);
        unsigned short* queue = M.queue[half][min(lr, N - 1)];
        int qc = 0;  // EPI 0: queued hits of row lr
#pragma unroll 1
        for (int p = half * WP; p < half * WP + WP; ++p) {
            const int gam = M.gam[p];
            if (gam < 0) break;
            const int g1 = M.g1[p], g2 = M.g2[p], q0 = M.q0[p], p0 = M.p0[p];
            double A0[3], A1[3], A2[3], c[9][2];
            efrag(A2, P.evg + (size_t)g2 * 36, lr, lc);
            efrag(A1, P.evg + (size_t)g1 * 36, lr, lc);
            efrag(A0, P.ev0 + (size_t)p0 * 36, lr, lc);
            constexpr int NV = EPI == 0 ? (2 * N * NT + 31) / 32 : 1;
            double xn[NV];  // n of q1 and q2, on its way to shared memory
            if (EPI == 0)
#pragma unroll
                for (int h = 0; h < NV; ++h) {
                    const int i = lane + 32 * h, t = i % NT, ls = i / NT;
                    if (i < 2 * N * NT && t < a.nT)
                        xn[h] = P.nbeg[((size_t)t * a.nq + (ls < N ? g1 : g2)) * N + ls % N];
                }
#pragma unroll
            for (int k = 0; k < 3; ++k) A0[k] *= S.mrs[(4 * k + lc) % 6 / 3];
            double2* D = M.D[p];
            product(c, A2, D, boff, neg);  // T1: row s2, column (mu a) 6 + nu b
            __syncwarp();
            if (lr < N)
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int col = 4 * t + lc, ma = col * 43 >> 8, nb = col - 6 * ma;
                    D[nb * ST + ma * 6 + lr] = make_double2(c[t][0], c[t][1]);
                }
            __syncwarp();
            product(c, A1, D, boff, neg);  // T2: row s1, column (mu a) 6 + s2
            __syncwarp();
            if (lr < N)
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int col = 4 * t + lc, ma = col * 43 >> 8, s2 = col - 6 * ma;
                    D[ma * ST + lr * 6 + s2] = make_double2(c[t][0], c[t][1]);
                }
            __syncwarp();
            product(c, A0, D, boff, neg);  // Phi: row s0, column s1 6 + s2
            __syncwarp();
            const int s0 = min(lr, N - 1);
            const bool gq0 = gam & 1, gq1 = gam & 2, gq2 = gam & 4;
            const double w0 = M.w[p][0][s0], ob0 = M.ob[p][0][s0];
            double* Ws = reinterpret_cast<double*>(D);
            if (EPI == 0 || EPI == 1)
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int col = 4 * t + lc, s1 = col * 43 >> 8, s2 = col - 6 * s1;
                    const bool zero = (gq0 && s0 < 3) || (gq1 && s1 < 3) || (gq2 && s2 < 3);
                    const double abs2 = c[t][0] * c[t][0] + c[t][1] * c[t][1];
                    const double W = zero ? 0.0 : abs2 * (ob0 * M.ob[p][1][s1] * M.ob[p][2][s2]) * a.mfac;
                    if (lr < N) Ws[s0 * 36 + col] = W;
                }
            if (EPI == 0) {
#pragma unroll
                for (int h = 0; h < NV; ++h)
                    if (lane + 32 * h < 2 * N * NT) Ws[216 + lane + 32 * h] = xn[h];
                // FP32 screen, one bit per check set outside, wider than the underflow point by more than its
                // rounding
                const float f0 = M.wf[p][0][s0];
                float big = fabsf(f0);
#pragma unroll
                for (int s = 0; s < N; ++s) big = fmaxf(big, fmaxf(fabsf(M.wf[p][1][s]), fabsf(M.wf[p][2][s])));
                const float r = (float)(sqrt(2.0 * EXP_UNDERFLOW) / a.onebysigma) * 1.0001f + 4e-6f * big;
                unsigned out = 0, live = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int col = 4 * t + lc, s1 = col * 43 >> 8, s2 = col - 6 * s1;
                    const float f1 = M.wf[p][1][s1], f2 = M.wf[p][2][s2];
                    out = __funnelshift_l(__float_as_uint(r - fabsf(f0 - f1 - f2)), out, 1);
                    out = __funnelshift_l(__float_as_uint(r - fabsf(f0 + f1 - f2)), out, 1);
                    out = __funnelshift_l(__float_as_uint(r - fabsf(f0 - f1 + f2)), out, 1);
                    const bool on = s1 >= a.pol_lo[1] && s1 <= a.pol_hi[1] && s2 >= a.pol_lo[2] && s2 <= a.pol_hi[2] &&
                                    !(gq1 && s1 < 3) && !(gq2 && s2 < 3);
                    if (on) live |= 7u << (24 - 3 * t);
                }
                if (lr >= N || s0 < a.pol_lo[0] || s0 > a.pol_hi[0]) live = 0;
                unsigned in = ~out & live;
                const int cnt = __popc(in);
                const int x1 = __shfl_up_sync(0xffffffffu, cnt, 1, 4);
                int pos = cnt + (lc >= 1 ? x1 : 0);
                const int x2 = __shfl_up_sync(0xffffffffu, pos, 2, 4);
                pos += lc >= 2 ? x2 : 0;
                const int tot = __shfl_sync(0xffffffffu, pos, 3, 4);
                pos += qc - cnt;
                qc += tot;
                const unsigned base = lc | (p & 1) << 11;
                while (in) {  // bit 26 - 3 t - ch
                    const int b = 26 - (31 - __clz(in));
                    in &= ~(1u << (26 - b));
                    const int t = b / 3;
                    queue[pos++] = (unsigned short)((base + 4 * t) | (b - 3 * t) << 6);
                }
                __syncwarp();
                if (p + 1 < half * WP + WP && M.gam[p + 1] >= 0 && M.q0[p + 1] == q0) continue;
                // the queued hits of this q0, one s0 at a time
                const double pre = a.onebysigma * ONEBYSQRT2PI;
#pragma unroll 1
                for (int z = 0; z < N; ++z) {
                    const int cz = __shfl_sync(0xffffffffu, qc, 4 * z);
                    if (cz == 0) continue;
                    double acc[NT + 1];
#pragma unroll
                    for (int t = 0; t <= NT; ++t) acc[t] = 0.0;
                    const unsigned short* qz = M.queue[half][z];
                    for (int i = lane; i < cz; i += 64) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const bool have = i + 32 * h < cz;
                            const unsigned code = qz[have ? i + 32 * h : i];
                            const int cc = code & 63, ch = code >> 6 & 3, pp = half * WP + (code >> 11);
                            const int s1 = cc * 43 >> 8, s2 = cc - 6 * s1;
                            const double v0 = M.w[pp][0][z], w1 = M.w[pp][1][s1], w2 = M.w[pp][2][s2];
                            const double d = ch == 0 ? v0 - w1 - w2 : (ch == 1 ? v0 + w1 - w2 : v0 - w1 + w2);
                            const double x = 0.5 * a.onebysigma2 * (d * d);
                            const double mult = M.g1[pp] != M.g2[pp] ? 2.0 : 1.0;
                            const double e = have && x < EXP_UNDERFLOW ? mult * (pre * exp(-x)) : 0.0;
                            const double* Wp = reinterpret_cast<const double*>(M.D[pp]);
                            acc[NT] += e;
                            const double v = Wp[z * 36 + cc] * (ch == 2 ? -e : e);
                            const double *n1 = Wp + 216 + s1 * NT, *n2 = Wp + 216 + (N + s2) * NT;
#pragma unroll
                            for (int t = 0; t < NT; ++t)
                                if (t < a.nT) acc[t] = fma(v, ch == 0 ? n1[t] + n2[t] + 1.0 : n1[t] - n2[t], acc[t]);
                        }
                    }
                    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                        for (int t = 0; t <= NT; ++t) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
#pragma unroll
                    for (int t = 0; t < NT; ++t)
                        if (lane == t && t < a.nT && acc[t] != 0.0)
                            atomicAdd(&P.out_lw[((size_t)t * a.nq0 + q0) * N + z], acc[t]);
                    if (lane == NT && acc[NT] != 0.0) atomicAdd(&P.out_p3[(size_t)q0 * N + z], acc[NT]);
                }
                qc = 0;
                __syncwarp();
            } else if (EPI == 1) {
                __syncwarp();
                const int slot = q0 - a.q0_first;
                double2* o1 = reinterpret_cast<double2*>(P.out_w + ((size_t)slot * a.nq + g1) * 216);
                double2* o2 = reinterpret_cast<double2*>(P.out_w + ((size_t)slot * a.nq + g2) * 216);
                for (int i = lane; i < 108; i += 32) {
                    o1[i] = D[i];
                    const int z = i / 18, sa = i / 3 % 6, sb = i % 3 * 2;  // o2[z][sa][sb, sb + 1]
                    if (g1 != g2) o2[i] = make_double2(Ws[z * 36 + sb * 6 + sa], Ws[z * 36 + sb * 6 + 6 + sa]);
                }
            } else {
                // EPI 2: this lane's operator entries (columns 4 t + lc), appended with one atomic per warp
                const double pre = a.onebysigma * ONEBYSQRT2PI;
                const bool self = g1 == g2;
                double bP[9], bQ[9];
                int cnt = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    bP[t] = bQ[t] = 0.0;
                    const int col = 4 * t + lc, s1 = col * 43 >> 8, s2 = col - 6 * s1;
                    const bool zero = (gq0 && s0 < 3) || (gq1 && s1 < 3) || (gq2 && s2 < 3);
                    const double abs2 = c[t][0] * c[t][0] + c[t][1] * c[t][1];
                    const double W = zero || lr >= N ? 0.0 : abs2 * (ob0 * M.ob[p][1][s1] * M.ob[p][2][s2]) * a.mfac;
                    if (W == 0.0) continue;
                    const double w1 = M.w[p][1][s1], w2 = M.w[p][2][s2];
                    const double da = w0 + w1 - w2, db = w0 + w2 - w1, dm = w0 - w1 - w2;
                    const double xa = 0.5 * a.onebysigma2 * (da * da), xb = 0.5 * a.onebysigma2 * (db * db),
                                 xm = 0.5 * a.onebysigma2 * (dm * dm);
                    const double ea = xa < EXP_CUT_BTE ? pre * exp(-xa) : 0.0;
                    const double eb = (!self && xb < EXP_CUT_BTE) ? pre * exp(-xb) : 0.0;
                    const double em = xm < EXP_CUT_BTE ? pre * exp(-xm) : 0.0;
                    bP[t] = 4.0 * W * (ea - eb);
                    bQ[t] = 4.0 * W * (self ? 0.5 : 1.0) * em;
                    cnt += (bP[t] != 0.0 || bQ[t] != 0.0) ? 1 : 0;
                }
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                unsigned long long base = 0;
                if (lane == 31 && total > 0) base = atomicAdd(P.item_ctr, (unsigned long long)total);
                base = __shfl_sync(0xffffffffu, base, 31);
                unsigned long long pos = base + (unsigned long long)(incl - cnt);
                BteEntry* out = static_cast<BteEntry*>(P.out_items);
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    if (bP[t] == 0.0 && bQ[t] == 0.0) continue;
                    const int col = 4 * t + lc, s1 = col * 43 >> 8, s2 = col - 6 * s1;
                    if ((long long)pos < P.item_cap) {
                        BteEntry e;
                        e.r0 = (q0 - a.q0_first) * N + s0;
                        e.k1 = g1 * N + s1;
                        e.k2 = g2 * N + s2;
                        e.pad = 0;
                        e.P = bP[t];
                        e.Q = bQ[t];
                        out[pos] = e;
                    }
                    ++pos;
                }
            }
        }
    }
}

S3Ptrs v3s_ptrs(spring_ctx* c, const PairSet& ps, const Q0View& v, double* lw, double* p3, double* w) {
    return S3Ptrs{ps.pairs.p, ps.pair_q0.p, c->d_fc3.p, c->d_fc3_posr.p, c->d_fc3_off.p,
                  c->d_mass_rs.p, c->d_qpnt.p, v.q0_int, v.q0_grid, v.evec, v.omega, v.oneby, c->ph_grid.evec.p,
                  c->ph_grid.omega.p, c->ph_grid.oneby.p, c->ph_grid.nbe.p, lw, p3, w, nullptr, nullptr, 0};
}

template <int EPI, int NT>
int launch_kernel(spring_ctx* c, const S3Args& a, const S3Ptrs& P, long long bound, const int* range, int n_q0, int cap,
                  const char* name) {
    cudaFuncSetAttribute(k_v3s<EPI, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
    int dev_sms = 148;
    cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, c->device);
    const int grid = (int)std::min<long long>((bound + GP - 1) / GP, dev_sms);
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "v3: injected launch failure");
    k_v3s<EPI, NT><<<grid, 64 * TEAMS, sizeof(Smem), c->stream>>>(a, P, range, n_q0, cap);
    return launch_check(c, name);
}

}  // namespace

bool v3s_takes(const spring_ctx* c) { return c->nb == NB && c->na3 == NA && c->nT <= MAXT; }

// Launch the specialised kernel when the cell fits it; *handled tells the caller.
int launch_v3s(spring_ctx* c, const PairSet& ps, const Q0View& v, int q0_first, int n_q0, int epi, double sigma,
               const Pol* pol, double* lw, double* p3, double* w, bool* handled, const int* plist, int nlist) {
    *handled = v3s_takes(c);
    if (!*handled) return SPRING_OK;
    S3Args a{};
    a.nq = c->nq;
    a.nT = c->nT;
    a.nq0 = ps.n0;
    a.q0_first = q0_first;
    // Host offsets when they were read already; otherwise the kernel reads its range on the device
    // and the grid is sized by the bound of at most Nq/2 + 8 pairs per q0 (no readback, no wait).
    const int* range = nullptr;
    long long bound;
    a.plist = plist;
    if (plist) {  // an explicit list of pairs (the Gaussian window's pre-screen)
        a.pair_end = nlist;
        bound = nlist;
    } else if (ps.h_ok) {
        a.pair_first = ps.h_pairoff[q0_first];
        a.pair_end = ps.h_pairoff[q0_first + n_q0];
        bound = a.pair_end - a.pair_first;
    } else {
        range = ps.pairoff.p + q0_first;
        bound = std::min<long long>((long long)n_q0 * (c->nq / 2 + 8), ps.cap);
    }
    a.mfac = host_constants().Sctr3THz2 / double(c->nq);
    if (epi == 0) {
        a.onebysigma = 1.0 / sigma;
        a.onebysigma2 = a.onebysigma * a.onebysigma;
        for (int k = 0; k < 3; ++k) {
            a.pol_lo[k] = pol->lo[k];
            a.pol_hi[k] = pol->hi[k];
        }
    }
    if (bound == 0) return SPRING_OK;
    const S3Ptrs P = v3s_ptrs(c, ps, v, lw, p3, w);
    if (epi == 1) return launch_kernel<1, 1>(c, a, P, bound, range, n_q0, ps.cap, "k_v3s<wgrid>");
    return c->nT <= 3 ? launch_kernel<0, 3>(c, a, P, bound, range, n_q0, ps.cap, "k_v3s<gauss>")
                      : launch_kernel<0, MAXT>(c, a, P, bound, range, n_q0, ps.cap, "k_v3s<gauss>");
}

// Entries of the Gaussian BTE operator (EPI 2) of pair set ps, q0 block [q0_first, +n_q0): every
// mode triple with a delta weight above the exp(-40) cut is appended to `items` (capacity cap) at
// *ctr (zeroed by the caller); *ctr ends as the number of entries, those past cap not written.
int launch_v3s_bte(spring_ctx* c, const PairSet& ps, const Q0View& v, int q0_first, int n_q0, double sigma,
                   void* items, unsigned long long* ctr, long long cap, bool* handled) {
    *handled = c->nb == NB && c->na3 == NA;
    if (!*handled) return SPRING_OK;
    S3Args a{};
    a.nq = c->nq;
    a.nT = c->nT;
    a.nq0 = ps.n0;
    a.q0_first = q0_first;
    SPRING_CHECK(pairoff_host(c, ps));
    a.pair_first = ps.h_pairoff[q0_first];
    a.pair_end = ps.h_pairoff[q0_first + n_q0];
    a.mfac = host_constants().Sctr3THz2 / double(c->nq);
    a.onebysigma = 1.0 / sigma;
    a.onebysigma2 = a.onebysigma * a.onebysigma;
    if (a.pair_end == a.pair_first) return SPRING_OK;
    S3Ptrs P = v3s_ptrs(c, ps, v, nullptr, nullptr, nullptr);
    P.out_items = items;
    P.item_ctr = ctr;
    P.item_cap = cap;
    return launch_kernel<2, 1>(c, a, P, a.pair_end - a.pair_first, nullptr, n_q0, ps.cap, "k_v3s<bte>");
}

}  // namespace spring
