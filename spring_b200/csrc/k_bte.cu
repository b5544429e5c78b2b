// Iterative (non-RTA) Boltzmann transport of kappa_iter.x on the device.
//
// Reference (src/Kappa/Src_iterative): the time-reversal irreducible set
// (Irr_q_point_m.f90:216-335), W+ = W (n1 - n2) and W- = W (1 + n1 + n2) per
// pair (Quasi_momentum_consrv.f90:567-621, Sctr3THz2 with pi/4), 1/tau from the
// tetrahedron sums TetrahedronWplus / TetrahedronWminus (:701-1208, strict case
// bounds, a vertex set counts only when |sum I - 1| < 5e-5), CreateFzero,
// TetrahedronIterPlus / Minus (TetrahedronDeltaSum.f90:22-607), multiplyTaudFnew,
// kappa (HelperSubroutines.f90:118-347) and the loop of main.f90:295-361.
// The test on sum I is not made: for distinct energies every difference in the weights is exact or rounded
// once, and no sum of them cancels, so the four add up to one within a few roundings however close the
// energies lie (3e5 random sets, energies one rounding apart among them: 4.4e-16) and it rejects nothing.
//
// Representatives of the time-reversal pairs {q, -q} are the smaller grid
// index (the reference takes the first one met while building tetrahedra);
// F(-q) = -F(q).  The W of a vertex comes from kappa.x's W grid of the same q0,
// which stores both orientations of every pair; 4 W there is kappa_iter's W.
//   plus  channel, vertex x:  partner -p(x),  M = w(-p(x),s2) - w(x,s1),
//                             W+ = 4 W3(q0; x s1; p(x) s2) (n(x,s1) - n(p(x),s2)),
//                             dF term (F(-p(x),s2) - F(x,s1));
//   minus channel, vertex v:  partner u = -p(-v), M = w(v,s1) + w(u,s2),
//                             W- = 4 W3(q0; -v s1; p(-v) s2) (1 + n(-v,s1) + n(p(-v),s2)),
//                             dF term 0.5 (F(u,s2) + F(v,s1));
// with p(x) = grid(-q0 - x).  Because F(-q) = -F(q), both terms are -(F(x, s1) + F(p(x), s2)) times a
// coefficient at the grid modes (x, s1), (p(x), s2) - x = -v for the minus channel - that depends on the
// temperature only through n there (points that are their own inverse: see bte_entry).  So the tetrahedron
// weights are computed once: every (tetrahedron, mode triple) whose energy range holds w0 adds its vertex
// weights to a dense (P, Q) grid of its q0, and the non-zero entries, with 4 W folded in and the two
// orderings of a pair merged, go to HBM as rows of the same operator the Gaussian form uses; an iteration is
// one pass over it.  When the operator does not fit (half the free memory), the (P, Q) grids are rebuilt batch
// by batch on every pass instead.
// Weights: FP32 screen and queued FP64 evaluation as in k_tetra3.  The former kernel evaluated the
// weights of every tetrahedron again in every iteration.
// Roofline: FP64 ALU for the weights, HBM / L2 (24 bytes and two gathers per entry) for the iterations.
#include <algorithm>
#include <cmath>
#include <cub/cub.cuh>

#include "spring_internal.cuh"
#include "tetra.cuh"
#include "v3s.cuh"

namespace spring {
namespace {

constexpr int NS0 = 6, BS2 = 6, TW = 4;
constexpr double ZERO_PREC = 5.0e-5;
constexpr double FUNIT_E = 1.054571817 / 1.380649;  // FunitE_11m_K (Src_iterative/constants.f90:56)
constexpr double KW_MK = 1.054571817 * 0.001;       // kW_mK (:58)

__global__ void k_bte_wf(int nq, int n, const double* __restrict__ om, float* __restrict__ wf) {  // [s][q]
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq * n; i += gridDim.x * blockDim.x)
        wf[(size_t)(i % n) * nq + i / n] = (float)om[i];
}

struct WgtArgs {
    int n, nq, ntet, q0_first;
    int per1, nb1, nb2;         // s1 values of a unit; s1 and s2 blocks
    long long units;
    const int* tr_grid;         // [ntr]
    const int* neg;             // [nq]
    const int* partner;         // [ntr][nq]
    const float* wf;            // [n][nq]
    const double* omega;        // [nq][n]
    double2* pq;                // [slot][s0][s1][s2][x] (P, Q), zeroed
};

// Tetrahedron weights of the plus (P) and minus (Q, half weight) channel of every q0 of a batch: warps
// screen 32 tetrahedra at a time in FP32, queue the (tetrahedron, s1, s2, s0, channel) whose range holds
// w0, and evaluate 32 of them at a time (k_tetra.cu has the reasons).
__global__ void __launch_bounds__(32 * TW, 4) k_bte_weights(WgtArgs a, const int4* __restrict__ tet) {
    constexpr int K = 2 * NS0;
    __shared__ unsigned queue_[TW][32 * K + 32];
    __shared__ float o2_[TW][BS2][8][32];
    __shared__ double w0d[NS0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = blockIdx.y, q0 = a.q0_first + slot;
    const int n = a.n, nq = a.nq;
    const int s0a = blockIdx.z * NS0, s0n = min(NS0, n - s0a);
    const int* __restrict__ p = a.partner + (size_t)q0 * nq;
    const int* __restrict__ neg = a.neg;
    double* pq = reinterpret_cast<double*>(a.pq) + ((size_t)slot * n + s0a) * n * n * nq * 2;
    if (threadIdx.x < NS0)
        w0d[threadIdx.x] = threadIdx.x < s0n ? a.omega[(size_t)a.tr_grid[q0] * n + s0a + threadIdx.x] : 0.0;
    __syncthreads();
    float w0[NS0];
    unsigned live = 0;
#pragma unroll
    for (int i = 0; i < NS0; ++i) {
        w0[i] = (float)w0d[i];
        if (i < s0n) live |= (1u << (K - 1 - i)) | (1u << (NS0 - 1 - i));
    }
    unsigned* queue = queue_[warp];
    float(*o2)[8][32] = o2_[warp];
    const long long stride = (long long)gridDim.x * TW;
    for (long long u = (long long)blockIdx.x * TW + warp; u < a.units; u += stride) {
        const int b2 = (int)(u % a.nb2), b1 = (int)(u / a.nb2 % a.nb1), g = (int)(u / ((long long)a.nb2 * a.nb1));
        const int s1a = b1 * a.per1, s1e = min(s1a + a.per1, n);
        const int s2a = b2 * BS2, s2n = min(BS2, n - s2a);
        const bool on = g * 32 + lane < a.ntet;
        const int4 tv = on ? tet[g * 32 + lane] : make_int4(0, 0, 0, 0);
        const int x[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int pp = neg[p[x[v]]], pm = neg[p[neg[x[v]]]];
            for (int k = 0; k < s2n; ++k) {
                o2[k][v][lane] = a.wf[(size_t)(s2a + k) * nq + pp];
                o2[k][4 + v][lane] = a.wf[(size_t)(s2a + k) * nq + pm];
            }
        }
        auto evaluate = [&](unsigned code) {
            const int tl = code & 31, s1 = (code >> 5) & 31, s2 = (code >> 10) & 31;
            const int k = K - 1 - (int)(code >> 15), ch = k / NS0, si = k % NS0;
            const int4 t = tet[g * 32 + tl];
            int at[4] = {t.x, t.y, t.z, t.w}, row[4];
            double M[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                row[v] = ch == 0 ? at[v] : neg[at[v]];
                const double w1 = a.omega[(size_t)at[v] * n + s1], w2 = a.omega[(size_t)neg[p[row[v]]] * n + s2];
                M[v] = ch == 0 ? w2 - w1 : w1 + w2;
            }
            tet::sort4_carry(M, row, at);
            double gw, A[4];
            if (!tet::g_weights<true>(w0d[si], M, gw, A)) return;
            const double f = ch == 0 ? 1.0 : 0.5;
            double* o = pq + ((size_t)(si * n + s1) * n + s2) * nq * 2 + ch;
#pragma unroll
            for (int v = 0; v < 4; ++v) atomicAdd(o + 2 * (size_t)row[v], f * A[v]);
        };
        int qn = 0;
        for (int s1 = s1a; s1 < s1e; ++s1) {
            float o1[4], e1 = 0.0f;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                o1[v] = a.wf[(size_t)s1 * nq + x[v]];
                e1 += fabsf(o1[v]);
            }
#pragma unroll 1
            for (int k = 0; k < s2n; ++k) {
                unsigned out = 0;  // one bit per check, set outside
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    const float a0 = o2[k][4 * ch][lane], a1 = o2[k][4 * ch + 1][lane], a2 = o2[k][4 * ch + 2][lane],
                                a3 = o2[k][4 * ch + 3][lane];
                    const float margin = 1e-6f * (e1 + (fabsf(a0) + fabsf(a1) + fabsf(a2) + fabsf(a3)));
                    const float sg = ch == 0 ? -1.0f : 1.0f;
                    const float m0 = fmaf(sg, o1[0], a0), m1 = fmaf(sg, o1[1], a1), m2 = fmaf(sg, o1[2], a2),
                                m3 = fmaf(sg, o1[3], a3);
                    const float lo = fminf(fminf(m0, m1), fminf(m2, m3)), hi = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                    const float mid = 0.5f * (lo + hi), half = fmaf(0.5f, hi - lo, margin);
#pragma unroll
                    for (int i = 0; i < NS0; ++i)
                        out = __funnelshift_l(__float_as_uint(half - fabsf(w0[i] - mid)), out, 1);
                }
                unsigned in = on ? ~out & live : 0u;
                const unsigned c = __popc(in);
                unsigned pre = 0, tot = 0;
                const unsigned lt = (1u << lane) - 1;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const unsigned m = __ballot_sync(0xffffffffu, (c >> b) & 1);
                    pre += __popc(m & lt) << b;
                    tot += __popc(m) << b;
                }
                if (tot == 0) continue;
                const unsigned base = lane | s1 << 5 | (s2a + k) << 10;
                unsigned pos = qn + pre;
                while (in) {
                    const int b = __ffs(in) - 1;
                    in &= in - 1;
                    queue[pos++] = base | b << 15;
                }
                qn += tot;
                __syncwarp();
                while (qn >= 32) {
                    qn -= 32;
                    evaluate(queue[qn + lane]);
                }
                __syncwarp();
            }
        }
        if (lane < qn) evaluate(queue[lane]);
        __syncwarp();
    }
}

struct RowArgs {
    int n, nq, q0_first;
    const int* partner;    // [ntr][nq]
    const int* neg;        // [nq]
    const double2* pq;     // [slot][s0][s1][s2][x]
    const double* wgrid;   // [slot][x][s0][s1][s2]
};

// The merged entries of grid modes k1 = (x, s1), k2 = (p(x), s2) of one row, element j = (s1 n + s2) nq + x of its
// (P, Q) block.  With c = (n1 - n2) P + (1 + n1 + n2) Q of e[0], both orderings of the pair add c to 1/tau and
// -c (F(k1) + F(k2)) to dF.  W is stored both ways round for different points; at x = p(x) W(s1, s2) and
// W(s2, s1) differ unless FC3 is symmetric in its two neighbours, and so do their terms.
// The sum F(k1) + F(k2) comes of F(-q) = -F(q).  A point that is its own inverse has F(-q) = F(q) instead, and F
// vanishes there only when W is the same for (q1, q2) and (-q1, -q2) - again with symmetric FC3 only.  e[1] and
// e[2] (in the same form, n of their own mode first) are what is missing from F(k1) and F(k2) then, to be
// subtracted from dF and not part of 1/tau.
// Returns which of the three are not zero, bit by bit; none when another element stands for this one.
__device__ __forceinline__ unsigned bte_entry(const RowArgs& a, int j, int s0, const int* __restrict__ p,
                                              const double2* __restrict__ pq, const double* __restrict__ W, int2& kk,
                                              double2* e) {
    const int n = a.n, nq = a.nq, x = j % nq, s12 = j / nq, s1 = s12 / n, s2 = s12 % n, px = p[x];
    if (px < x || (px == x && s2 < s1)) return 0;
    double2 u = pq[j], v = make_double2(0.0, 0.0);
    if (px != x || s1 != s2) v = pq[(s2 * n + s1) * nq + px];
    else u.x = 0.0;
    if (u.x == 0.0 && u.y == 0.0 && v.x == 0.0 && v.y == 0.0) return 0;
    const double* w = W + (size_t)x * n * n * n + (size_t)s0 * n * n;
    const double w1 = 4.0 * w[s1 * n + s2], w2 = px == x ? 4.0 * w[s2 * n + s1] : w1;
    kk = make_int2(x * n + s1, px * n + s2);
    e[0] = make_double2((u.x - v.x) * w1, (u.y + v.y) * w1);
    if (w2 != w1) e[0] = make_double2(u.x * w1 - v.x * w2, u.y * w1 + v.y * w2);
    unsigned m = e[0].x != 0.0 || e[0].y != 0.0 ? 1 : 0;
    if (a.neg[x] == x) {
        e[1] = make_double2(2.0 * v.x * w2, -2.0 * e[0].y);
        if (e[1].x != 0.0 || e[1].y != 0.0) m |= 2;
    }
    if (a.neg[px] == px) {
        e[2] = make_double2(2.0 * u.x * w1, -2.0 * e[0].y);
        if (e[2].x != 0.0 || e[2].y != 0.0) m |= 4;
    }
    return m;
}

// One block per segment of a row: blockIdx.x = (slot n + s0) nseg + segment, [seg, seg + 1) / nseg of the
// row's elements.  COUNT: its entries to cnt.  Otherwise they are written in element order from base + boff
// on, and that offset to off.
template <bool COUNT>
__global__ void __launch_bounds__(256) k_bte_entries(RowArgs a, int nseg, int* __restrict__ cnt,
                                                     const int* __restrict__ boff, long long base0, int last,
                                                     int* __restrict__ off, int2* __restrict__ kk,
                                                     double2* __restrict__ pqo) {
    __shared__ int wsum[8];
    const int n = a.n, nq = a.nq, row = blockIdx.x / nseg, seg = blockIdx.x % nseg;
    const int slot = row / n, s0 = row % n, len = n * n * nq;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int step = ((len + nseg - 1) / nseg + 255) / 256 * 256;
    const int j1 = min(len, (seg + 1) * step);
    const int* p = a.partner + (size_t)(a.q0_first + slot) * nq;
    const double2* pq = a.pq + (size_t)row * len;
    const double* W = a.wgrid + (size_t)slot * nq * n * n * n;
    int total = 0;
    long long base = 0;
    if (!COUNT) {
        const size_t g = (size_t)a.q0_first * n * nseg + blockIdx.x;
        base = base0 + boff[blockIdx.x];
        if (threadIdx.x == 0) off[g] = (int)base;
        if (threadIdx.x == 0 && last && blockIdx.x == gridDim.x - 1) off[g + 1] = (int)(base0 + boff[blockIdx.x + 1]);
    }
    for (int j0 = seg * step; j0 < j1; j0 += 256) {
        const int j = j0 + (int)threadIdx.x;
        int2 k;
        double2 e[3];
        const unsigned on = j < j1 ? bte_entry(a, j, s0, p, pq, W, k, e) : 0u;
        if (COUNT) {
            total += __popc(on);
            continue;
        }
        unsigned m[3];
#pragma unroll
        for (int h = 0; h < 3; ++h) m[h] = __ballot_sync(0xffffffffu, on >> h & 1);
        if (lane == 0) wsum[warp] = __popc(m[0]) + __popc(m[1]) + __popc(m[2]);
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            before += w < warp ? wsum[w] : 0;
            all += wsum[w];
        }
        long long o = base + before;
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            if (on >> h & 1) {
                const long long i = o + __popc(m[h] & ((1u << lane) - 1));
                kk[i] = h == 0 ? k : (h == 1 ? make_int2(~k.x, k.y) : make_int2(~k.y, k.x));
                pqo[i] = e[h];
            }
            o += __popc(m[h]);
        }
        base += all;
        __syncthreads();
    }
    if (COUNT) {
        for (int o = 16; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
        if (lane == 0) wsum[warp] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < 8; ++w) t += wsum[w];
            cnt[blockIdx.x] = t;
        }
    }
}

// Sums of one block's 256 threads: thread k < NV gets v[k] summed.
template <int NV>
__device__ __forceinline__ double block_sum(const double* v, double (*red)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double x[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) x[k] = v[k];
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; ++k) x[k] += __shfl_down_sync(0xffffffffu, x[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[k][warp] = x[k];
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < NV)
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
    return t;
}

// Row sums straight from the (P, Q) blocks of a batch (the operator did not fit): MODE 0 1/tau, MODE 1
// dF = -sum c (F(k1) + F(k2)).
template <int MODE>
__global__ void __launch_bounds__(256) k_bte_dense(RowArgs a, const double* __restrict__ nbe,
                                                   const double* __restrict__ Fg, double* __restrict__ out) {
    __shared__ double red[3][8];
    const int n = a.n, nq = a.nq, slot = blockIdx.x / n, s0 = blockIdx.x % n, len = n * n * nq;
    const int* p = a.partner + (size_t)(a.q0_first + slot) * nq;
    const double2* pq = a.pq + (size_t)blockIdx.x * len;
    const double* W = a.wgrid + (size_t)slot * nq * n * n * n;
    double v[3] = {0.0, 0.0, 0.0};
    for (int j = threadIdx.x; j < len; j += 256) {
        int2 k;
        double2 e[3];
        const unsigned on = bte_entry(a, j, s0, p, pq, W, k, e);
        if (!on) continue;
        const double n1 = nbe[k.x], n2 = nbe[k.y];
        const double c = (n1 - n2) * e[0].x + (1.0 + n1 + n2) * e[0].y;
        if (MODE == 0) {
            v[0] += c;
            continue;
        }
        const double c1 = on & 2 ? (n1 - n2) * e[1].x + (1.0 + n1 + n2) * e[1].y : 0.0;
        const double c2 = on & 4 ? (n2 - n1) * e[2].x + (1.0 + n1 + n2) * e[2].y : 0.0;
        for (int d = 0; d < 3; ++d) {
            const double f1 = Fg[4 * (size_t)k.x + d], f2 = Fg[4 * (size_t)k.y + d];
            v[d] -= c * (f1 + f2) + (c1 * f1 + c2 * f2);
        }
    }
    constexpr int NV = MODE == 0 ? 1 : 3;
    const double t = block_sum<NV>(v, red);
    if (threadIdx.x < NV) out[((size_t)a.q0_first * n + blockIdx.x) * NV + threadIdx.x] = t;
}

struct StepArgs {
    int ntr, n, nq;
    double vol, T;
    const int* tr_grid;
    const int* neg;
    const int* deg;
    const double* omega;
    const double* nbe;      // at this temperature
    const double* vel;
    const double* inv_tau;
    const double* dF;       // [row][parts][3]
    int parts;
    double* F0;
    double* F;              // [row][3], or null
    double* Fg;             // [g][s][4] F at every grid mode, padded to one 32-byte sector, or null
    double* part;           // [blocks][9] kappa partial sums
    unsigned* ticket;       // zero between launches
    double* kappa;          // [9] of this iteration
};

// One iteration's end for every mode of the time-reversal set: F = F0 (INIT, CreateFzero:
// F0 = FunitE w v / (1/tau T^2) where |1/tau| > zero_prec) or F0 + dF tau (multiplyTaudFnew); F at both
// grid points of the pair (F(-q) = -F(q)); and kappa = kW_mK / (Nq V) sum deg w n (n+1) v (x) F, block
// sums added in a fixed order by the last block to finish.
template <bool INIT>
__global__ void __launch_bounds__(256) k_bte_step(StepArgs a) {
    __shared__ double red[9][8];
    __shared__ bool last;
    const int n = a.n;
    double acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.ntr * n; i += gridDim.x * blockDim.x) {
        const int q = i / n, s = i % n, g0 = a.tr_grid[q], gn = a.neg[g0];
        const double it = a.inv_tau[i];
        const bool zero = g0 == 0 && s < 3;
        const bool scale = !zero && fabs(it) > ZERO_PREC;
        const double w = a.omega[(size_t)g0 * n + s];
        const double* v = a.vel + ((size_t)g0 * n + s) * 3;
        double f[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (INIT) {
                f[k] = scale ? FUNIT_E * w * v[k] / (it * (a.T * a.T)) : 0.0;
                a.F0[(size_t)i * 3 + k] = f[k];
            } else {
                double d = 0.0;
                for (int h = 0; h < a.parts; ++h) d += a.dF[((size_t)i * a.parts + h) * 3 + k];
                if (scale) d /= it;
                f[k] = a.F0[(size_t)i * 3 + k] + d;
            }
        }
        if (a.F)
            for (int k = 0; k < 3; ++k) a.F[(size_t)i * 3 + k] = f[k];
        if (a.Fg) {
            double2* o = reinterpret_cast<double2*>(a.Fg + 4 * ((size_t)g0 * n + s));
            o[0] = make_double2(f[0], f[1]);
            o[1] = make_double2(f[2], 0.0);
        }
        if (a.Fg && gn != g0) {
            double2* o = reinterpret_cast<double2*>(a.Fg + 4 * ((size_t)gn * n + s));
            o[0] = make_double2(-f[0], -f[1]);
            o[1] = make_double2(-f[2], 0.0);
        }
        if (zero) continue;
        const double nb = a.nbe[(size_t)g0 * n + s];
        const double pre = double(a.deg[q]) * w * nb * (nb + 1.0);
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int y = 0; y < 3; ++y) acc[3 * x + y] += pre * (v[x] * f[y]);
    }
    const double part = block_sum<9>(acc, red);
    if (threadIdx.x < 9) {
        a.part[9 * (size_t)blockIdx.x + threadIdx.x] = part;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // at most 148 block sums: a warp per component, in a fixed order (components 0..7, then 8)
    __threadfence();
    for (int k = threadIdx.x >> 5; k < 9; k += 8) {
        double t = 0.0;
        for (unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32) t += __ldcg(a.part + 9 * (size_t)b + k);
        t = tet::warp_sum(t);
        if ((threadIdx.x & 31) == 0) a.kappa[k] = KW_MK * (1.0 / (double(a.nq) * a.vol)) * t;
    }
    if (threadIdx.x == 0) *a.ticket = 0;
}

// Time-reversal set on the host from the grid addresses.
int build_tr_set(spring_ctx* c) {
    const int nq = c->nq;
    std::vector<int> qint((size_t)nq * 3);
    SPRING_CHECK(d2h(c, qint.data(), c->d_qint.p, sizeof(int) * qint.size(), "grid addresses"));
    auto gidx = [&](int x, int y, int z) {
        auto m = [](int a, int n) { int r = a % n; return r < 0 ? r + n : r; };
        return m(x, c->mesh[0]) + c->mesh[0] * (m(y, c->mesh[1]) + c->mesh[1] * m(z, c->mesh[2]));
    };
    std::vector<int> neg(nq), rep(nq);
    for (int q = 0; q < nq; ++q) {
        neg[q] = gidx(-qint[3 * q], -qint[3 * q + 1], -qint[3 * q + 2]);
        rep[q] = std::min(q, neg[q]);
    }
    std::vector<int> grid;
    for (int q = 0; q < nq; ++q)
        if (rep[q] == q) grid.push_back(q);
    const int ntr = (int)grid.size();
    std::vector<int> slot(nq, -1), pos(nq), sgn(nq), deg(ntr, 0), tint((size_t)ntr * 3);
    for (int i = 0; i < ntr; ++i) {
        slot[grid[i]] = i;
        for (int d = 0; d < 3; ++d) tint[3 * i + d] = qint[3 * grid[i] + d];
    }
    for (int q = 0; q < nq; ++q) {
        pos[q] = slot[rep[q]];
        sgn[q] = q == rep[q] ? 1 : -1;
        deg[pos[q]] += 1;
    }
    SPRING_CHECK(dalloc(c, c->d_tr_int, tint.size(), "time-reversal set"));
    SPRING_CHECK(dalloc(c, c->d_tr_grid, ntr, "time-reversal set"));
    SPRING_CHECK(dalloc(c, c->d_tr_pos, nq, "time-reversal set"));
    SPRING_CHECK(dalloc(c, c->d_tr_sgn, nq, "time-reversal set"));
    SPRING_CHECK(dalloc(c, c->d_tr_deg, ntr, "time-reversal set"));
    SPRING_CHECK(dalloc(c, c->d_neg, nq, "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_tr_int.p, tint.data(), sizeof(int) * tint.size(), "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_tr_grid.p, grid.data(), sizeof(int) * ntr, "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_tr_pos.p, pos.data(), sizeof(int) * nq, "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_tr_sgn.p, sgn.data(), sizeof(int) * nq, "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_tr_deg.p, deg.data(), sizeof(int) * ntr, "time-reversal set"));
    SPRING_CHECK(h2d(c, c->d_neg.p, neg.data(), sizeof(int) * nq, "time-reversal set"));
    c->ntr = ntr;
    c->ps_tr.n0 = ntr;
    c->ps_tr.q0_int = c->d_tr_int.p;
    c->ps_tr.q0_grid = c->d_tr_grid.p;
    c->ps_tr.done = false;
    return SPRING_OK;
}

// ---------------------------------------------------------------- Gaussian operator
// The iterative BTE with Gaussian delta weights in place of the tetrahedra (build-side form): per
// enumerated pair (q0 of the time-reversal set, q1, q2 = p(q1)) and mode triple with a weight above
// the exp(-40) cut, one operator entry (r0, k1, k2, P, Q); with c = (n1 - n2) P + (1 + n1 + n2) Q,
//   1/tau(r0) = sum c,   dF(r0) = -sum c (F(k1) + F(k2)),
// which is the reference's two channels (TetrahedronWplus / Wminus and TetrahedronIterPlus / Minus,
// Quasi_momentum_consrv.f90:701-1208, TetrahedronDeltaSum.f90:22-607) summed over every grid q1 with
// d(w0 - M): the plus channel at q1 and at q2 gives (n1 - n2) d(w0 + w1 - w2) + (n2 - n1) d(w0 + w2 - w1)
// and the minus channel at -q1 and -q2 gives (1 + n1 + n2) d(w0 - w1 - w2), each times 4 W3 and -(F1 + F2)
// because F(-q) = -F(q).  The entries are sorted by row once and kept in HBM (CSR); an iteration is one
// pass over them.
// Sort keys (row, k1, s2): unique within an operator, so that a rebuilt one has the same order and sums to the
// same bits however its entries were appended.
__global__ void k_bteg_keys(long long cnt, int n, int bits, const s3::BteEntry* __restrict__ e,
                            unsigned long long* __restrict__ key, int* __restrict__ idx) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (long long)gridDim.x * blockDim.x) {
        const s3::BteEntry x = e[i];
        key[i] = ((unsigned long long)x.r0 << bits | (unsigned)x.k1) << 3 | (unsigned)(x.k2 % n);
        idx[i] = (int)i;
    }
}
// The sorted operator, and the first entry of every row (rows without entries included).
__global__ void k_bteg_gather(long long cnt, int rows, int shift, const s3::BteEntry* __restrict__ e,
                              const unsigned long long* __restrict__ key, const int* __restrict__ idx,
                              int* __restrict__ rowoff, int2* __restrict__ kk, double2* __restrict__ pq) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i <= cnt; i += (long long)gridDim.x * blockDim.x) {
        const int r = i < cnt ? (int)(key[i] >> shift) : rows, before = i > 0 ? (int)(key[i - 1] >> shift) : -1;
        for (int k = before + 1; k <= r; ++k) rowoff[k] = (int)i;
        if (i == cnt) continue;
        const s3::BteEntry x = e[idx[i]];
        kk[i] = make_int2(x.k1, x.k2);
        pq[i] = make_double2(x.P, x.Q);
    }
}

// The modes whose F an entry adds up: k1 and k2, or twice k1 where k1 is stored as its complement (e[1] and e[2]
// of bte_entry; their coefficients are halved).
__device__ __forceinline__ int2 bte_legs(int2 k) { return k.x < 0 ? make_int2(~k.x, ~k.x) : k; }

// Row r holds the entries off[r nseg] .. off[(r + 1) nseg].  One block per row: c = (n1 - n2) P + (1 + n1 + n2) Q of
// its entries at one temperature, and their sum, 1/tau.
__global__ void __launch_bounds__(256) k_bteg_coef(int nseg, const int* __restrict__ off, const int2* __restrict__ kk,
                                                  const double2* __restrict__ pq, const double* __restrict__ nbe,
                                                  double* __restrict__ cf, double* __restrict__ inv_tau) {
    __shared__ double red[1][8];
    double v[1] = {0.0};
    const int end = off[((size_t)blockIdx.x + 1) * nseg];
    for (int i = off[(size_t)blockIdx.x * nseg] + threadIdx.x; i < end; i += 256) {
        const int2 k = kk[i];
        const double2 e = pq[i];
        const double n1 = nbe[k.x < 0 ? ~k.x : k.x], n2 = nbe[k.y];
        const double c = (n1 - n2) * e.x + (1.0 + n1 + n2) * e.y;
        cf[i] = k.x < 0 ? 0.5 * c : c;
        if (k.x >= 0) v[0] += c;
    }
    const double t = block_sum<1>(v, red);
    if (threadIdx.x == 0) inv_tau[blockIdx.x] = t;
}

// dF[r] = -sum c (Fg[k1] + Fg[k2]), one block per row (Fg: four doubles per mode, the fourth zero).
__global__ void __launch_bounds__(256) k_bteg_rows(int nseg, const int* __restrict__ off, const int2* __restrict__ kk,
                                                  const double* __restrict__ cf, const double* __restrict__ Fg,
                                                  double* __restrict__ dF) {
    __shared__ double red[3][8];
    double v[3] = {0.0, 0.0, 0.0};
    const int end = off[((size_t)blockIdx.x + 1) * nseg];
    for (int i = off[(size_t)blockIdx.x * nseg] + threadIdx.x; i < end; i += 256) {
        const double c = cf[i];
        const int2 k = bte_legs(kk[i]);
        const double2* f1 = reinterpret_cast<const double2*>(Fg + 4 * (size_t)k.x);
        const double2* f2 = reinterpret_cast<const double2*>(Fg + 4 * (size_t)k.y);
        const double2 u1 = f1[0], v1 = f1[1], u2 = f2[0], v2 = f2[1];
        v[0] -= c * (u1.x + u2.x);
        v[1] -= c * (u1.y + u2.y);
        v[2] -= c * (v1.x + v2.x);
    }
    const double t = block_sum<3>(v, red);
    if (threadIdx.x < 3) dF[3 * (size_t)blockIdx.x + threadIdx.x] = t;
}

// (k1, k2) of every entry as modes of the time-reversal set in 16 bits each (at most 8533 rows fit the shared
// memory), the top bit set where F changes sign.
__global__ void k_bteg_encode(long long cnt, int n, const int2* __restrict__ kk, const int* __restrict__ pos,
                              const int* __restrict__ sgn, unsigned* __restrict__ ke) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (long long)gridDim.x * blockDim.x) {
        const int2 k = bte_legs(kk[i]);
        const int a = k.x / n, b = k.y / n;
        const unsigned x = (pos[a] * n + k.x % n) | (sgn[a] < 0 ? 0x8000 : 0), y = (pos[b] * n + k.y % n) | (sgn[b] < 0 ? 0x8000 : 0);
        ke[i] = x | y << 16;
    }
}

// The same sums with F of the whole time-reversal set in shared memory (24 bytes a mode).  The two gathers of
// an entry are what bounds k_bteg_rows - 64 bytes of L2 traffic beside 16 of operator, about 5 TB/s - and F is
// small: 125 KB at 12^3.  One CTA per SM; a warp takes a quarter of a row, so that uneven rows spread, and
// k_bte_step adds the quarters in order.  12^3 (3.5e6 entries): 45.7 -> 27 us per pass,
// now bound by the bank conflicts of six random 8-byte reads an entry (more unrolling, smaller parts or blocks
// change nothing; entries in k1 order rather than as appended: 31 -> 27).
constexpr int ROW_PARTS = 4, RSM = 1024;
__global__ void __launch_bounds__(RSM, 1) k_bteg_rows_sm(int rows, int nseg, const int* __restrict__ off,
                                                          const unsigned* __restrict__ ke, const double* __restrict__ cf,
                                                          const double* __restrict__ F, double* __restrict__ dF) {
    extern __shared__ double sF[];
    for (int i = threadIdx.x; i < 3 * rows; i += RSM) sF[i] = F[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warps = gridDim.x * (RSM / 32);
    for (int u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < rows * ROW_PARTS; u += warps) {
        const int r = u / ROW_PARTS, part = u % ROW_PARTS;
        const int b = off[(size_t)r * nseg], e = off[((size_t)r + 1) * nseg];
        const int step = ((e - b + ROW_PARTS - 1) / ROW_PARTS + 31) & ~31;
        const int i1 = min(b + (part + 1) * step, e);
        double v0 = 0.0, v1 = 0.0, v2 = 0.0;
#pragma unroll 4
        for (int i = b + part * step + lane; i < i1; i += 32) {
            const double c = cf[i];
            const unsigned k = ke[i];
            const double c1 = k & 0x8000u ? c : -c, c2 = k & 0x80000000u ? c : -c;
            const double* f1 = sF + 3 * (k & 0x7fffu);
            const double* f2 = sF + 3 * (k >> 16 & 0x7fffu);
            v0 += c1 * f1[0] + c2 * f2[0];
            v1 += c1 * f1[1] + c2 * f2[1];
            v2 += c1 * f1[2] + c2 * f2[2];
        }
        for (int o = 16; o > 0; o >>= 1) {
            v0 += __shfl_xor_sync(0xffffffffu, v0, o);
            v1 += __shfl_xor_sync(0xffffffffu, v1, o);
            v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        }
        if (lane < 3) dF[3 * (size_t)u + lane] = lane == 0 ? v0 : (lane == 1 ? v1 : v2);
    }
}

}  // namespace

namespace {

// The loop of main.f90:295-361 at every temperature: tau(T) fills w.inv_tau, df(T) fills w.dF from w.Fg
// (F at the grid modes) or, with several partial sums per row (`parts`), from w.F (F by rows).
// `ahead`: iterations queued before kappa is read back and the convergence test made (iterations past
// the converged one change no output).
template <class Tau, class DF>
int bte_iterate(spring_ctx* c, double eps_k, int max_iter, int ahead, int parts, Tau tau, DF df, double* h_kappa,
                double* h_kappa_rta, int* h_iters) {
    const int n = c->ndof, ntr = c->ntr, nq = c->nq, rows = ntr * n;
    constexpr int MAX_AHEAD = 16;
    const int blocks = std::max(1, std::min((rows + 255) / 256, 148));
    BteWork& w = c->bte;
    // one buffer: Fg | F0 | F | dF | 1/tau | kappa partial sums | kappa of the queued iterations | ticket
    const size_t nFg = (size_t)nq * n * 4, nF = (size_t)rows * 3;
    SPRING_CHECK(dalloc(c, w.vec, nFg + (2 + parts) * nF + rows + (size_t)blocks * 9 + 9 * (MAX_AHEAD + 1) + 1, "BTE vectors"));
    w.Fg = w.vec.p;
    w.F0 = w.Fg + nFg;
    w.F = w.F0 + nF;
    w.dF = w.F + nF;
    w.inv_tau = w.dF + parts * nF;
    double* part = w.inv_tau + rows;
    double* hist = part + (size_t)blocks * 9;
    unsigned* ticket = reinterpret_cast<unsigned*>(hist + 9 * (MAX_AHEAD + 1));
    SPRING_CHECK(zero(c, ticket, sizeof(double), "BTE ticket"));
    auto step = [&](bool init, int T, int at) -> int {
        const StepArgs a{ntr, n, nq, c->vol, c->temps[T], c->d_tr_grid.p, c->d_neg.p, c->d_tr_deg.p, c->ph_grid.omega.p,
                         c->ph_grid.nbe.p + (size_t)T * nq * n, c->ph_grid.vel.p, w.inv_tau, w.dF, parts, w.F0, parts > 1 ? w.F : nullptr,
                         parts > 1 ? nullptr : w.Fg, part, ticket, hist + 9 * at};
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        if (init) k_bte_step<true><<<blocks, 256, 0, c->stream>>>(a);
        else k_bte_step<false><<<blocks, 256, 0, c->stream>>>(a);
        return launch_check(c, init ? "k_bte_step<init>" : "k_bte_step");
    };
    for (int T = 0; T < c->nT; ++T) {
        SPRING_CHECK(tau(T));
        SPRING_CHECK(step(true, T, 0));
        double kap[(MAX_AHEAD + 1) * 9], k0[9], kold[9], knew[9];
        int iter = 0, chunk = std::min(ahead, MAX_AHEAD);
        double dprev = 0.0, d = 0.0;
        for (bool done = false, first = true; !done; first = false) {
            chunk = std::max(1, std::min(chunk, max_iter + 1 - iter));
            for (int k = 1; k <= chunk; ++k) {
                SPRING_CHECK(df(T));
                SPRING_CHECK(step(false, T, k));
            }
            SPRING_CHECK(d2h(c, kap, hist, sizeof(double) * 9 * (chunk + 1), "kappa"));
            if (first) {
                std::copy(kap, kap + 9, k0);
                std::copy(kap, kap + 9, kold);
            }
            for (int k = 1; k <= chunk && !done; ++k) {
                ++iter;
                std::copy(kap + 9 * k, kap + 9 * k + 9, knew);
                dprev = d;
                d = 0.0;
                for (int x = 0; x < 9; ++x) d = std::max(d, std::fabs(knew[x] - kold[x]));
                done = d < eps_k || iter > max_iter;
                if (!done) std::copy(knew, knew + 9, kold);
            }
            if (ahead > 1) {  // the rest at the present rate of convergence
                chunk = ahead;
                if (d > 0.0 && dprev > d) chunk = (int)std::min(double(MAX_AHEAD), std::ceil(std::log(d / eps_k) / std::log(dprev / d)));
            }
        }
        if (h_kappa) std::copy(knew, knew + 9, h_kappa + 9 * T);
        if (h_kappa_rta) std::copy(k0, k0 + 9, h_kappa_rta + 9 * T);
        if (h_iters) h_iters[T] = iter;
    }
    return SPRING_OK;
}

// The iterations over an operator in HBM: `cnt` entries, row r at off[r nseg] .. off[(r + 1) nseg].
int bte_operator_run(spring_ctx* c, int rows, int nseg, const int* off, const int2* kk, const double2* pq, long long cnt,
                     double eps_k, int max_iter, double* h_kappa, double* h_kappa_rta, int* h_iters) {
    BteWork& w = c->bte;
    SPRING_CHECK(dalloc(c, w.cf, std::max<long long>(cnt, 1), "operator coefficients"));
    auto tau = [&](int T) -> int {
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        k_bteg_coef<<<rows, 256, 0, c->stream>>>(nseg, off, kk, pq, c->ph_grid.nbe.p + (size_t)T * c->nq * c->ndof, w.cf.p,
                                                w.inv_tau);
        return launch_check(c, "k_bteg_coef");
    };
    // F in shared memory where it fits beside the block (about 14^3 for a two-atom cell) and the operator is
    // long enough to pay for loading it into every SM
    const size_t smem = sizeof(double) * 3 * rows;
    const bool in_smem = smem <= 200 * 1024 && cnt >= 16 * (long long)rows;
    int sms = 148;
    if (in_smem) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
        allow_smem(k_bteg_rows_sm);
        SPRING_CHECK(dalloc(c, w.ke, cnt, "operator modes"));
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        k_bteg_encode<<<(int)std::min<long long>((cnt + 255) / 256, 148LL * 16), 256, 0, c->stream>>>(
            cnt, c->ndof, kk, c->d_tr_pos.p, c->d_tr_sgn.p, w.ke.p);
        SPRING_CHECK(launch_check(c, "k_bteg_encode"));
    }
    auto df = [&](int) -> int {
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        if (in_smem)
            k_bteg_rows_sm<<<std::min(sms, (rows * ROW_PARTS + RSM / 32 - 1) / (RSM / 32)), RSM, smem, c->stream>>>(rows, nseg, off, w.ke.p,
                                                                                                w.cf.p, w.F, w.dF);
        else
            k_bteg_rows<<<rows, 256, 0, c->stream>>>(nseg, off, kk, w.cf.p, w.Fg, w.dF);
        return launch_check(c, "k_bteg_rows<dF>");
    };
    // A pass over few entries is shorter than the wait for kappa: several are queued per readback.
    const int rc = bte_iterate(c, eps_k, max_iter, cnt < (4 << 20) ? 8 : 1, in_smem ? ROW_PARTS : 1, tau, df, h_kappa, h_kappa_rta, h_iters);
    cudaStreamSynchronize(c->stream);
    if (w.cf.n > (8u << 20)) dfree(w.cf);  // large ones are given back
    if (w.ke.n > (8u << 20)) dfree(w.ke);
    return rc;
}

}  // namespace

int run_bte_gauss(spring_ctx* c, double sigma, double eps_k, int max_iter, double* h_kappa, double* h_kappa_rta,
                  int* h_iters, double* h_stats) {
    if (c->nb != 2 || c->na3 != 7) return fail(c, SPRING_ERR_UNSUPPORTED, "Gaussian iterative kappa: two-atom cells with 7-atom FC3 clusters");
    if (c->ntr == 0) SPRING_CHECK(build_tr_set(c));
    if (!c->ps_tr.done) SPRING_CHECK(run_enumerate3(c, c->ps_tr));
    SPRING_CHECK(pairoff_host(c, c->ps_tr));
    const int n = c->ndof, ntr = c->ntr, nq = c->nq, rows = ntr * n;
    const Q0View view{c->d_tr_int.p, c->d_tr_grid.p, c->ph_grid.evec.p, c->ph_grid.omega.p, c->ph_grid.oneby.p};
    const long long npairs = c->ps_tr.h_pairoff[ntr];
    const int threads = 256;
    auto blocks_for = [&](long long m) { return (int)std::max<long long>(1, std::min<long long>((m + threads - 1) / threads, 148LL * 16)); };
    // ---- the operator: entries, sorted by row (kept until sigma, the phonons or the pairs change)
    if (!(c->bteg_sigma == sigma && c->bteg_gen == c->ph_gen && c->bteg_pairs == c->ps_tr.gen && c->bteg_n > 0 &&
          c->bteg_prec == c->precision)) {
        c->bteg_n = 0;
        BteWork& w = c->bte;
        SPRING_CHECK(dalloc(c, w.ctr, 1, "operator count"));
        SPRING_CHECK(dalloc(c, c->d_bteg_row, rows + 1, "operator rows"));
        constexpr long long EB = sizeof(s3::BteEntry);
        long long cap = std::max<long long>(1 << 20, npairs * 216 / 40);  // the window passes ~1-2% of the triples
        cap = std::max<long long>(cap, w.ent.n / EB);
        long long cnt = 0;
        int rc = SPRING_OK;
        for (int attempt = 0; rc == SPRING_OK && attempt < 2; ++attempt) {
            rc = dalloc(c, w.ent, (size_t)(cap * EB), "BTE operator entries");
            if (rc == SPRING_OK) rc = zero(c, w.ctr.p, sizeof(unsigned long long), "operator count");
            bool handled = false;
            // BF16 / BF16x3 contexts: the tensor-core pass writes the entries; FP64: the FP64 pass
            if (rc == SPRING_OK) rc = run_v3tc_bte(c, 0, ntr, sigma, w.ent.p, w.ctr.p, cap, &handled);
            if (rc == SPRING_OK && !handled)
                rc = launch_v3s_bte(c, c->ps_tr, view, 0, ntr, sigma, w.ent.p, w.ctr.p, cap, &handled);
            unsigned long long h = 0;
            if (rc == SPRING_OK) rc = d2h(c, &h, w.ctr.p, sizeof h, "operator count");
            cnt = (long long)h;
            if (cnt <= cap) break;
            cap = cnt + cnt / 16 + 1024;
        }
        if (rc == SPRING_OK && cnt > cap) rc = fail(c, SPRING_ERR_CUDA, "BTE operator: entry count changed between runs");
        if (rc == SPRING_OK && cnt > 0x7fffffffLL) rc = fail(c, SPRING_ERR_UNSUPPORTED, "BTE operator above 2^31 entries");
        if (rc == SPRING_OK) rc = dalloc(c, c->d_bteg_kk, cnt, "BTE operator");
        if (rc == SPRING_OK) rc = dalloc(c, c->d_bteg_pq, cnt, "BTE operator");
        const auto* ent = reinterpret_cast<const s3::BteEntry*>(w.ent.p);
        int bits = 1;
        while ((1LL << bits) < (long long)nq * n) ++bits;
        int rbits = 1;
        while ((1 << rbits) < rows) ++rbits;
        const int top = bits + 3 + rbits;
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, (unsigned long long*)nullptr, (unsigned long long*)nullptr, (int*)nullptr,
                                        (int*)nullptr, (int)cnt, 0, top, c->stream);
        for (int k = 0; k < 2; ++k) {
            if (rc == SPRING_OK) rc = dalloc(c, w.key[k], cnt, "operator keys");
            if (rc == SPRING_OK) rc = dalloc(c, w.idx[k], cnt, "operator keys");
        }
        if (rc == SPRING_OK) rc = dalloc(c, w.tmp, std::max<size_t>(tb, 1), "operator sort");
        if (rc == SPRING_OK && launch_injected(c)) rc = fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        if (rc == SPRING_OK && cnt > 0) {
            k_bteg_keys<<<blocks_for(cnt), threads, 0, c->stream>>>(cnt, n, bits, ent, w.key[0].p, w.idx[0].p);
            rc = launch_check(c, "k_bteg_keys");
            if (rc == SPRING_OK) {
                const cudaError_t e = cub::DeviceRadixSort::SortPairs(w.tmp.p, tb, w.key[0].p, w.key[1].p, w.idx[0].p,
                                                                      w.idx[1].p, (int)cnt, 0, top, c->stream);
                c->launches += 1;
                if (e != cudaSuccess) rc = cuda_fail(c, e, "operator sort");
            }
        }
        if (rc == SPRING_OK && launch_injected(c)) rc = fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        if (rc == SPRING_OK) {
            k_bteg_gather<<<blocks_for(cnt + 1), threads, 0, c->stream>>>(cnt, rows, bits + 3, ent, w.key[1].p, w.idx[1].p,
                                                                         c->d_bteg_row.p, c->d_bteg_kk.p, c->d_bteg_pq.p);
            rc = launch_check(c, "k_bteg_gather");
        }
        if (w.ent.n > ((size_t)256 << 20)) {  // large ones are given back
            cudaStreamSynchronize(c->stream);
            dfree(w.ent);
            for (int k = 0; k < 2; ++k) {
                dfree(w.key[k]);
                dfree(w.idx[k]);
            }
            dfree(w.tmp);
        }
        if (rc != SPRING_OK) return rc;
        c->bteg_n = cnt;
        c->bteg_sigma = sigma;
        c->bteg_gen = c->ph_gen;
        c->bteg_pairs = c->ps_tr.gen;
        c->bteg_prec = c->precision;
    }
    const long long cnt = c->bteg_n;
    if (h_stats) {
        h_stats[0] = (double)cnt;
        h_stats[1] = (double)npairs;
    }
    return bte_operator_run(c, rows, 1, c->d_bteg_row.p, c->d_bteg_kk.p, c->d_bteg_pq.p, cnt, eps_k, max_iter, h_kappa,
                            h_kappa_rta, h_iters);
}

// The stored tetrahedron operator no longer holds.  A small one's memory serves the next; a large one goes back, so
// that calls which size themselves by the free memory find it.
void bte_stale(spring_ctx* c) {
    c->bt_gen = -1;
    if (c->d_bt_kk.n * sizeof(int2) + c->d_bt_pq.n * sizeof(double2) <= ((size_t)256 << 20)) return;
    dfree(c->d_bt_kk);
    dfree(c->d_bt_pq);
}

int run_bte(spring_ctx* c, double eps_k, int max_iter, double* h_kappa, double* h_kappa_rta, int* h_iters) {
    if (c->ntr == 0) SPRING_CHECK(build_tr_set(c));
    if (!c->ps_tr.done) SPRING_CHECK(run_enumerate3(c, c->ps_tr));
    const int n = c->ndof, ntr = c->ntr, nq = c->nq, rows = ntr * n;
    const size_t slot = (size_t)nq * n * n * n;
    const Q0View view{c->d_tr_int.p, c->d_tr_grid.p, c->ph_grid.evec.p, c->ph_grid.omega.p, c->ph_grid.oneby.p};
    // q0 per batch: their (P, Q) and W grids stay around the L2 size
    const int batch = (int)std::max<size_t>(1, std::min<size_t>(ntr, ((size_t)96 << 20) / (slot * sizeof(double2))));
    BteWork& w = c->bte;
    // W and the tetrahedron weights of q0 b .. b + nb - 1 into d_w and w.pq
    auto build = [&](int b, int nb) -> int {
        SPRING_CHECK(run_v3_wgrid(c, c->ps_tr, view, b, nb, c->d_w.p));
        SPRING_CHECK(zero(c, w.pq.p, sizeof(double2) * slot * nb, "tetrahedron weights"));
        WgtArgs a{};
        a.n = n;
        a.nq = nq;
        a.ntet = 6 * nq;
        a.q0_first = b;
        a.tr_grid = c->d_tr_grid.p;
        a.neg = c->d_neg.p;
        a.partner = c->ps_tr.partner.p;
        a.wf = w.wf.p;
        a.omega = c->ph_grid.omega.p;
        a.pq = w.pq.p;
        const int groups = (a.ntet + 31) / 32, passes = (n + NS0 - 1) / NS0;
        a.nb2 = (n + BS2 - 1) / BS2;
        a.per1 = 6;  // as in k_tetra3: shorter units while the chip is not full
        while (a.per1 > 1 && (long long)groups * a.nb2 * ((n + a.per1 - 1) / a.per1) * nb * passes < 148LL * 32) --a.per1;
        a.nb1 = (n + a.per1 - 1) / a.per1;
        a.units = (long long)groups * a.nb1 * a.nb2;
        const long long cap = std::max<long long>(1, 148LL * 8 / ((long long)nb * passes));
        const dim3 grid((unsigned)std::max<long long>(1, std::min<long long>((a.units + TW - 1) / TW, cap)), nb, passes);
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        k_bte_weights<<<grid, 32 * TW, 0, c->stream>>>(a, reinterpret_cast<const int4*>(c->d_tetra.p));
        return launch_check(c, "k_bte_weights");
    };
    auto row_args = [&](int b) { return RowArgs{n, nq, b, c->ps_tr.partner.p, c->d_neg.p, w.pq.p, c->d_w.p}; };
    bool stored = c->bt_gen == c->ph_gen && c->bt_pairs == c->ps_tr.gen && c->bt_n >= 0;
    const int len = n * n * nq;
    const int nseg = std::max(1, std::min(16, len / 4096));
    int rc = SPRING_OK;
    if (!stored) {
        c->bt_gen = -1;
        rc = dalloc(c, w.wf, (size_t)nq * n, "FP32 frequencies");
        if (rc == SPRING_OK) rc = dalloc(c, c->d_w, slot * batch, "W buffer");
        if (rc == SPRING_OK) rc = dalloc(c, w.pq, slot * batch, "tetrahedron weights");
        if (rc == SPRING_OK) rc = dalloc(c, w.cnt, (size_t)batch * n * nseg + 1, "operator counts");
        if (rc == SPRING_OK) rc = dalloc(c, w.boff, (size_t)batch * n * nseg + 1, "operator counts");
        if (rc == SPRING_OK) rc = dalloc(c, c->d_bt_off, (size_t)rows * nseg + 1, "operator rows");
        if (rc == SPRING_OK && launch_injected(c)) rc = fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
        if (rc == SPRING_OK) {
            k_bte_wf<<<std::min((nq * n + 255) / 256, 148 * 8), 256, 0, c->stream>>>(nq, n, c->ph_grid.omega.p, w.wf.p);
            rc = launch_check(c, "k_bte_wf");
        }
        // entries to store at most; the free memory is asked for only when the kept buffers are too small
        const long long per = sizeof(int2) + sizeof(double2);
        const long long held = (long long)std::min(c->d_bt_kk.n, c->d_bt_pq.n);
        const long long cap_entries = c->bte_max_entries < 0 ? 0x7fffffffLL : c->bte_max_entries;
        long long most = std::min(held, cap_entries);
        bool asked = false;
        long long total = 0;
        stored = true;
        for (int b = 0; rc == SPRING_OK && stored && b < ntr; b += batch) {
            const int nb = std::min(batch, ntr - b), segs = nb * n * nseg;
            if ((rc = build(b, nb)) != SPRING_OK) break;
            if ((rc = zero(c, w.cnt.p + segs, sizeof(int), "operator counts")) != SPRING_OK) break;
            if (launch_injected(c)) { rc = fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure"); break; }
            k_bte_entries<true><<<segs, 256, 0, c->stream>>>(row_args(b), nseg, w.cnt.p, nullptr, 0, 0, nullptr, nullptr, nullptr);
            if ((rc = launch_check(c, "k_bte_entries<count>")) != SPRING_OK) break;
            if ((rc = run_exclusive_scan(c, w.cnt.p, w.boff.p, segs + 1)) != SPRING_OK) break;
            int here = 0;
            if ((rc = d2h(c, &here, w.boff.p + segs, sizeof here, "operator count")) != SPRING_OK) break;
            const long long need = total + here;
            if (need > most && !asked) {
                size_t free_b = 0, total_b = 0;
                cudaMemGetInfo(&free_b, &total_b);
                most = std::max<long long>(held, (long long)(std::min((size_t)40 << 30, free_b / 2) / per));
                most = std::min(most, cap_entries);
                asked = true;
            }
            if (need > most) { stored = false; break; }
            if (need > (long long)std::min(c->d_bt_kk.n, c->d_bt_pq.n)) {
                // room for the remaining rows at the fill seen so far
                const long long done_rows = (long long)(b + nb);
                long long cap = (long long)((double)need * ntr / done_rows * 1.1) + 1024;
                cap = std::max(need, std::min(cap, most));
                DBuf<int2> kk;
                DBuf<double2> pq;
                rc = dalloc(c, kk, cap, "BTE operator");
                if (rc == SPRING_OK) rc = dalloc(c, pq, cap, "BTE operator");
                if (rc == SPRING_OK && total > 0 &&
                    (cudaMemcpyAsync(kk.p, c->d_bt_kk.p, sizeof(int2) * total, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess ||
                     cudaMemcpyAsync(pq.p, c->d_bt_pq.p, sizeof(double2) * total, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess))
                    rc = fail(c, SPRING_ERR_CUDA, "BTE operator copy");
                cudaStreamSynchronize(c->stream);
                if (rc == SPRING_ERR_ALLOC) {  // it does not fit after all
                    dfree(kk);
                    dfree(pq);
                    rc = SPRING_OK;
                    stored = false;
                    break;
                }
                std::swap(kk, c->d_bt_kk);
                std::swap(pq, c->d_bt_pq);
                dfree(kk);
                dfree(pq);
                if (rc != SPRING_OK) break;
            }
            if (launch_injected(c)) { rc = fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure"); break; }
            k_bte_entries<false><<<segs, 256, 0, c->stream>>>(row_args(b), nseg, nullptr, w.boff.p, total, b + nb == ntr,
                                                             c->d_bt_off.p, c->d_bt_kk.p, c->d_bt_pq.p);
            rc = launch_check(c, "k_bte_entries");
            total = need;
        }
        if (rc == SPRING_OK && stored) {
            c->bt_n = total;
            c->bt_gen = c->ph_gen;
            c->bt_pairs = c->ps_tr.gen;
        }
    }
    if (rc == SPRING_OK && stored) {
        rc = bte_operator_run(c, rows, nseg, c->d_bt_off.p, c->d_bt_kk.p, c->d_bt_pq.p, c->bt_n, eps_k, max_iter, h_kappa,
                              h_kappa_rta, h_iters);
    } else if (rc == SPRING_OK) {
        dfree(c->d_bt_kk);
        dfree(c->d_bt_pq);
        c->bt_n = -1;
        auto pass = [&](int mode, int T) -> int {
            for (int b = 0; b < ntr; b += batch) {
                const int nb = std::min(batch, ntr - b);
                SPRING_CHECK(build(b, nb));
                if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "bte: injected launch failure");
                const double* nbe = c->ph_grid.nbe.p + (size_t)T * nq * n;
                if (mode == 0) k_bte_dense<0><<<nb * n, 256, 0, c->stream>>>(row_args(b), nbe, nullptr, w.inv_tau);
                else k_bte_dense<1><<<nb * n, 256, 0, c->stream>>>(row_args(b), nbe, w.Fg, w.dF);
                SPRING_CHECK(launch_check(c, mode == 0 ? "k_bte_dense<tau>" : "k_bte_dense<dF>"));
            }
            return SPRING_OK;
        };
        rc = bte_iterate(c, eps_k, max_iter, 1, 1, [&](int T) { return pass(0, T); }, [&](int T) { return pass(1, T); },
                         h_kappa, h_kappa_rta, h_iters);
    }
    if (w.pq.n * sizeof(double2) > ((size_t)256 << 20)) {  // one q0 of a large cell
        cudaStreamSynchronize(c->stream);
        dfree(w.pq);
    }
    return rc;
}

}  // namespace spring
