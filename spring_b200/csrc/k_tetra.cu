// Linear-tetrahedron delta sums on the device.
//
// 3-phonon: CalculateLwTetrahedron (src/Kappa/Src/ThirdOrder_m.f90:169-275)
// with FindFandOmegaAtVertices / FindgAndIver / my_sort / FindIverxFver
// (src/Kappa/Src/TetrahedronIntegration_m.f90:18-295).
// Isotope: CalculateIsoW + CalculateIsoLwTetra (src/Kappa/Src/IsotopicScatter.f90:36-168),
// and a Gaussian form delta(omega0 - omega1).
//
// Nearly every (tetrahedron, s0, s1, s2) misses: at 16^3 about 2 % of the energies w0 lie inside a
// tetrahedron's range.  So each warp screens 32 tetrahedra at a time in FP32 (range of the vertex
// energies against the w0 of the pass, widened by far more than the rounding), queues the hits in
// shared memory, and evaluates them 32 at a time in FP64 with the exact bounds: no lane idles through
// another lane's divisions.  Screening reads single-precision frequencies and the evaluation reads mode
// records (n(T), w), both laid out [s][q] so that a warp's neighbouring tetrahedra share cache lines.
// With the same branch window on both legs the sums use the partner map's symmetry: p maps the
// tetrahedra onto themselves and swaps the legs, W with them, so channel 3 equals channel 2 (weight 2)
// and channel 1 needs s1 <= s2 only (weight 2 off the diagonal).  W is stored both ways round for a pair of
// different points; where q1 = p(q1) (at most eight points) W(s1, s2) equals W(s2, s1) only for FC3 that is
// symmetric in its two neighbours, so the fold takes their mean there.
// Case bounds and formulas follow the reference; the summation order differs (per-lane sums, then
// warp/CTA reduction).
// Roofline: issue (the screen) and the FP64 pipe (the evaluation); W is read from the L2-resident grid.
// Two-atom cell, three temperatures, every irreducible q0: 16^3 140.7 -> 2.2 ms, 24^3 1135 -> 17.8 ms
// against one thread per (tetrahedron, s1, s2) that ran every weight formula any lane of its warp needed.
// Three blocks per SM (170 registers) beat four and five (17.8, 18.3, 19.3 ms at 24^3): the evaluation
// waits on dependent loads, and more of them in flight per lane help more than more warps.
#include "spring_internal.cuh"
#include "tetra.cuh"

namespace spring {
namespace {

constexpr int NS0 = 6;   // s0 values per pass
constexpr int BS2 = 6;   // s2 values of a unit, held in shared memory
constexpr int TW = 4;    // warps per block

struct TetArgs {
    int n, nq, nq0, nT, ntet;
    int q0_first;
    int lo0, hi0;        // s0 window
    int lo1, hi1, lo2, hi2;
    int per1;            // s1 values of a unit
    int nb1, nb2;        // s1 and s2 blocks
    long long units;     // (32-tetrahedron group, s1 block, s2 block) of one slot
};

// Doubles of a mode record: n(T), w, padded to an even number.
__host__ __device__ constexpr int rec_size(int nt) { return (nt + 2) / 2 * 2; }

// Table of `rows` grid (or path) points, [slot][s][q]: records of `rs` doubles (n(T), 0, w), and behind
// them FP32 w.
__global__ void k_tet_tables(int n, int nq, int nT, int rs, long long rows, const double* __restrict__ om,
                             const double* __restrict__ nbe, double* __restrict__ rec) {
    float* wf = reinterpret_cast<float*>(rec + rows * n * rs);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows * n;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / n;
        const int s = (int)(i % n);
        const long long o = (row / nq * n + s) * nq + row % nq;
        const double w = om[i];
        wf[o] = (float)w;
        double* r = rec + o * rs;
        for (int t = 0; t < rs - 1; ++t) r[t] = t < nT ? nbe[(long long)t * rows * n + i] : 0.0;
        r[rs - 1] = w;
    }
}

template <int NT>
struct TetSmem {
    double acc[TW][NS0 * (NT + 1)][32];  // per-lane sums
    unsigned queue[TW][32 * 24 + 32];
    float o2[TW][BS2][4][32];  // second-leg frequencies of the unit
    double w0[NS0];
};

// Q2TAB = false: kappa.x, the q2 of vertex q1 is the grid partner p(q1) of this q0.
// Q2TAB = true: LineWidth.x path mode, the q2 phonons of vertex q1 come from a per-q1 table
// (omega_q2All / nBE_q2All of Linewidth_m.f90:48-231) of this slot.
// SYM: both legs have the same branch window (never in path mode).
template <int NT, bool STRICT, bool Q2TAB, bool SYM>
__global__ void __launch_bounds__(32 * TW, 3) k_tetra3(TetArgs a, const int4* __restrict__ tet,
                                                    const int* __restrict__ partner, const double* __restrict__ wgrid,
                                                    const double* __restrict__ om0, const double* __restrict__ rec1,
                                                    const double* __restrict__ rec2, long long rows2,
                                                    double* __restrict__ out_lw, double* __restrict__ out_p3) {
    constexpr int RS = rec_size(NT), NCH = SYM ? 2 : 3, NP = SYM ? 2 : 1, PER = NCH * NS0, K = NP * PER;
    constexpr int NPLANE = K < 16 ? 4 : 5;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TetSmem<NT>& S = *reinterpret_cast<TetSmem<NT>*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = blockIdx.y, q0 = a.q0_first + slot;
    const int s0a = a.lo0 + blockIdx.z * NS0, s0n = min(NS0, a.hi0 - s0a + 1);
    const int n = a.n, nq = a.nq;
    const int n3 = n * n * n;
    const int* __restrict__ part = Q2TAB ? nullptr : partner + (size_t)q0 * nq;
    const size_t off2 = Q2TAB ? (size_t)slot * n * nq : 0;
    const float* __restrict__ wf1 = reinterpret_cast<const float*>(rec1 + (size_t)nq * n * RS);
    const float* __restrict__ f2 = reinterpret_cast<const float*>(rec2 + rows2 * n * RS) + off2;
    const double* __restrict__ r2 = rec2 + off2 * RS;
    const double* __restrict__ W = wgrid + (size_t)slot * nq * n3 + (size_t)s0a * n * n;
    for (int i = lane; i < NS0 * (NT + 1) * 32; i += 32) (&S.acc[warp][0][0])[i] = 0.0;
    if (threadIdx.x < NS0) S.w0[threadIdx.x] = threadIdx.x < s0n ? om0[(size_t)q0 * n + s0a + threadIdx.x] : 0.0;
    __syncthreads();
    float w0[NS0];
#pragma unroll
    for (int i = 0; i < NS0; ++i) w0[i] = (float)S.w0[i];
    unsigned live = 0;  // checks of existing s0
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (k % NS0 < s0n) live |= 1u << (K - 1 - k);
    double(*acc)[32] = S.acc[warp];
    unsigned* queue = S.queue[warp];
    float(*o2s)[4][32] = S.o2[warp];  // a lane reads back only what it wrote

    const long long stride = (long long)gridDim.x * TW;
    for (long long u = (long long)blockIdx.x * TW + warp; u < a.units; u += stride) {
        const int b2 = (int)(u % a.nb2), b1 = (int)(u / a.nb2 % a.nb1), g = (int)(u / ((long long)a.nb2 * a.nb1));
        const int s1a = a.lo1 + b1 * a.per1, s1e = min(s1a + a.per1 - 1, a.hi1);
        const int s2a = a.lo2 + b2 * BS2, s2n = min(BS2, a.hi2 - s2a + 1);
        const bool on = g * 32 + lane < a.ntet;
        const int4 tv = on ? tet[g * 32 + lane] : make_int4(0, 0, 0, 0);
        const int v1[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int v2 = Q2TAB ? v1[v] : part[v1[v]];
#pragma unroll
            for (int k = 0; k < BS2; ++k) o2s[k][v][lane] = k < s2n ? f2[(size_t)(s2a + k) * nq + v2] : 0.0f;
        }

        // FP64 evaluation of one queued hit: lane of the tetrahedron | s1 | s2 | check
        auto evaluate = [&](unsigned code) {
            const int tl = code & 31, s1 = (code >> 5) & 31, s2b = (code >> 10) & 31;
            const int k = K - 1 - (int)(code >> 15);
            const int s2 = s2b + k / PER, ch = k % PER / NS0, si = k % NS0;
            const int4 t = tet[g * 32 + tl];
            int x1[4] = {t.x, t.y, t.z, t.w}, x2[4];
            const double* __restrict__ ra = rec1 + (size_t)s1 * nq * RS;
            const double* __restrict__ rb = r2 + (size_t)s2 * nq * RS;
            double M[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                x2[v] = Q2TAB ? x1[v] : part[x1[v]];
                const double p = ra[(size_t)x1[v] * RS + RS - 1], q = rb[(size_t)x2[v] * RS + RS - 1];
                M[v] = ch == 0 ? p + q : (ch == 1 ? q - p : p - q);
            }
            tet::sort4_carry(M, x1, x2);
            double gw, A[4];
            if (!tet::g_weights<STRICT>(S.w0[si], M, gw, A)) return;
            const double f = SYM ? (ch == 0 && s1 == s2 ? 1.0 : 2.0) : 1.0;
            const double sg = !SYM && ch == 2 ? -1.0 : f;
            const int col = (si * n + s1) * n + s2;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double* w = W + (size_t)x1[v] * n3;
                double wv = w[col];
                if (SYM && x1[v] == x2[v]) wv = 0.5 * (wv + w[(si * n + s2) * n + s1]);  // see the note on the fold
                A[v] *= sg * wv;
            }
            double(*o)[32] = acc + si * (NT + 1);
            o[NT][lane] += f * gw;
#pragma unroll
            for (int T0 = 0; T0 < NT; T0 += 2) {  // records are read two doubles at a time
                if (T0 >= a.nT) break;
                double sa = 0.0, sb = 0.0;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const double2 na = *reinterpret_cast<const double2*>(ra + (size_t)x1[v] * RS + T0);
                    const double2 nb = *reinterpret_cast<const double2*>(rb + (size_t)x2[v] * RS + T0);
                    sa = fma(A[v], ch == 0 ? na.x + nb.x + 1.0 : na.x - nb.x, sa);
                    if (T0 + 1 < NT) sb = fma(A[v], ch == 0 ? na.y + nb.y + 1.0 : na.y - nb.y, sb);
                }
                o[T0][lane] += sa;
                if (T0 + 1 < NT) o[T0 + 1][lane] += sb;
            }
        };

        int qn = 0;
        for (int s1 = s1a; s1 <= s1e; ++s1) {
            float o1[4], e1 = 0.0f;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                o1[v] = wf1[(size_t)s1 * nq + v1[v]];
                e1 += fabsf(o1[v]);
            }
#pragma unroll 1
            for (int kb = 0; kb < s2n; kb += NP) {
                unsigned out = 0;  // one bit per check, set outside (the sign of half width - distance)
#pragma unroll
                for (int kk = 0; kk < NP; ++kk) {
                    const int k = kb + kk;
                    const float q0f = o2s[k][0][lane], q1f = o2s[k][1][lane], q2f = o2s[k][2][lane], q3f = o2s[k][3][lane];
                    // FP32 rounding of the energies is below 4e-7 of the sum of magnitudes
                    const float margin = 1e-6f * (e1 + (fabsf(q0f) + fabsf(q1f) + fabsf(q2f) + fabsf(q3f)));
                    const float p0 = o1[0] + q0f, p1 = o1[1] + q1f, p2 = o1[2] + q2f, p3 = o1[3] + q3f;
                    const float m0 = q0f - o1[0], m1 = q1f - o1[1], m2 = q2f - o1[2], m3 = q3f - o1[3];
                    const float pl = fminf(fminf(p0, p1), fminf(p2, p3)), ph = fmaxf(fmaxf(p0, p1), fmaxf(p2, p3));
                    const float ml = fminf(fminf(m0, m1), fminf(m2, m3)), mh = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                    const float pm = 0.5f * (pl + ph), pr = fmaf(0.5f, ph - pl, margin);
                    const float mm = 0.5f * (ml + mh), mr = fmaf(0.5f, mh - ml, margin);
#pragma unroll
                    for (int i = 0; i < NS0; ++i)
                        out = __funnelshift_l(__float_as_uint(pr - fabsf(w0[i] - pm)), out, 1);
#pragma unroll
                    for (int i = 0; i < NS0; ++i)
                        out = __funnelshift_l(__float_as_uint(mr - fabsf(w0[i] - mm)), out, 1);
                    if (!SYM)
#pragma unroll
                        for (int i = 0; i < NS0; ++i)
                            out = __funnelshift_l(__float_as_uint(mr - fabsf(w0[i] + mm)), out, 1);
                }
                unsigned in = on ? ~out & live : 0u;
#pragma unroll
                for (int kk = 0; kk < NP; ++kk) {
                    unsigned drop = 0;
                    if (kb + kk >= s2n) drop = (1u << PER) - 1;
                    else if (SYM && s2a + kb + kk < s1) drop = ((1u << NS0) - 1) << NS0;  // channel 1: s1 <= s2
                    in &= ~(drop << ((NP - 1 - kk) * PER));
                }
                const unsigned c = __popc(in);
                unsigned pre = 0, tot = 0;
                const unsigned lt = (1u << lane) - 1;
#pragma unroll
                for (int b = 0; b < NPLANE; ++b) {
                    const unsigned m = __ballot_sync(0xffffffffu, (c >> b) & 1);
                    pre += __popc(m & lt) << b;
                    tot += __popc(m) << b;
                }
                if (tot == 0) continue;
                const unsigned base = lane | s1 << 5 | (s2a + kb) << 10;
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
    // reduce: the block's warps and lanes, then global
    __syncthreads();
    for (int i = warp; i < NS0 * (NT + 1); i += TW) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < TW; ++w) v += S.acc[w][i][lane];
        v = tet::warp_sum(v);
        const int si = i / (NT + 1), T = i % (NT + 1);
        if (lane != 0 || si >= s0n || v == 0.0) continue;
        if (T < NT) {
            if (T < a.nT) atomicAdd(&out_lw[((size_t)T * a.nq0 + q0) * n + s0a + si], v);
        } else {
            atomicAdd(&out_p3[(size_t)q0 * n + s0a + si], v);
        }
    }
}

// ---- isotope ------------------------------------------------------------
// W_iso(s1,s0,q1) = pi w0(s0)^2 / 2 / Nq * sum_b g2(b) |e1(b,s1)^H e0(b,s0)|^2.  One thread per (s1, q1) with
// q1 along the warp forms it for NS0 values of s0, e0 in shared memory.  The Gaussian form weights it with
// the delta at once; most (s0, s1) bands are further apart than the delta reaches for all 32 points, and the
// warp skips them.  The tetrahedron form stores it as [slot][s0][s1][q1], where the vertices of neighbouring
// tetrahedra share cache lines (forming it per vertex in the evaluation gathered 96 bytes a vertex: 5.7 ms).
// Sums stay in registers or per-lane words until the block's end; one shared atomic per term had made the
// kernels 26 ms (tetrahedron) and 4.2 ms (Gaussian) per call at 24^3, two-atom cell.  Now 4.3 ms and
// 1.0 ms; 16^3: 3.4 -> 0.53 ms and 0.47 -> 0.12 ms.
struct IsoArgs {
    int n, nb, nq, nq0, nT, ntet;
    int q0_first, per;  // per: 32-tetrahedron groups of a unit (at most 8)
    double scale, os, os2;
    double g2[MAX_NB];
};
constexpr int ISW = 4;  // warps per block

__device__ __forceinline__ double iso_pref(const IsoArgs& a, double acc, double w0) {
    return acc * a.scale * (w0 * w0) * 0.5 / double(a.nq);
}

// GAUSS: out is the rate; else the W grid of the slots.
template <bool GAUSS>
__global__ void __launch_bounds__(32 * ISW) k_iso_w(IsoArgs a, const double2* __restrict__ ev0,
                                                    const double* __restrict__ om0, const double2* __restrict__ evg,
                                                    const double* __restrict__ omg, double* __restrict__ out) {
    __shared__ double2 e0[NS0 * MAX_NDOF];
    __shared__ double red[ISW][NS0], w0s[NS0];
    const int n = a.n, q0 = a.q0_first + blockIdx.y, s0a = blockIdx.z * NS0, s0n = min(NS0, n - s0a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < NS0 * n; i += blockDim.x)
        e0[i] = i < s0n * n ? ev0[((size_t)q0 * n + s0a) * n + i] : make_double2(0.0, 0.0);
    if (threadIdx.x < NS0) w0s[threadIdx.x] = threadIdx.x < s0n ? om0[(size_t)q0 * n + s0a + threadIdx.x] : 0.0;
    __syncthreads();
    double sum[NS0];
#pragma unroll
    for (int i = 0; i < NS0; ++i) sum[i] = 0.0;
    const int chunks = (a.nq + 31) / 32;
    for (int u = blockIdx.x * ISW + warp; u < chunks * n; u += gridDim.x * ISW) {
        const int s1 = u / chunks, q1 = u % chunks * 32 + lane;
        const bool on = q1 < a.nq;
        const size_t it = (size_t)(on ? q1 : 0) * n + s1;
        const double w1 = omg[it];
        const double2* e1 = evg + it * n;
        double W[NS0], x[NS0];
        unsigned near = 0;  // s0 with a lane whose exp does not underflow to 0 (a NaN counts)
#pragma unroll
        for (int i = 0; i < NS0; ++i) {
            W[i] = 0.0;
            const double d = w0s[i] - w1;
            x[i] = -0.5 * a.os2 * d * d;
            if (!GAUSS || __any_sync(0xffffffffu, on && !(x[i] <= -745.2))) near |= 1u << i;
        }
        if (near == 0) continue;
        for (int b = 0; b < a.nb; ++b) {
            const double2 p0 = e1[3 * b], p1 = e1[3 * b + 1], p2 = e1[3 * b + 2];
            const double g = a.g2[b];
#pragma unroll
            for (int i = 0; i < NS0; ++i) {
                if (!(near >> i & 1)) continue;
                const double2* y = e0 + i * n + 3 * b;
                double dr = 0.0, di = 0.0;  // conj(e1) * e0
                dr += p0.x * y[0].x + p0.y * y[0].y;
                di += p0.x * y[0].y - p0.y * y[0].x;
                dr += p1.x * y[1].x + p1.y * y[1].y;
                di += p1.x * y[1].y - p1.y * y[1].x;
                dr += p2.x * y[2].x + p2.y * y[2].y;
                di += p2.x * y[2].y - p2.y * y[2].x;
                W[i] += g * (dr * dr + di * di);
            }
        }
#pragma unroll
        for (int i = 0; i < NS0; ++i)
            if (GAUSS) {
                if ((near >> i & 1) && on) sum[i] += iso_pref(a, W[i], w0s[i]) * a.os * ONEBYSQRT2PI * exp(x[i]);
            } else if (on && i < s0n) {
                out[(((size_t)blockIdx.y * n + s0a + i) * n + s1) * a.nq + q1] = iso_pref(a, W[i], w0s[i]);
            }
    }
    if (!GAUSS) return;
#pragma unroll
    for (int i = 0; i < NS0; ++i) {
        const double v = tet::warp_sum(sum[i]);
        if (lane == 0) red[warp][i] = v;
    }
    __syncthreads();
    if (threadIdx.x < s0n) {
        double v = 0.0;
        for (int w = 0; w < ISW; ++w) v += red[w][threadIdx.x];
        if (v != 0.0)
            for (int T = 0; T < a.nT; ++T) atomicAdd(&out[((size_t)T * a.nq0 + q0) * n + s0a + threadIdx.x], v);
    }
}

// Tetrahedron: warps screen 32 tetrahedra for four s1 at a time and evaluate the queued hits, as k_tetra3.
__global__ void __launch_bounds__(32 * ISW, 4) k_iso_tetra(IsoArgs a, const int4* __restrict__ tet,
                                                           const double* __restrict__ wiso,
                                                           const double* __restrict__ om0,
                                                           const double* __restrict__ omg, double* __restrict__ out) {
    constexpr int S1B = 4, K = S1B * NS0;
    __shared__ double acc_[ISW][NS0][32], w0s[NS0];
    __shared__ unsigned queue_[ISW][32 * K + 32];
    const int n = a.n, q0 = a.q0_first + blockIdx.y, s0a = blockIdx.z * NS0, s0n = min(NS0, n - s0a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double(*acc)[32] = acc_[warp];
    unsigned* queue = queue_[warp];
    const double* __restrict__ Wi = wiso + ((size_t)blockIdx.y * n + s0a) * n * a.nq;
    if (threadIdx.x < NS0) w0s[threadIdx.x] = threadIdx.x < s0n ? om0[(size_t)q0 * n + s0a + threadIdx.x] : 0.0;
#pragma unroll
    for (int i = 0; i < NS0; ++i) acc[i][lane] = 0.0;
    __syncthreads();
    float w0[NS0];
#pragma unroll
    for (int i = 0; i < NS0; ++i) w0[i] = (float)w0s[i];
    const int groups = (a.ntet + 31) / 32, nb1 = (n + S1B - 1) / S1B, blocks = (groups + a.per - 1) / a.per;
    const long long units = (long long)blocks * nb1;
    for (long long u = (long long)blockIdx.x * ISW + warp; u < units; u += (long long)gridDim.x * ISW) {
        const int t0 = (int)(u / nb1) * a.per * 32, s1a = (int)(u % nb1) * S1B;
        auto evaluate = [&](unsigned code) {
            const int k = K - 1 - (int)(code >> 8), s1 = s1a + k / NS0, si = k % NS0;
            const int4 t = tet[t0 + (code & 255)];
            int x[4] = {t.x, t.y, t.z, t.w}, unused[4] = {0, 0, 0, 0};
            double M[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) M[v] = omg[(size_t)x[v] * n + s1];
            tet::sort4_carry(M, x, unused);
            double gw, A[4], s = 0.0;
            if (!tet::g_weights<false>(w0s[si], M, gw, A)) return;
            const double* w = Wi + ((size_t)si * n + s1) * a.nq;
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if (!isnan(A[v])) s += A[v] * w[x[v]];  // undefined weights count as zero
            acc[si][lane] += s;
        };
        unsigned qn = 0;
        for (int gi = 0; gi < a.per && t0 + gi * 32 < a.ntet; ++gi) {
            const bool on = t0 + gi * 32 + lane < a.ntet;
            const int4 tv = on ? tet[t0 + gi * 32 + lane] : make_int4(0, 0, 0, 0);
            unsigned out_bits = 0;  // one bit per check, set outside
#pragma unroll
            for (int k = 0; k < S1B; ++k) {
                const bool have = on && s1a + k < n;
                const int s1 = have ? s1a + k : 0;
                const float m0 = (float)omg[(size_t)tv.x * n + s1], m1 = (float)omg[(size_t)tv.y * n + s1],
                            m2 = (float)omg[(size_t)tv.z * n + s1], m3 = (float)omg[(size_t)tv.w * n + s1];
                const float lo = fminf(fminf(m0, m1), fminf(m2, m3)), hi = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                const float mid = 0.5f * (lo + hi);
                const float half = fmaf(0.5f, hi - lo, 1e-6f * (fabsf(m0) + fabsf(m1) + fabsf(m2) + fabsf(m3)));
#pragma unroll
                for (int i = 0; i < NS0; ++i)
                    out_bits = __funnelshift_l(have && i < s0n ? __float_as_uint(half - fabsf(w0[i] - mid)) : 0x80000000u,
                                               out_bits, 1);
            }
            unsigned in = ~out_bits & ((1u << K) - 1);
            const unsigned c = __popc(in);
            unsigned pos = 0, tot = 0;
            const unsigned lt = (1u << lane) - 1;
#pragma unroll
            for (int b = 0; b < 5; ++b) {
                const unsigned m = __ballot_sync(0xffffffffu, (c >> b) & 1);
                pos += __popc(m & lt) << b;
                tot += __popc(m) << b;
            }
            pos += qn;
            while (in) {
                const int b = __ffs(in) - 1;
                in &= in - 1;
                queue[pos++] = lane | gi << 5 | b << 8;
            }
            qn += tot;
            __syncwarp();
            while (qn >= 32) {
                qn -= 32;
                evaluate(queue[qn + lane]);
            }
            __syncwarp();
        }
        if (lane < qn) evaluate(queue[lane]);
        __syncwarp();
    }
    __syncthreads();
    for (int i = warp; i < s0n; i += ISW) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < ISW; ++w) v += acc_[w][i][lane];
        v = tet::warp_sum(v);
        if (lane == 0 && v != 0.0)
            for (int T = 0; T < a.nT; ++T) atomicAdd(&out[((size_t)T * a.nq0 + q0) * n + s0a + i], v);
    }
}

template <int NT, bool STRICT, bool Q2TAB, bool SYM>
int launch_one(spring_ctx* c, const TetArgs& a, dim3 grid, const double* d_w, const int* part, const double* om0,
               const double* rec2, long long rows2, double* d_lw, double* d_p3) {
    const size_t smem = sizeof(TetSmem<NT>);
    auto kern = k_tetra3<NT, STRICT, Q2TAB, SYM>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "tetra3: injected launch failure");
    kern<<<grid, 32 * TW, smem, c->stream>>>(a, reinterpret_cast<const int4*>(c->d_tetra.p), part, d_w, om0,
                                             c->d_tet_tab.p, rec2, rows2, d_lw, d_p3);
    return launch_check(c, Q2TAB ? "k_tetra3<path>" : "k_tetra3");
}

template <bool STRICT, bool Q2TAB>
int launch_tetra3(spring_ctx* c, TetArgs a, int n_q0, const Pol& pol, const double* d_w, const int* part,
                  const double* om0, const double* rec2, long long rows2, double* d_lw, double* d_p3) {
    if (c->nT > 9)
        return fail(c, SPRING_ERR_UNSUPPORTED, "tetrahedron integration supports at most 9 temperatures per call");
    a.lo0 = pol.lo[0];
    a.hi0 = pol.hi[0];
    a.lo1 = pol.lo[1];
    a.hi1 = pol.hi[1];
    a.lo2 = pol.lo[2];
    a.hi2 = pol.hi[2];
    a.nb2 = (a.hi2 - a.lo2 + BS2) / BS2;
    const int n1 = a.hi1 - a.lo1 + 1, groups = (a.ntet + 31) / 32, passes = (a.hi0 - a.lo0 + NS0) / NS0;
    // Units are as long as the chip stays full (16 resident warps per SM): the s2 frequencies are
    // loaded, and the queue's tail evaluated, once per unit.
    a.per1 = 6;
    while (a.per1 > 1 && (long long)groups * a.nb2 * ((n1 + a.per1 - 1) / a.per1) * n_q0 * passes < 148LL * 32) --a.per1;
    a.nb1 = (n1 + a.per1 - 1) / a.per1;
    a.units = (long long)groups * a.nb1 * a.nb2;
    const long long cap = std::max<long long>(1, 148LL * 8 / ((long long)n_q0 * passes));
    const dim3 grid((unsigned)std::max<long long>(1, std::min<long long>((a.units + TW - 1) / TW, cap)), n_q0, passes);
    const bool sym = !Q2TAB && a.lo1 == a.lo2 && a.hi1 == a.hi2;
#define SPRING_T3(NT)                                                                                                 \
    return sym ? launch_one<NT, STRICT, Q2TAB, !Q2TAB>(c, a, grid, d_w, part, om0, rec2, rows2, d_lw, d_p3)             \
               : launch_one<NT, STRICT, Q2TAB, false>(c, a, grid, d_w, part, om0, rec2, rows2, d_lw, d_p3)
    if (c->nT == 1) SPRING_T3(1);
    if (c->nT <= 3) SPRING_T3(3);
    SPRING_T3(9);
#undef SPRING_T3
}

// Record size of a context's tables: the kernel variant its temperature count selects.
int tet_rs(const spring_ctx* c) { return rec_size(c->nT == 1 ? 1 : (c->nT <= 3 ? 3 : 9)); }

int build_tables(spring_ctx* c, long long rows, const double* om, const double* nbe, double* rec) {
    const int threads = 256;
    const int blocks = (int)std::min<long long>((rows * c->ndof + threads - 1) / threads, 148LL * 16);
    if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "tetra3: injected launch failure");
    k_tet_tables<<<blocks, threads, 0, c->stream>>>(c->ndof, c->nq, c->nT, tet_rs(c), rows, om, nbe, rec);
    return launch_check(c, "k_tet_tables");
}

}  // namespace

// The grid's tables, allocated with the phonons (the no-allocation entry point fills them in place)
// and filled by run_tetra_tables before run_tetra3 / run_tetra3_path.
int alloc_tetra_tables(spring_ctx* c) {
    if (c->nT > 9) return SPRING_OK;  // refused by run_tetra3
    return dalloc(c, c->d_tet_tab, c->nq * tetra_table_doubles(c), "tetrahedron tables");
}

int run_tetra_tables(spring_ctx* c) {
    if (c->nT > 9) return SPRING_OK;
    return build_tables(c, c->nq, c->ph_grid.omega.p, c->ph_grid.nbe.p, c->d_tet_tab.p);
}

// Doubles per table row: ndof records and ndof floats.
size_t tetra_table_doubles(const spring_ctx* c) { return (size_t)c->ndof * (tet_rs(c) + 1); }

int run_tetra3(spring_ctx* c, int q0_first, int n_q0, const double* d_w, const Pol& pol, double* d_lw, double* d_p3) {
    TetArgs a{};
    a.n = c->ndof;
    a.nq = c->nq;
    a.nq0 = c->nq0;
    a.nT = c->nT;
    a.ntet = 6 * c->nq;
    a.q0_first = q0_first;
    return launch_tetra3<false, false>(c, a, n_q0, pol, d_w, c->ps_irr.partner.p, c->ph_irr.omega.p, c->d_tet_tab.p,
                                       c->nq, d_lw, d_p3);
}

int run_tetra3_path(spring_ctx* c, int p_first, int n_slots, int n_path, const double* d_w, const double* om0,
                    const double* om2t, const double* nbe2t, double* tab2, double* d_lw, double* d_scratch) {
    TetArgs a{};
    a.n = c->ndof;
    a.nq = c->nq;
    a.nq0 = n_path;
    a.nT = c->nT;
    a.ntet = 6 * c->nq;
    a.q0_first = p_first;
    SPRING_CHECK(run_tetra_tables(c));
    SPRING_CHECK(build_tables(c, (long long)n_slots * c->nq, om2t, nbe2t, tab2));
    Pol pol;
    for (int k = 0; k < 3; ++k) {
        pol.lo[k] = 0;
        pol.hi[k] = c->ndof - 1;
    }
    return launch_tetra3<true, true>(c, a, n_slots, pol, d_w, nullptr, om0, tab2, (long long)n_slots * c->nq, d_lw, d_scratch);
}

int run_iso(spring_ctx* c, int q0_first, int n_q0, int delta_mode, double sigma, const double* g2, double* d_rate) {
    IsoArgs a{};
    a.n = c->ndof;
    a.nb = c->nb;
    a.nq = c->nq;
    a.nq0 = c->nq0;
    a.nT = c->nT;
    a.ntet = 6 * c->nq;
    a.scale = PI;
    for (int b = 0; b < c->nb; ++b) a.g2[b] = g2[b];
    const bool tetra = delta_mode == SPRING_DELTA_TETRA;
    if (!tetra) {
        a.os = 1.0 / sigma;
        a.os2 = 1.0 / (sigma * sigma);
    }
    const int passes = (c->ndof + NS0 - 1) / NS0;
    const int groups = (a.ntet + 31) / 32, nb1 = (c->ndof + 3) / 4;
    const long long wunits = (long long)((c->nq + 31) / 32) * c->ndof;
    const size_t per = (size_t)c->nq * c->ndof * c->ndof;
    // q0 per launch: the grid's y extent; tetrahedron: a W grid around the L2 size
    int slots = 32768;
    if (tetra) {
        slots = (int)std::max<size_t>(1, std::min<size_t>(slots, ((size_t)64 << 20) / (per * sizeof(double))));
        slots = std::min(slots, n_q0);
        SPRING_CHECK(dalloc(c, c->d_wiso, per * slots, "isotope W"));
    }
    for (int b = 0; b < n_q0; b += slots) {
        const int ns = std::min(slots, n_q0 - b);
        a.q0_first = q0_first + b;
        // one unit a warp until the chip is full, then as few blocks as fill it
        const long long cap = std::max<long long>(1, 148LL * 16 / ((long long)ns * passes));
        const dim3 wgrid((unsigned)std::min((wunits + ISW - 1) / ISW, cap), ns, passes);
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "iso: injected launch failure");
        if (!tetra) {
            k_iso_w<true><<<wgrid, 32 * ISW, 0, c->stream>>>(a, c->ph_irr.evec.p, c->ph_irr.omega.p, c->ph_grid.evec.p,
                                                             c->ph_grid.omega.p, d_rate);
            SPRING_CHECK(launch_check(c, "k_iso_gauss"));
            continue;
        }
        k_iso_w<false><<<wgrid, 32 * ISW, 0, c->stream>>>(a, c->ph_irr.evec.p, c->ph_irr.omega.p, c->ph_grid.evec.p,
                                                          c->ph_grid.omega.p, c->d_wiso.p);
        SPRING_CHECK(launch_check(c, "k_iso_w"));
        a.per = 8;  // long units keep the evaluations full; shorter while the chip is not
        while (a.per > 1 && (long long)(groups + a.per - 1) / a.per * nb1 * ns * passes < 148LL * 32) --a.per;
        const long long units = (long long)((groups + a.per - 1) / a.per) * nb1;
        if (launch_injected(c)) return fail(c, SPRING_ERR_INJECTED, "iso: injected launch failure");
        k_iso_tetra<<<dim3((unsigned)std::min((units + ISW - 1) / ISW, cap), ns, passes), 32 * ISW, 0, c->stream>>>(
            a, reinterpret_cast<const int4*>(c->d_tetra.p), c->d_wiso.p, c->ph_irr.omega.p, c->ph_grid.omega.p, d_rate);
        SPRING_CHECK(launch_check(c, "k_iso_tetra"));
    }
    return SPRING_OK;
}

}  // namespace spring
