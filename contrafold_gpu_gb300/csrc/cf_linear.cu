// cf_linear.cu -- log Z as sums of products instead of log-sum-exp chains.
//
// The log-domain kernels (cf_inside.cuh) spend about 40 instructions (expf,
// log1pf) on every term of a sum, and walk a cell's interior loops one by one.
// Here the tables hold the weights themselves, so a term is one fused
// multiply-add, and the interior-loop sum of a cell
//
//     W(i, j) = sum over l1 + l2 <= 30 of cs(l1, l2) G(i + 1 + l1, j - l2)
//
// (G: inside weight of a pair as seen from a loop around it, 0 where the two
// bases cannot pair) is a dense two-dimensional stencil: for each total length
// t a one-dimensional convolution along the diagonal d - 2 - t.  The last 32
// diagonals of G stay in shared memory; a lane takes four neighbouring cells,
// so that a 16-byte load of G and one of the weights feed 16 multiply-adds.
//
// Range.  A float holds 10^+-38.  Values are scaled by CF_LIN_SCALE per
// position; a sequence any of whose values leaves [lo, hi] (Range below: far
// inside what a float holds, so that no sum has lost a term that counts) is
// put on a list and folded by the log-domain kernel instead (k_inside_redo).
// Random and probed RNAs of up to 512 nt stay inside; a helix of some hundred
// pairs or a sequence whose halves differ by 40 nats does not.
//
// Accuracy (float, GB300, against 64 bits, relative 2-norm): 1e-7, where the
// chains of rounded logarithms have 1.6e-6 at 128 nt and 8e-6 at 50-500 nt.
// Sums run in a fixed order that depends on the length alone, so a sequence's
// result is the same in every batch, mode and schedule.
#include "cf_linear.h"

#include <cmath>
#include <cstddef>

namespace cf {
namespace {

constexpr int kLinWarps = kLinThreads / 32;
constexpr int kRing = 32;      // diagonals of G held: d - 32 .. d - 1
constexpr int kParts = 8;      // partial sums of a cell's stencil
template <typename R>
constexpr int kSplitParts = sizeof(R) == 4 ? 8 : 4;   // and of its splits (double: shared memory)

template <typename R>
struct Range;
template <>
struct Range<float> {
    static __device__ __forceinline__ float lo() { return 1e-28f; }
    static __device__ __forceinline__ float hi() { return 1e20f; }
};
template <>
struct Range<double> {
    static __device__ __forceinline__ double lo() { return 1e-280; }
    static __device__ __forceinline__ double hi() { return 1e200; }
};

template <typename R>
struct LinHead {
    LinWeights<R> w;
    R kp[32];         // CF_LIN_SCALE^t
    int npair[2];     // double: pairable cells of the diagonal (by parity)
    int bad;
};

static_assert(offsetof(LinHead<float>, w) % 16 == 0 && offsetof(LinWeights<float>, csf) % 16 == 0,
              "stencil weights are read as float4");

__host__ __device__ __forceinline__ int lin_code_stride(int L) { return (L + 2 + 15) & ~15; }
__host__ __device__ __forceinline__ int lin_row(int L) { return (L + 48 + 3) & ~3; }    // ring row
__host__ __device__ __forceinline__ int lin_cells(int L) { return (L + 4 + 3) & ~3; }   // partial-sum row

// Dynamic shared memory after the head, in elements of R unless noted
struct LinLayout {
    int gs, cs;
    int G, B, M, W, S, F5, kpow, list, codes, total;   // byte offsets
};
template <typename R>
__host__ __device__ __forceinline__ LinLayout lin_layout(int L) {
    LinLayout Y;
    Y.gs = lin_row(L);
    Y.cs = lin_cells(L);
    int o = (int)((sizeof(LinHead<R>) + 15) & ~size_t(15));
    const int e = (int)sizeof(R);
    Y.G = o; o += kRing * Y.gs * e;
    Y.B = o; o += 4 * Y.gs * e;
    Y.M = o; o += 4 * Y.gs * e;
    Y.W = o; o += kParts * Y.cs * e;
    Y.S = o; o += kSplitParts<R> * Y.cs * e;
    Y.F5 = o; o += Y.cs * e;
    Y.kpow = o; o += Y.cs * e;
    Y.list = o; o += sizeof(R) == 8 ? 2 * Y.cs * 2 : 0;
    o = (o + 15) & ~15;
    Y.codes = o; o += 2 * lin_code_stride(L);
    Y.total = o;
    return Y;
}

// Loop lengths t of stencil part g: lengths t and 32 - t together have 34
// taps, two such pairs a part, and t = 16 alone in the last.
__device__ __forceinline__ int part_len(int g, int k) {
    if (g == 7) return k == 0 ? 16 : 31;
    return k == 0 ? 30 - g : k == 1 ? 23 - g : k == 2 ? 9 + g : 2 + g;
}

// Interior-loop sums of cells i = 1 + 4 q .. 4 + 4 q of diagonal d, part g.
__device__ __forceinline__ void stencil4(const float* __restrict__ G, const LinHead<float>* h, int gs, int d, int q,
                                         int g, float* __restrict__ out) {
    const int tmax = d - 2 < 30 ? d - 2 : 30;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int t = part_len(g, k);
        if (t > tmax) continue;
        const float4* gp = reinterpret_cast<const float4*>(G + ((d - 2 - t) & (kRing - 1)) * gs + 4 + 4 * q);
        const float4* wp = reinterpret_cast<const float4*>(h->w.csf + t * 32);
        float4 x = gp[0];
        float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
        for (int l = 0; l <= t; l += 4) {
            const float4 y = *++gp;
            const float4 w = *wp++;
            b0 = fmaf(w.x, x.x, b0); b1 = fmaf(w.x, x.y, b1); b2 = fmaf(w.x, x.z, b2); b3 = fmaf(w.x, x.w, b3);
            b0 = fmaf(w.y, x.y, b0); b1 = fmaf(w.y, x.z, b1); b2 = fmaf(w.y, x.w, b2); b3 = fmaf(w.y, y.x, b3);
            b0 = fmaf(w.z, x.z, b0); b1 = fmaf(w.z, x.w, b1); b2 = fmaf(w.z, y.x, b2); b3 = fmaf(w.z, y.y, b3);
            b0 = fmaf(w.w, x.w, b0); b1 = fmaf(w.w, y.x, b1); b2 = fmaf(w.w, y.y, b2); b3 = fmaf(w.w, y.z, b3);
            x = y;
        }
        const float kt = h->kp[t];
        a0 = fmaf(kt, b0, a0); a1 = fmaf(kt, b1, a1); a2 = fmaf(kt, b2, a2); a3 = fmaf(kt, b3, a3);
    }
    *reinterpret_cast<float4*>(out + 4 * q) = make_float4(a0, a1, a2, a3);
}

// The same for one pairable cell i in double (the FP64 pipe bounds it, at 2
// multiply-adds a cycle and SM, so only cells that need the sum take part).
__device__ __forceinline__ void stencil1(const double* __restrict__ G, const LinHead<double>* h, int gs, int d, int i,
                                         int g, double* __restrict__ out) {
    const int tmax = d - 2 < 30 ? d - 2 : 30;
    double a = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int t = part_len(g, k);
        if (t > tmax) continue;
        const double* gp = G + ((d - 2 - t) & (kRing - 1)) * gs + 3 + i;
        const double* wp = h->w.csf + t * 32;
        double b0 = 0.0, b1 = 0.0;
        int l = 0;
        for (; l + 1 <= t; l += 2) {
            b0 = fma(wp[l], gp[l], b0);
            b1 = fma(wp[l + 1], gp[l + 1], b1);
        }
        if (l <= t) b0 = fma(wp[l], gp[l], b0);
        a = fma(h->kp[t], b0 + b1, a);
    }
    out[i - 1] = a;
}

// Part q of FM2(i, i + d) = sum over s of FM1(i, i + s) FM(i + s, i + d):
// s = 1 + q, 1 + q + N, ... < d for N parts.
template <typename R, int N>
__device__ __forceinline__ R splits(const R* __restrict__ FM1, const R* __restrict__ FM, int m, int d, int i, int q) {
    // tri_off(s + N) - tri_off(s) = N m - N s - N (N - 1) / 2, smaller by N^2 at each step
    constexpr int T = N * (N - 1) / 2, Q = N * N;
    int s = 1 + q;
    int o1 = tri_off(s, m) + i, o2 = tri_off(d - s, m) + i + s;
    int d1 = N * m - N * s - T, d2 = N * m - N * (d - s - N) - T - N;
    R a = R(0), b = R(0);
    for (; s + 3 * N < d; s += 4 * N) {   // four terms' loads in flight
        const int o1b = o1 + d1, o1c = o1b + d1 - Q, o1d = o1c + d1 - 2 * Q;
        const int o2b = o2 - d2, o2c = o2b - d2 - Q, o2d = o2c - d2 - 2 * Q;
        const R x0 = FM1[o1], y0 = FM[o2], x1 = FM1[o1b], y1 = FM[o2b];
        const R x2 = FM1[o1c], y2 = FM[o2c], x3 = FM1[o1d], y3 = FM[o2d];
        a = fma(x0, y0, a); b = fma(x1, y1, b);
        a = fma(x2, y2, a); b = fma(x3, y3, b);
        o1 = o1d + d1 - 3 * Q; d1 -= 4 * Q;
        o2 = o2d - d2 - 3 * Q; d2 += 4 * Q;
    }
    for (; s < d; s += N) {
        a = fma(FM1[o1], FM[o2], a);
        o1 += d1; d1 -= Q;
        o2 -= d2; d2 += Q;
    }
    return a + b;
}

// Weight of the pair (a, b) closing a multiloop, and of its outer side as a
// branch of one or of the exterior loop (cpu.py:224-228, 237-241).
template <typename R>
__device__ __forceinline__ R w_multi(const LinWeights<R>& w, const int8_t* s, int a, int b) {
    const int x = s[a] * 5 + s[b];
    return w.hc[x] * w.dl[x * 5 + s[a + 1]] * w.dr[x * 5 + s[b - 1]];
}
template <typename R>
__device__ __forceinline__ R w_end(const LinWeights<R>& w, const int8_t* s, int L, int a, int b) {
    const int x = s[b] * 5 + s[a];
    R v = w.hc[x];
    if (b < L) v *= w.dl[x * 5 + s[b + 1]];
    if (a > 1) v *= w.dr[x * 5 + s[a - 1]];
    return v;
}

// Offset of E(a, a + 1): rows a = 1 .. L - 1 of b = a + 1 .. L
__device__ __forceinline__ int e_row(int a, int L) { return (a - 1) * L - ((a * (a - 1)) >> 1); }

template <typename R>
__device__ __forceinline__ void lin_inside(const LinArgs& A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* h = reinterpret_cast<LinHead<R>*>(smem_raw);
    const SeqDesc D = A.descs[blockIdx.x];
    const int L = D.L, m = L + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LinLayout Y = lin_layout<R>(L);
    R* G = reinterpret_cast<R*>(smem_raw + Y.G);
    R* B = reinterpret_cast<R*>(smem_raw + Y.B);
    R* M = reinterpret_cast<R*>(smem_raw + Y.M);
    R* W = reinterpret_cast<R*>(smem_raw + Y.W);
    R* S = reinterpret_cast<R*>(smem_raw + Y.S);
    R* F5 = reinterpret_cast<R*>(smem_raw + Y.F5);
    R* kpow = reinterpret_cast<R*>(smem_raw + Y.kpow);
    int16_t* list = reinterpret_cast<int16_t*>(smem_raw + Y.list);   // double only
    int8_t* s = reinterpret_cast<int8_t*>(smem_raw + Y.codes);
    int8_t* pc = s + lin_code_stride(L);
    const int gs = Y.gs, cs = Y.cs;
    constexpr int SP = kSplitParts<R>;

    // tables in the arena: FM and FM1 by diagonals, E by rows
    R* base = reinterpret_cast<R*>(A.ws + D.ws_off);
    const int64_t tri = pad32(tri_size(L));
    R* FM = base;
    R* FM1 = base + tri;
    R* E = base + 2 * tri;

    {   // weights
        const R* src = static_cast<const R*>(A.weights);
        R* dst = reinterpret_cast<R*>(&h->w);
        for (int k = tid; k < (int)(sizeof(LinWeights<R>) / sizeof(R)); k += kLinThreads) dst[k] = src[k];
    }
    for (int k = tid; k < L + 2; k += kLinThreads) {   // CF_LIN_SCALE^k by repeated squaring
        R p = R(1), b = R(CF_LIN_SCALE);
        for (int e = k; e; e >>= 1, b *= b)
            if (e & 1) p *= b;
        kpow[k] = p;
        if (k < 32) h->kp[k] = p;
    }
    for (int k = L + 2 + tid; k < 32; k += kLinThreads) h->kp[k] = R(0);   // loops longer than the sequence
    for (int k = tid; k < (kRing + 8) * gs; k += kLinThreads) G[k] = R(0);   // and B, M
    if (tid == 0) h->bad = h->npair[0] = h->npair[1] = 0;
    encode_seq(A.seqs, A.mask, D.seq_off, L, s, pc);
    __syncthreads();

    const LinWeights<R>& w = h->w;
    const R muk = w.mu * R(CF_LIN_SCALE), k1 = R(CF_LIN_SCALE), k2 = k1 * k1;
    const R mm = w.mp * w.mb;
    bool bad = false;
    auto check = [&](R v) { bad |= !(v >= Range<R>::lo() && v <= Range<R>::hi()); };
    auto check0 = [&](R v) { bad |= !(v == R(0) || (v >= Range<R>::lo() && v <= Range<R>::hi())); };

    for (int d = 0; d <= L - 2; ++d) {
        const int c = L - 1 - d;   // cells i = 1 .. c
        // partial sums: stencil parts (four cells a lane) and split parts (one cell a lane)
        const int np = sizeof(R) == 8 ? h->npair[d & 1] : 0;
        const int nst = d >= 4 ? kParts * (sizeof(R) == 4 ? (c + 127) >> 7 : (np + 31) >> 5) : 0;
        const int nsp = d >= 4 ? SP * ((c + 31) >> 5) : 0;   // FM1 and FM begin at d = 2
        for (int u = warp; u < nst + nsp; u += kLinWarps) {
            if (u < nst) {
                const int g = u % kParts, q = (u / kParts) * 32 + lane;
                if constexpr (sizeof(R) == 4) {
                    if (4 * q < c) stencil4(G, h, gs, d, q, g, W + g * cs);
                } else {
                    if (q < np) stencil1(G, h, gs, d, list[(d & 1) * cs + q], g, W + g * cs);
                }
            } else {
                const int v = u - nst, g = v % SP, i = 1 + (v / SP) * 32 + lane;
                if (i <= c) S[g * cs + i - 1] = splits<R, SP>(FM1, FM, m, d, i, g);
            }
        }
        __syncthreads();
        R* Gd = G + (d & (kRing - 1)) * gs + 2;
        R* Bd = B + (d & 3) * gs;
        R* Md = M + (d & 3) * gs;
        const R* B2 = B + ((d + 2) & 3) * gs;   // diagonal d - 2
        const R* M2 = M + ((d + 2) & 3) * gs;
        const R* G3 = G + ((d - 3) & (kRing - 1)) * gs + 2;
        const R* G4 = G + ((d - 4) & (kRing - 1)) * gs + 2;
        const int off = tri_off(d, m);
        for (int i = 1 + tid; i <= c + 40; i += kLinThreads) {
            if (i > c) {   // the row of 32 diagonals ago was longer
                if (i + 2 < gs) Gd[i] = R(0);
                continue;
            }
            const int j = i + d;
            R f2 = R(0), fm1 = R(0), fm = R(0);
            if (d >= 4) {
#pragma unroll
                for (int g = 0; g < SP; ++g) f2 += S[g * cs + i - 1];
            }
            if (d >= 2) {
                fm1 = M2[i + 1] * w.mp + FM1[tri_off(d - 1, m) + i + 1] * muk;
                fm = f2 + FM[tri_off(d - 1, m) + i] * muk + fm1;
                check0(fm1);
                check0(fm);
            }
            FM1[off + i] = fm1;
            FM[off + i] = fm;
            R b = R(0), gg = R(0), mm1 = R(0);
            if (pairable_codes(pc[i], pc[j + 1])) {
                const int si = s[i], sj1 = s[j + 1], si1 = s[i + 1], sj = s[j];
                const int key = idx4(si, sj1, si1, sj);
                R win = R(0);
                if (d >= 4) {
#pragma unroll
                    for (int g = 0; g < kParts; ++g) win += W[g * cs + i - 1];
                    win += k2 * w.cs11 * w.i11[si1 * 5 + sj] * G4[i + 2];
                }
                if (d >= 3) win += k1 * (w.cs01 * w.b01[sj] * G3[i + 1] + w.cs10 * w.b01[si1] * G3[i + 2]);
                R fc = w.close[key] * (w.hp[d <= DHP ? d : DHP] * kpow[d] + win);
                if (d >= 2) fc += w.stack[key] * B2[i + 1] + mm * w_multi(w, s, i, j + 1) * f2;
                b = fc * w.bp[si * 5 + sj1] * k2;
                gg = b * w.close[idx4(sj1, si, s[j + 2], s[i - 1])];
                mm1 = b * w_end(w, s, L, i, j + 1);
                check(fc);
                check(b);
                check(gg);
                check(mm1);
            }
            Gd[i] = gg;
            Bd[i] = b;
            Md[i] = mm1;
            E[e_row(i, L) + d] = mm1;   // b - a - 1 = d
        }
        if constexpr (sizeof(R) == 8) {   // pairable cells of the next diagonal
            if (warp == kLinWarps - 1) {
                int n = 0;
                for (int i0 = 1; i0 <= c - 1; i0 += 32) {
                    const int i = i0 + lane;
                    const bool p = i <= c - 1 && pairable_codes(pc[i], pc[i + d + 2]);
                    const unsigned bits = __ballot_sync(0xffffffffu, p);
                    if (p) list[((d + 1) & 1) * cs + n + __popc(bits & ((1u << lane) - 1u))] = (int16_t)i;
                    n += __popc(bits);
                }
                if (lane == 0) h->npair[(d + 1) & 1] = n;
            }
        }
        __syncthreads();
    }

    // exterior: F5[k + 1] = F5[k] eu + sum over a <= k of F5[a - 1] E(a, k + 1) ep.  Thread t keeps the sums of
    // positions t + 1 and t + 1 + kLinThreads; each step adds the newest F5 to all later ones (rows loaded ahead).
    R acc0 = R(0), acc1 = R(0), f = R(1);
    const int j0 = tid + 1, j1 = tid + 1 + kLinThreads;
    const R euk = w.eu * R(CF_LIN_SCALE);
    auto row = [&](int a, int j) -> R { return (a < L && j > a && j <= L) ? E[e_row(a, L) + j - a - 1] : R(0); };
    R n0[4], n1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        n0[u] = row(1 + u, j0);
        n1[u] = L > kLinThreads ? row(1 + u, j1) : R(0);
    }
    if (tid == 0) F5[0] = R(1);
    for (int k0 = 0; k0 < L; k0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u;
            if (k < L) {   // uniform over the CTA
                const R e0 = n0[u], e1 = n1[u];
                n0[u] = row(k + 5, j0);
                if (L > kLinThreads) n1[u] = row(k + 5, j1);
                const R fe = f * w.ep;
                if (j0 == k + 1 || j1 == k + 1) F5[k + 1] = f * euk + (j0 == k + 1 ? acc0 : acc1);
                acc0 = fma(fe, e0, acc0);
                acc1 = fma(fe, e1, acc1);
                __syncthreads();
                f = F5[k + 1];
                check(f);
            }
        }
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) A.fails[1 + atomicAdd(A.fails, 1)] = blockIdx.x;
    } else if (tid == 0) {
        static_cast<R*>(A.logz)[D.idx] = (R)(log((double)f) - (double)L * CF_LIN_LOG_SCALE);
    }
}

template <typename R>
void fill_weights(const double* b, LinWeights<R>* w) {
    auto e = [](double x) { return (R)std::exp(x); };
    for (int k = 0; k < 625; ++k) {
        w->stack[k] = e(b[CF_OFF_STACK + k]);
        w->close[k] = e(b[CF_OFF_HC + k / 25] + b[CF_OFF_TM + k]);
    }
    for (int k = 0; k < 25; ++k) {
        w->bp[k] = e(b[CF_OFF_BP + k]);
        w->hc[k] = e(b[CF_OFF_HC + k]);
        w->i11[k] = e(b[CF_OFF_I11 + k]);
    }
    for (int k = 0; k < 125; ++k) {
        w->dl[k] = e(b[CF_OFF_DL + k]);
        w->dr[k] = e(b[CF_OFF_DR + k]);
    }
    for (int k = 0; k < 32; ++k) w->hp[k] = k <= DHP ? e(b[CF_OFF_HPCUM + k]) : R(0);
    for (int k = 0; k < 8; ++k) w->b01[k] = k < 5 ? e(b[CF_OFF_B01 + k]) : R(0);
    w->mb = e(b[CF_OFF_MB]); w->mu = e(b[CF_OFF_MU]); w->mp = e(b[CF_OFF_MP]);
    w->eu = e(b[CF_OFF_EU]); w->ep = e(b[CF_OFF_EP]);
    auto cs = [&](int l1, int l2) { return e(b[CF_OFF_CS + l1 * 31 + l2]); };
    w->cs01 = cs(0, 1); w->cs10 = cs(1, 0); w->cs11 = cs(1, 1);
    for (int t = 0; t <= CMAX; ++t)
        for (int l = 0; l < 32; ++l)
            w->csf[t * 32 + l] = (t < 2 || l > t || (t == 2 && l == 1)) ? R(0) : cs(l, t - l);
}

}  // namespace

void lin_weights(const double* blob, LinWeights<float>* w) { fill_weights(blob, w); }
void lin_weights(const double* blob, LinWeights<double>* w) { fill_weights(blob, w); }

// 1,000 x 128 nt: see the header of this file for what bounds it
__global__ void __launch_bounds__(kLinThreads, 4) k_lin_inside32(LinArgs A) { lin_inside<float>(A); }
__global__ void __launch_bounds__(kLinThreads, 2) k_lin_inside64(LinArgs A) { lin_inside<double>(A); }

size_t lin_inside_smem_bytes(int Lmax, bool fp64) {
    return fp64 ? lin_layout<double>(Lmax).total : lin_layout<float>(Lmax).total;
}

}  // namespace cf
