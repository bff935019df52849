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
// position; a sequence any of whose values leaves [lo, hi] (Range below) is put
// on a list and folded by the log-domain kernel instead (k_inside_redo).  lo:
// a product that underflowed is below 1e-10 of any sum in range.  hi: a
// derivative that underflowed belongs to a probability below 1e-38 hi = 1e-8.
// Inside stay random RNAs of even composition up to 512 nt.  Helices leave it
// from 50 pairs on (4 of 16 random hairpins with arms of 50 nt, 10 of 55, all of
// 60), GC-rich RNAs with their length (i.i.d., of 8: 60 % GC 1 at 512 nt; 70 % 0
// at 300, 4 at 400, 8 at 512; 80 % 0 at 200, 8 at 300), and a sequence whose
// halves differ by 40 nats.  Those cost what the log domain costs, and the sums
// that were in vain beside it.
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

constexpr int kRing = 32;      // diagonals of G held: d - 32 .. d - 1
constexpr int kParts = 8;      // partial sums of a cell's stencil
template <typename R>
constexpr int kSplitParts = sizeof(R) == 4 ? 8 : 4;   // and of its splits (double: shared memory)

template <typename R>
struct Range;
template <>
struct Range<float> {
    static __device__ __forceinline__ float lo() { return 1e-28f; }
    static __device__ __forceinline__ float hi() { return 1e30f; }
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
};

static_assert(offsetof(LinHead<float>, w) % 16 == 0 && offsetof(LinWeights<float>, csf) % 16 == 0,
              "stencil weights are read as float4");

__host__ __device__ __forceinline__ int lin_code_stride(int L) { return (L + 2 + 15) & ~15; }
__host__ __device__ __forceinline__ int lin_row(int L) { return (L + 48 + 3) & ~3; }    // ring row
__host__ __device__ __forceinline__ int lin_cells(int L) { return (L + 4 + 3) & ~3; }   // partial-sum row

// Dynamic shared memory after the head, in elements of R unless noted
struct LinLayout {
    int gs, cs;
    int G, B, M, W, S, F5, kpow, sig, list, codes, total;   // byte offsets
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
    Y.sig = o; o += Y.cs * e;
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

// sum of x[o1] y[o2] over n terms N diagonals apart in triangular tables:
// tri_off(s + N) - tri_off(s) = N m - N s - N (N - 1) / 2, so both offsets'
// steps d1, d2 shrink by N^2 from term to term.
template <typename R, int N>
__device__ __forceinline__ R dot_tri(const R* __restrict__ x, int o1, int d1, const R* __restrict__ y, int o2, int d2,
                                     int n) {
    constexpr int Q = N * N, U = sizeof(R) == 4 ? 8 : 4;   // terms whose loads are in flight together
    R a = R(0), b = R(0);
    for (; n >= U; n -= U) {
        R xs[U], ys[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            xs[u] = x[o1];
            ys[u] = y[o2];
            o1 += d1 - u * Q;
            o2 += d2 - u * Q;
        }
        d1 -= U * Q;
        d2 -= U * Q;
#pragma unroll
        for (int u = 0; u < U; u += 2) {
            a = fma(xs[u], ys[u], a);
            b = fma(xs[u + 1], ys[u + 1], b);
        }
    }
    for (; n > 0; --n) {
        a = fma(x[o1], y[o2], a);
        o1 += d1; d1 -= Q;
        o2 += d2; d2 -= Q;
    }
    return a + b;
}

// terms 1 + q, 1 + q + N, ... <= most
template <int N>
__device__ __forceinline__ int part_terms(int most, int q) { return most >= 1 + q ? (most - 1 - q) / N + 1 : 0; }

// Part q of FM2(i, i + d) = sum over 0 < s < d of FM1(i, i + s) FM(i + s, i + d).
template <typename R, int N>
__device__ __forceinline__ R splits(const R* __restrict__ FM1, const R* __restrict__ FM, int m, int d, int i, int q) {
    constexpr int T = N * (N - 1) / 2;
    const int s = 1 + q;
    return dot_tri<R, N>(FM1, tri_off(s, m) + i, N * m - N * s - T, FM, tri_off(d - s, m) + i + s,
                         N * (d - s) - N * m - N * N + T + N, part_terms<N>(d - 1, q));
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

// CF_LIN_SCALE^k by repeated squaring
template <typename R>
__device__ __forceinline__ R scale_pow(int k) {
    R p = R(1), b = R(CF_LIN_SCALE);
    for (; k; k >>= 1, b *= b)
        if (k & 1) p *= b;
    return p;
}

// Offset of E(a, a + 1): rows a = 1 .. L - 1 of b = a + 1 .. L
__device__ __forceinline__ int e_row(int a, int L) { return (a - 1) * L - ((a * (a - 1)) >> 1); }

template <typename R, bool TRAIN, int NT>
__device__ __forceinline__ void lin_inside(const LinArgs& A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* h = reinterpret_cast<LinHead<R>*>(smem_raw);
    const SeqDesc D = A.descs[A.first + blockIdx.x];
    const int L = D.L, m = L + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LinLayout Y = lin_layout<R>(L);
    R* G = reinterpret_cast<R*>(smem_raw + Y.G);
    R* B = reinterpret_cast<R*>(smem_raw + Y.B);
    R* M = reinterpret_cast<R*>(smem_raw + Y.M);
    R* W = reinterpret_cast<R*>(smem_raw + Y.W);
    R* S = reinterpret_cast<R*>(smem_raw + Y.S);
    R* F5 = reinterpret_cast<R*>(smem_raw + Y.F5);
    R* kpow = reinterpret_cast<R*>(smem_raw + Y.kpow);
    R* sig = reinterpret_cast<R*>(smem_raw + Y.sig);
    int16_t* list = reinterpret_cast<int16_t*>(smem_raw + Y.list);   // double only
    int8_t* s = reinterpret_cast<int8_t*>(smem_raw + Y.codes);
    int8_t* pc = s + lin_code_stride(L);
    const int gs = Y.gs, cs = Y.cs;
    constexpr int SP = kSplitParts<R>;

    // tables in the arena: FM and FM1 by diagonals, then the pairs' ends E by rows; for gradients FM2 and the pairs
    // by diagonals instead (E is their product with the end weights)
    R* base = reinterpret_cast<R*>(A.ws + D.ws_off);
    const int64_t tri = pad32(tri_size(L));
    R* FM = base;
    R* FM1 = base + tri;
    R* E = base + 2 * tri;
    R* F2 = base + 2 * tri;
    R* Bt = base + 3 * tri;

    {   // weights
        const R* src = static_cast<const R*>(A.weights);
        R* dst = reinterpret_cast<R*>(&h->w);
        for (int k = tid; k < (int)(sizeof(LinWeights<R>) / sizeof(R)); k += NT) dst[k] = src[k];
    }
    for (int k = tid; k < L + 2; k += NT) {
        const R p = scale_pow<R>(k);
        kpow[k] = p;
        if (k < 32) h->kp[k] = p;
        // a paired position's factor: its unpaired bonus u is in every scaled value of an interval around it, so
        // unpaired positions cost the scale alone and paired ones exp(-u) more
        sig[k] = R(CF_LIN_SCALE);
        if constexpr (TRAIN)
            if (A.bonus != nullptr && k >= 1 && k <= L) sig[k] *= (R)expf(-A.bonus[D.seq_off + k - 1]);
    }
    for (int k = L + 2 + tid; k < 32; k += NT) h->kp[k] = R(0);   // loops longer than the sequence
    for (int k = tid; k < (kRing + 8) * gs; k += NT) G[k] = R(0);   // and B, M
    if (tid == 0) h->npair[0] = h->npair[1] = 0;
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
        for (int u = warp; u < nst + nsp; u += (NT / 32)) {
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
        for (int i = 1 + tid; i <= c + 40; i += NT) {
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
                b = fc * w.bp[si * 5 + sj1] * (sig[i] * sig[j + 1]);
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
            if constexpr (TRAIN) {
                F2[off + i] = f2;
                Bt[off + i] = b;
            } else {
                E[e_row(i, L) + d] = mm1;   // b - a - 1 = d
            }
        }
        if constexpr (sizeof(R) == 8) {   // pairable cells of the next diagonal
            if (warp == (NT / 32) - 1) {
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
    // positions t + 1 and t + 1 + NT; each step adds the newest F5 to all later ones (rows loaded ahead).
    R acc0 = R(0), acc1 = R(0), f = R(1);
    const int j0 = tid + 1, j1 = tid + 1 + NT;   // NT >= 256, L <= 512
    const R euk = w.eu * R(CF_LIN_SCALE);
    auto row = [&](int a, int j) -> R {
        if (a >= L || j <= a || j > L) return R(0);
        return TRAIN ? Bt[tri_off(j - a - 1, m) + a] : E[e_row(a, L) + j - a - 1];
    };
    auto ended = [&](R v, int a, int j) -> R { return TRAIN && v != R(0) ? v * w_end(w, s, L, a, j) : v; };
    R n0[4], n1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        n0[u] = row(1 + u, j0);
        n1[u] = L > NT ? row(1 + u, j1) : R(0);
    }
    if (tid == 0) F5[0] = R(1);
    for (int k0 = 0; k0 < L; k0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u;
            if (k < L) {   // uniform over the CTA
                const R e0 = ended(n0[u], k + 1, j0), e1 = ended(n1[u], k + 1, j1);
                n0[u] = row(k + 5, j0);
                if (L > NT) n1[u] = row(k + 5, j1);
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
    double bonus = 0.0;
    if constexpr (TRAIN) {
        float* F5g = A.ws + D.ws_off + 4 * tri;
        for (int k = tid; k <= L; k += NT) F5g[k] = (float)F5[k];
        if (warp == 0 && A.bonus != nullptr) {
            for (int k = lane; k < L; k += 32) bonus += (double)A.bonus[D.seq_off + k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) bonus += __shfl_xor_sync(0xffffffffu, bonus, o);
        }
    }
    const bool left = __syncthreads_or(bad);
    if (tid == 0) {
        if (left) A.fails[1 + atomicAdd(A.fails, 1)] = A.first + blockIdx.x;
        else static_cast<R*>(A.logz)[D.idx] = (R)(log((double)f) - (double)L * CF_LIN_LOG_SCALE + bonus);
        if constexpr (TRAIN) A.ws[D.ws_off + 4 * tri + L + 1] = left ? 0.f : 1.f;
    }
}

// ---------------------------------------------------------------------------
// Gradients: d log Z / d (every weight's logarithm), by the chain rule through
// the sums above in reverse order.  f(i, j) is the derivative to the inside of
// the pair (i, j + 1), g = f x its close weight (so g G is the probability of
// an interior loop but for its length factor), m, o and two those to FM, FM1
// and FM2.  Per diagonal, from the longest:
//
//   warps 0-7   interior loops around the diagonal's pairs: the stencil over
//               the 32 diagonals of g above, weights reversed, a part a warp;
//   warps 8-15  loops closed by the pairs of the diagonal above: for each
//               (l1, l2) of the warp's part the sum of g G over the sequence,
//               84 running sums in each lane's registers (four cells a lane),
//               and each cell's own sum for its close weight's count;
//   all warps   split sums for m and o, units of 32 cells;
//   a thread a cell  the derivatives and the probability of each transition.
//
// Counts need no atomics: thread i takes the cells (i, .), so the bases on one
// side of its pairs never change, and it adds into rows of its own, one for
// each choice of the bases on the other side.  Every sum has a fixed order.
// ---------------------------------------------------------------------------
constexpr int kOutSplit = 4;    // parts of a split sum
constexpr int kOutWarps = kLinOutThreads / 32;
constexpr int kCsrRow = 36;
enum { kRowClose = 0, kRowV01 = 10, kRowV11 = 15, kRowStack = 20, kRowMulti = 30, kRowOut = 40, kRowEnd = 50, kRows = 60 };
constexpr int kOwnRows = 20;    // rows that are always in shared memory

struct LinOutHead {
    LinHead<float> h;
    float csr[31 * kCsrRow];    // reversed weights of loop length t, behind (-t) & 3 zeros
    float csm[961];             // counts of cs(l1, l2)
    float hp[31 * kOutWarps];
    float red[8 * kOutWarps];
    int ctr[2];
};
struct LinOutLayout {
    int gs, go, cs;
    int G, g, O, Wp, Pm, Po, f, m, o, F5o, sig, pd, rows, codes, total;
    bool rows_shared;           // the kRowStack .. rows too
};
__host__ __device__ __forceinline__ LinOutLayout lin_out_layout(int L) {
    LinOutLayout Y;
    Y.gs = lin_row(L);
    Y.go = lin_row(L);
    Y.cs = lin_cells(L);
    int o = (int)((sizeof(LinOutHead) + 15) & ~size_t(15));
    auto take = [&](int elems) { const int at = o; o += 4 * elems; return at; };
    Y.G = take(kRing * Y.gs);
    Y.g = take(kRing * Y.go);
    Y.O = take(kParts * Y.cs);
    Y.Wp = take(kParts * Y.cs);
    Y.Pm = take(kOutSplit * Y.cs);
    Y.Po = take(kOutSplit * Y.cs);
    Y.f = take(4 * Y.cs);
    Y.m = take(2 * Y.cs);
    Y.o = take(4 * Y.cs);
    Y.F5o = take(Y.cs);
    Y.sig = take(Y.cs);
    Y.pd = take(2 * Y.cs);
    Y.rows = take(kOwnRows * Y.cs);
    const int codes = 2 * lin_code_stride(L);
    Y.rows_shared = o + 4 * (kRows - kOwnRows) * Y.cs + codes <= kLinSmemMax;
    if (Y.rows_shared) take((kRows - kOwnRows) * Y.cs);
    Y.codes = o;
    Y.total = o + codes;
    return Y;
}

// derivative to the loop sum seen by the pairs a = 1 + 4 q .. 4 + 4 q of diagonal d, part g (pairs (a - 1 - l1, .) around)
__device__ __forceinline__ void stencil4_around(const float* __restrict__ gr, const LinOutHead* h, int go, int d, int top,
                                                int q, int g, float* __restrict__ out) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int t = part_len(g, k);
        if (t > 30 || d + 2 + t > top) continue;
        const int lead = (-t) & 3;
        const float4* gp = reinterpret_cast<const float4*>(gr + ((d + 2 + t) & (kRing - 1)) * go + 4 * q + 32 - t - lead);
        const float4* wp = reinterpret_cast<const float4*>(h->csr + t * kCsrRow);
        float4 x = gp[0];
        float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
        for (int l = 0; l <= t + lead; l += 4) {
            const float4 y = *++gp;
            const float4 w = *wp++;
            b0 = fmaf(w.x, x.x, b0); b1 = fmaf(w.x, x.y, b1); b2 = fmaf(w.x, x.z, b2); b3 = fmaf(w.x, x.w, b3);
            b0 = fmaf(w.y, x.y, b0); b1 = fmaf(w.y, x.z, b1); b2 = fmaf(w.y, x.w, b2); b3 = fmaf(w.y, y.x, b3);
            b0 = fmaf(w.z, x.z, b0); b1 = fmaf(w.z, x.w, b1); b2 = fmaf(w.z, y.x, b2); b3 = fmaf(w.z, y.y, b3);
            b0 = fmaf(w.w, x.w, b0); b1 = fmaf(w.w, y.x, b1); b2 = fmaf(w.w, y.y, b2); b3 = fmaf(w.w, y.z, b3);
            x = y;
        }
        const float kt = h->h.kp[t];
        a0 = fmaf(kt, b0, a0); a1 = fmaf(kt, b1, a1); a2 = fmaf(kt, b2, a2); a3 = fmaf(kt, b3, a3);
    }
    *reinterpret_cast<float4*>(out + 4 * q) = make_float4(a0, a1, a2, a3);
}

// Loops of length t closed by cells i = 1 + 4 q ..: c[l1] += sum of g G, win += the cells' own sums.  N: taps, padded.
template <int N>
__device__ __forceinline__ void count_row(const float* __restrict__ G, const LinOutHead* h, int gs, int d, int t, int q,
                                          const float4 gq, float (&c)[N], float4& win) {
    if (t > 30 || t > d - 2) return;
    const float4* gp = reinterpret_cast<const float4*>(G + ((d - 2 - t) & (kRing - 1)) * gs + 4 + 4 * q);
    const float4* wp = reinterpret_cast<const float4*>(h->h.w.csf + t * 32);
    float4 x = gp[0];
    float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
#pragma unroll
    for (int l = 0; l < N; l += 4) {
        if (l <= t) {
            const float4 y = gp[l / 4 + 1];
            const float4 w = wp[l / 4];
            b0 = fmaf(w.x, x.x, b0); b1 = fmaf(w.x, x.y, b1); b2 = fmaf(w.x, x.z, b2); b3 = fmaf(w.x, x.w, b3);
            b0 = fmaf(w.y, x.y, b0); b1 = fmaf(w.y, x.z, b1); b2 = fmaf(w.y, x.w, b2); b3 = fmaf(w.y, y.x, b3);
            b0 = fmaf(w.z, x.z, b0); b1 = fmaf(w.z, x.w, b1); b2 = fmaf(w.z, y.x, b2); b3 = fmaf(w.z, y.y, b3);
            b0 = fmaf(w.w, x.w, b0); b1 = fmaf(w.w, y.x, b1); b2 = fmaf(w.w, y.y, b2); b3 = fmaf(w.w, y.z, b3);
            c[l] = fmaf(gq.x, x.x, fmaf(gq.y, x.y, fmaf(gq.z, x.z, fmaf(gq.w, x.w, c[l]))));
            c[l + 1] = fmaf(gq.x, x.y, fmaf(gq.y, x.z, fmaf(gq.z, x.w, fmaf(gq.w, y.x, c[l + 1]))));
            c[l + 2] = fmaf(gq.x, x.z, fmaf(gq.y, x.w, fmaf(gq.z, y.x, fmaf(gq.w, y.y, c[l + 2]))));
            c[l + 3] = fmaf(gq.x, x.w, fmaf(gq.y, y.x, fmaf(gq.z, y.y, fmaf(gq.w, y.z, c[l + 3]))));
            x = y;
        }
    }
    const float kt = h->h.kp[t];
    win.x = fmaf(kt, b0, win.x); win.y = fmaf(kt, b1, win.y); win.z = fmaf(kt, b2, win.z); win.w = fmaf(kt, b3, win.w);
}

__device__ __forceinline__ float warp_add(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// the warp's sums over all diagonals -> counts of cs(l1, t - l1)
template <int N>
__device__ __forceinline__ void count_out(LinOutHead* h, int t, const float (&c)[N], int lane) {
    if (t > 30) return;
#pragma unroll
    for (int l = 0; l < N; ++l) {
        if (l <= t) {
            const float v = warp_add(c[l]);
            if (lane == 0 && !(t == 2 && l == 1)) h->csm[l * 31 + t - l] = h->h.w.csf[t * 32 + l] * h->h.kp[t] * v;
        }
    }
}

// bases that pair with one base differ in this bit
__device__ __forceinline__ int side(int x) { return (x >> 1) & 1; }

}  // namespace

__global__ void __launch_bounds__(kLinOutThreads, 1) k_lin_outside32(LinArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* h = reinterpret_cast<LinOutHead*>(smem_raw);
    const SeqDesc D = A.descs[A.first + blockIdx.x];
    const int L = D.L, m = L + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LinOutLayout Y = lin_out_layout(L);
    auto at = [&](int o) { return reinterpret_cast<float*>(smem_raw + o); };
    float *G = at(Y.G), *gr = at(Y.g), *O = at(Y.O), *Wp = at(Y.Wp), *Pm = at(Y.Pm), *Po = at(Y.Po);
    float *fr = at(Y.f), *mr = at(Y.m), *orr = at(Y.o), *F5o = at(Y.F5o), *sig = at(Y.sig), *pd = at(Y.pd),
          *rows = at(Y.rows);
    int8_t* s = reinterpret_cast<int8_t*>(smem_raw + Y.codes);
    int8_t* pc = s + lin_code_stride(L);
    const int gs = Y.gs, go = Y.go, cs = Y.cs;

    float* base = A.ws + D.ws_off;
    const int64_t tri = pad32(tri_size(L));
    const float* FM = base;
    const float* FM1 = base + tri;
    float* two = base + 2 * tri;           // FM2; a cell's derivative takes its place
    const float* Bt = base + 3 * tri;
    const float* F5 = base + 4 * tri;
    if (F5[L + 1] == 0.f) return;         // on the list already
    // the rows beyond kOwnRows: behind them, or in the arena
    const int rs = Y.rows_shared ? cs : (int)pad32(L);
    float* more = Y.rows_shared ? rows + kOwnRows * cs : base + 4 * tri + pad32(L + 2);

    {
        const float* src = static_cast<const float*>(A.weights);
        float* dst = reinterpret_cast<float*>(&h->h.w);
        for (int k = tid; k < (int)(sizeof(LinWeights<float>) / 4); k += kLinOutThreads) dst[k] = src[k];
    }
    for (int k = tid; k < L + 2; k += kLinOutThreads) {
        if (k < 32) h->h.kp[k] = scale_pow<float>(k);
        sig[k] = (float)CF_LIN_SCALE;
        if (A.bonus != nullptr && k >= 1 && k <= L) sig[k] *= expf(-A.bonus[D.seq_off + k - 1]);
    }
    for (int k = L + 2 + tid; k < 32; k += kLinOutThreads) h->h.kp[k] = 0.f;
    for (int k = tid; k < kRing * (gs + go); k += kLinOutThreads) G[k] = 0.f;   // G and gr
    for (int k = tid; k < 10 * cs; k += kLinOutThreads) fr[k] = 0.f;            // f, m, o
    for (int k = tid; k < 2 * cs; k += kLinOutThreads) pd[k] = 0.f;
    for (int k = tid; k < kOwnRows * cs; k += kLinOutThreads) rows[k] = 0.f;
    for (int k = tid; k < (kRows - kOwnRows) * rs; k += kLinOutThreads) more[k] = 0.f;
    for (int k = tid; k < 961; k += kLinOutThreads) h->csm[k] = 0.f;
    for (int k = tid; k < 31 * kOutWarps; k += kLinOutThreads) h->hp[k] = 0.f;
    if (tid < 2) h->ctr[tid] = 0;
    encode_seq(A.seqs, A.mask, D.seq_off, L, s, pc);
    __syncthreads();
    for (int k = tid; k < 31 * kCsrRow; k += kLinOutThreads) {
        const int t = k / kCsrRow, x = k % kCsrRow - ((-t) & 3);
        h->csr[k] = x >= 0 && x <= t ? h->h.w.csf[t * 32 + t - x] : 0.f;
    }
    const LinWeights<float>& w = h->h.w;
    const float K1 = (float)CF_LIN_SCALE, muk = w.mu * K1, k2 = K1 * K1, mm = w.mp * w.mb, euk = w.eu * K1;
    bool bad = false;

    // exterior, from the end: thread t keeps the derivative sum of position t (rows of the pair (t + 1, j))
    {
        const float invZ = 1.0f / F5[L];
        float acc = 0.f, f = invZ;
        if (tid == 0) F5o[L] = invZ;
        auto col = [&](int j) -> float { return (j > tid + 1 && tid + 1 < L && j <= L) ? Bt[tri_off(j - tid - 2, m) + tid + 1] : 0.f; };
        float nx[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) nx[u] = col(L - u);
        for (int j0 = L; j0 >= 1; j0 -= 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 - u;   // F5o[j] = f known: to all earlier positions, then F5o[j - 1]
                if (j >= 1) {
                    const float e = nx[u] != 0.f ? nx[u] * w_end(w, s, L, tid + 1, j) : 0.f;
                    nx[u] = col(j - 4);
                    acc = fmaf(f * w.ep, e, acc);
                    if (tid == j - 1) F5o[j - 1] = fmaf(f, euk, acc);
                    __syncthreads();
                    f = F5o[j - 1];
                }
            }
        }
    }
    __syncthreads();

    // G of the 32 longest diagonals
    auto load_G = [&](int r, int a) {
        const int b = a + r + 1;
        const float v = Bt[tri_off(r, m) + a];
        G[(r & (kRing - 1)) * gs + a + 2] = v == 0.f ? 0.f : v * w.close[idx4(s[b], s[a], s[b + 1], s[a - 1])];
    };
    for (int r = max(0, L - 2 - (kRing - 1)); r <= L - 2; ++r)
        for (int a = 1 + tid; a <= L - 1 - r; a += kLinOutThreads) load_G(r, a);

    float cA[32], cB[24], cC[16], cD[12];   // warps 8-15: running sums of the part's loop lengths
#pragma unroll
    for (int k = 0; k < 32; ++k) cA[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 24; ++k) cB[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) cC[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 12; ++k) cD[k] = 0.f;
    // this thread's sums over its cells
    float s_mu = 0.f, s_one = 0.f, s_multi = 0.f, s_ext = 0.f, s01 = 0.f, s10 = 0.f, s11 = 0.f, s_hp = 0.f, end_last = 0.f;
    struct {   // of this thread's last pair: the row of its bases (-1: none), its hairpin and small loops
        int y;
        float loops;
    } before = {-1, 0.f};
    __syncthreads();

    for (int d = L - 2; d >= -1; --d) {
        const int c = L - 1 - d;   // cells i = 1 .. c of diagonal d; i = 1 .. c - 1 of d + 1
        if (warp < kParts) {
            if (d >= 0)
                for (int q = lane; 4 * q < c; q += 32) stencil4_around(gr, h, go, d, L - 2, q, warp, O + warp * cs);
        } else if (d + 1 >= 4 && c > 1) {
            const int g = warp - kParts;
            const float* g1 = gr + ((d + 1) & (kRing - 1)) * go + 33;   // cell i = 1
            for (int q = lane; 4 * q < c - 1; q += 32) {
                const float4 gq = make_float4(g1[4 * q], g1[4 * q + 1], g1[4 * q + 2], g1[4 * q + 3]);
                float4 win = make_float4(0.f, 0.f, 0.f, 0.f);
                count_row<32>(G, h, gs, d + 1, part_len(g, 0), q, gq, cA, win);
                count_row<24>(G, h, gs, d + 1, part_len(g, 1), q, gq, cB, win);
                if (g < 7) {
                    count_row<16>(G, h, gs, d + 1, part_len(g, 2), q, gq, cC, win);
                    count_row<12>(G, h, gs, d + 1, part_len(g, 3), q, gq, cD, win);
                }
                *reinterpret_cast<float4*>(Wp + g * cs + 4 * q) = win;
            }
        }
        if (d >= 2) {   // split sums, units of 32 cells dealt out as warps come free
            constexpr int N = kOutSplit, T = N * (N - 1) / 2;
            const int units = 2 * N * ((c + 31) >> 5);
            for (;;) {
                int u = 0;
                if (lane == 0) u = atomicAdd(&h->ctr[d & 1], 1);
                u = __shfl_sync(0xffffffffu, u, 0);
                if (u >= units) break;
                const int kind = u % 2, q = (u / 2) % N, i = 1 + (u / (2 * N)) * 32 + lane, j = i + d, x = 1 + q;
                if (i > c) continue;
                if (kind == 0) {          // m: two(i - x, j) FM1(i - x, i)
                    Pm[q * cs + i - 1] = dot_tri<float, N>(two, tri_off(d + x, m) + i - x, N * m - N * (d + x) - T - N,
                                                           FM1, tri_off(x, m) + i - x, N * m - N * x - T - N,
                                                           part_terms<N>(i - 1, q));
                } else {                  // o: two(i, j + x) FM(j, j + x)
                    Po[q * cs + i - 1] = dot_tri<float, N>(two, tri_off(d + x, m) + i, N * m - N * (d + x) - T,
                                                           FM, tri_off(x, m) + j, N * m - N * x - T,
                                                           part_terms<N>(L - 1 - j, q));
                }
            }
        }
        __syncthreads();
        if (tid == 0) h->ctr[(d & 1) ^ 1] = 0;
        const float kd = scale_pow<float>(max(d, 0));
        const int i = 1 + tid;
        // the loop sum of this thread's pair of diagonal d + 1, for its close weight's count
        if (d + 1 >= 0 && i <= c - 1 && before.y >= 0) {
            float win = 0.f;
            if (d + 1 >= 4) {
#pragma unroll
                for (int p = 0; p < kParts; ++p) win += Wp[p * cs + i - 1];
                win *= gr[((d + 1) & (kRing - 1)) * go + i + 32];
            }
            rows[(kRowClose + before.y) * cs + i] += before.loops + win;
        }
        before.y = -1;
        float v_hp = 0.f;
        if (d >= 0 && i <= c) {
            const int j = i + d, off = tri_off(d, m);
            const bool inner = i >= 2 && j + 1 <= L - 1;   // the cell (i - 1, j + 1) exists
            float mv = 0.f, ov = 0.f;
            if (d >= 2) {
#pragma unroll
                for (int p = 0; p < kOutSplit; ++p) {
                    mv += Pm[p * cs + i - 1];
                    ov += Po[p * cs + i - 1];
                }
                if (i <= c - 1) mv += mr[((d + 1) & 1) * cs + i] * muk;
                if (i >= 2) ov += orr[((d + 1) & 3) * cs + i - 1] * muk;
                ov += mv;
                const int o1 = tri_off(d - 1, m) + i;
                s_mu += mv * FM[o1] * muk + ov * FM1[o1 + 1] * muk;
                bad |= !(ov < 1e37f);
            }
            float tw = mv, fv = 0.f, gv = 0.f;
            if (pairable_codes(pc[i], pc[j + 1])) {
                const int b = j + 1, sa = s[i], sb = s[b], si1 = s[i + 1], sj = s[j], sl = s[i - 1], sr = s[b + 1];
                const float end = w_end(w, s, L, i, b);
                const float e_ext = F5[i - 1] * F5o[b] * w.ep * end;
                float e_one = 0.f, e_st = 0.f;
                if (inner) {
                    e_one = orr[((d + 2) & 3) * cs + i - 1] * w.mp * end;
                    e_st = fr[((d + 2) & 3) * cs + i - 1] * w.stack[idx4(sl, s[j + 2], sa, sb)];
                }
                const float* g3 = gr + ((d + 3) & (kRing - 1)) * go + 32;
                const float* g4 = gr + ((d + 4) & (kRing - 1)) * go + 32;
                float dG = K1 * (w.cs01 * w.b01[sr] * g3[i - 1] + w.cs10 * w.b01[sl] * g3[i - 2]) +
                           k2 * w.cs11 * w.i11[sl * 5 + sr] * g4[i - 2];
#pragma unroll
                for (int p = 0; p < kParts; ++p) dG += O[p * cs + i - 1];
                const float Bv = Bt[off + i], out = w.close[idx4(sb, sa, sr, sl)];
                const float bv = e_ext + e_one + e_st + dG * out;
                const float P = bv * Bv;
                bad |= !(P <= 1.01f);
                pd[i] += P;
                pd[cs + b] += P;
                const int key = idx4(sa, sb, si1, sj);
                fv = bv * w.bp[sa * 5 + sb] * (sig[i] * sig[b]);
                gv = fv * w.close[key];
                const float fm = fv * mm * w_multi(w, s, i, b);
                tw += fm;
                // probabilities of the transitions: as the outer pair ...
                v_hp = gv * w.hp[d <= DHP ? d : DHP] * kd;
                float v01 = 0.f, v10 = 0.f, v11 = 0.f, v_st = 0.f;
                if (d >= 2) v_st = fv * w.stack[key] * Bt[tri_off(d - 2, m) + i + 1];
                if (d >= 3) {
                    const float* G3 = G + ((d - 3) & (kRing - 1)) * gs + 2;
                    v01 = gv * K1 * w.cs01 * w.b01[sj] * G3[i + 1];
                    v10 = gv * K1 * w.cs10 * w.b01[si1] * G3[i + 2];
                }
                if (d >= 4) v11 = gv * k2 * w.cs11 * w.i11[si1 * 5 + sj] * G[((d - 4) & (kRing - 1)) * gs + 2 + i + 2];
                // (the multiloop as a product: what the other loops leave of P loses a rare one's digits, 9e-3 of the
                // count at 20 nt, 4e-4 at 30)
                const float v_multi = fm * two[off + i];
                const int y1 = side(sb) * 5 + sj, y2 = side(sb) * 5 + sr;
                before.loops = v_hp + v01 + v10 + v11;
                before.y = y1;
                more[(kRowMulti - kOwnRows + y1) * rs + i] += v_multi;
                s_multi += v_multi;
                rows[(kRowV01 + sj) * cs + i] += v01;
                rows[(kRowV11 + sj) * cs + i] += v11;
                more[(kRowStack - kOwnRows + y1) * rs + i] += v_st;
                // ... and as the inner one
                more[(kRowOut - kOwnRows + y2) * rs + i] += dG * out * Bv;
                const float v_one = e_one * Bv, v_ext = e_ext * Bv;
                if (b == L) end_last = v_one + v_ext;   // no base on its right: once for each i
                else more[(kRowEnd - kOwnRows + y2) * rs + i] += v_one + v_ext;
                s_one += v_one; s_ext += v_ext;
                s01 += v01; s10 += v10; s11 += v11;
                if (d >= DHP) s_hp += v_hp;
            }
            two[off + i] = tw;
            fr[(d & 3) * cs + i] = fv;
            mr[(d & 1) * cs + i] = mv;
            orr[(d & 3) * cs + i] = ov;
            gr[(d & (kRing - 1)) * go + i + 32] = gv;
        }
        if (d >= 0 && d < DHP) {
            const float v = warp_add(v_hp);
            if (lane == 0) h->hp[d * kOutWarps + warp] = v;
        }
        if (d >= kRing && i <= L - 1 - (d - kRing)) load_G(d - kRing, i);   // in the place of diagonal d
        __syncthreads();
    }

    // loop counts, sums of the threads' own sums
    float *v10r = Pm, *endL = Po;   // by i
    if (1 + tid <= L - 1) {
        v10r[1 + tid] = s10;
        endL[1 + tid] = end_last;
    }
    if (warp >= kParts) {
        const int g = warp - kParts;
        count_out<32>(h, part_len(g, 0), cA, lane);
        count_out<24>(h, part_len(g, 1), cB, lane);
        if (g < 7) {
            count_out<16>(h, part_len(g, 2), cC, lane);
            count_out<12>(h, part_len(g, 3), cD, lane);
        }
    }
    {
        float eu = 0.f;
        for (int j = 1 + tid; j <= L; j += kLinOutThreads) eu += F5o[j] * F5[j - 1] * euk;
        const float v[9] = {s_mu, s_one, s_multi, s_ext, s01, s10, s11, s_hp, eu};
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const float x = warp_add(v[k]);
            if (lane == 0) {
                if (k == 7) h->hp[DHP * kOutWarps + warp] = x;
                else h->red[(k == 8 ? 7 : k) * kOutWarps + warp] = x;
            }
        }
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) A.fails[1 + atomicAdd(A.fails, 1)] = A.first + blockIdx.x;
        return;
    }
    // sums over i of the threads' rows, by the bases beside i: T[class][s_i * 5 + neighbour][row]
    float* T = G;
    for (int e = tid; e < 1000; e += kLinOutThreads) {
        const int cl = e / 200, sx = (e % 200) / 50, nb = (e / 10) % 5, y = e % 10;
        const float* r = cl == 0 ? rows + (kRowClose + y) * cs : more + (kRowStack - kOwnRows + (cl - 1) * 10 + y) * rs;
        float v = 0.f;
        for (int i = cl == 4 ? 2 : 1; i <= L - 1; ++i)
            if (s[i] == sx && s[cl < 3 ? i + 1 : i - 1] == nb) v += r[i];
        T[e] = v;
    }
    __syncthreads();
    auto t1 = [&](int cl, int a, int b, int c, int d) {   // pair (a, b), c beside a and d beside b, inside it
        return a < 4 && pairable_codes(a, b) ? T[cl * 200 + (a * 5 + c) * 10 + side(b) * 5 + d] : 0.f;
    };
    auto t2 = [&](int cl, int a, int b, int c, int d) {   // bases b, a of the pair, d beside b's ... outside it
        return b < 4 && pairable_codes(b, a) ? T[cl * 200 + (b * 5 + d) * 10 + side(a) * 5 + c] : 0.f;
    };
    auto red = [&](int k) {
        float v = 0.f;
        for (int x = 0; x < kOutWarps; ++x) v += h->red[k * kOutWarps + x];
        return v;
    };
    // end weights of the pairs at either end of the sequence
    auto first = [&](int a, int b, int z) {   // (1, .): s_b = a, s_1 = b, base z right of it
        return L >= 2 && s[1] == b && b < 4 && pairable_codes(b, a) ? more[(kRowEnd - kOwnRows + side(a) * 5 + z) * rs + 1] : 0.f;
    };
    auto last = [&](int a, int b, int z) {    // (., L): base z left of it (-1: any)
        float v = 0.f;
        if (s[L] == a && b < 4 && pairable_codes(b, a))
            for (int i = z < 0 ? 1 : 2; i <= L - 1; ++i)
                if (s[i] == b && (z < 0 || s[i - 1] == z)) v += endL[i];
        return v;
    };
    double* out = A.counts + (int64_t)D.idx * CF_BLOB_LEN;
    for (int e = tid; e < CF_BLOB_LEN; e += kLinOutThreads) {
        float v = 0.f;
        if (e < CF_OFF_STACK) {
            const int a = e / 5, b = e % 5;
            for (int x = 0; x < 25; ++x)
                for (int cl = 0; cl < 3; ++cl) v += t1(cl, a, b, x / 5, x % 5);
        } else if (e < CF_OFF_TM) {
            const int k = e - CF_OFF_STACK;
            v = t1(1, k / 125, k / 25 % 5, k / 5 % 5, k % 5);
        } else if (e < CF_OFF_HC) {
            const int k = e - CF_OFF_TM;
            v = t1(0, k / 125, k / 25 % 5, k / 5 % 5, k % 5) + t2(3, k / 125, k / 25 % 5, k / 5 % 5, k % 5);
        } else if (e < CF_OFF_DL) {
            const int k = e - CF_OFF_HC, a = k / 5, b = k % 5;
            for (int x = 0; x < 25; ++x)
                v += t1(0, a, b, x / 5, x % 5) + t1(2, a, b, x / 5, x % 5) + t2(3, a, b, x / 5, x % 5) + t2(4, a, b, x / 5, x % 5);
            for (int z = 0; z < 5; ++z) v += first(a, b, z);
            v += last(a, b, -1);
        } else if (e < CF_OFF_DR) {
            const int k = e - CF_OFF_DL, a = k / 25, b = k / 5 % 5, z = k % 5;
            for (int x = 0; x < 5; ++x) v += t1(2, a, b, z, x) + t2(4, a, b, z, x);
            v += first(a, b, z);
        } else if (e < CF_OFF_HPCUM) {
            const int k = e - CF_OFF_DR, a = k / 25, b = k / 5 % 5, z = k % 5;
            for (int x = 0; x < 5; ++x) v += t1(2, a, b, x, z) + t2(4, a, b, x, z);
            v += last(a, b, z);
        } else if (e < CF_OFF_CS) {
            for (int x = 0; x < kOutWarps; ++x) v += h->hp[(e - CF_OFF_HPCUM) * kOutWarps + x];
        } else if (e < CF_OFF_I11) {
            const int k = e - CF_OFF_CS;
            v = k == 1 ? red(4) : k == 31 ? red(5) : k == 32 ? red(6) : h->csm[k];
        } else if (e < CF_OFF_B01) {
            const int x = (e - CF_OFF_I11) / 5, y = (e - CF_OFF_I11) % 5;
            for (int i = 1; i <= L - 1; ++i)
                if (s[i + 1] == x) v += rows[(kRowV11 + y) * cs + i];
        } else if (e < CF_OFF_MB) {
            const int x = e - CF_OFF_B01;
            for (int i = 1; i <= L - 1; ++i) v += rows[(kRowV01 + x) * cs + i] + (s[i + 1] == x ? v10r[i] : 0.f);
        } else {
            v = e == CF_OFF_MB ? red(2) : e == CF_OFF_MU ? red(0) : e == CF_OFF_MP ? red(1) + red(2) : e == CF_OFF_EU ? red(7) : red(3);
        }
        out[e] = (double)v;
    }
    for (int k = 1 + tid; k <= L; k += kLinOutThreads)
        A.unpaired[D.seq_off + k - 1] = 1.0 - ((double)pd[k] + (double)pd[cs + k]);
}

size_t lin_outside_smem_bytes(int Lmax) {
    size_t most = 0;   // not monotone: the rows move to the arena where they no longer fit
    for (int L = Lmax; L >= 0 && L >= Lmax - 512; --L) most = most > (size_t)lin_out_layout(L).total ? most : (size_t)lin_out_layout(L).total;
    return most;
}

namespace {
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

template <bool TRAIN, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_lin_inside32(LinArgs A) { lin_inside<float, TRAIN, NT>(A); }
__global__ void __launch_bounds__(256, 2) k_lin_inside64(LinArgs A) { lin_inside<double, false, 256>(A); }

// Threads by length: as many as keep an SM at about 1,024 threads with the
// CTAs its shared memory holds (four of 256 up to 160 nt, three up to 235, two of
// 512 up to 395; a few nt more would fit, but leave the splits no L1: 1,000 x 240
// nt with three, two CTAs 4.7, 4.6 ms, 1,000 x 405 nt with two, one 18.1, 16.0).
// On a shared device no more than other kernels' CTAs have (narrow).
LinKernel lin_inside_kernel(int L, bool fp64, bool train, bool narrow) {
    if (fp64) return {k_lin_inside64, 256};
    if (L <= 235 || narrow) return {train ? k_lin_inside32<true, 256> : k_lin_inside32<false, 256>, 256};
    if (L <= 395) return {train ? k_lin_inside32<true, 512> : k_lin_inside32<false, 512>, 512};
    return {train ? k_lin_inside32<true, 1024> : k_lin_inside32<false, 1024>, 1024};
}
// Last length of the launch class of L: sequences of a class share a launch,
// whose shared memory is its longest sequence's.  In float the classes end where
// an SM holds a CTA less (see above; 2,000 x 130-180 nt in one class of 235, two:
// 3.6, 3.4 ms).  In double the FP64 pipe, not the CTAs an SM holds, bounds all
// but the short ones, and a class more is a last wave more (300 x 150-180 nt with
// a class up to 160, up to 235: 5.2, 4.0 ms; 500 x 20-400 nt with these classes
// and with float's: 13.6, 13.9).
int lin_class_end(int L, bool fp64) {
    if (fp64) return L <= 96 ? 96 : L <= 235 ? 235 : kLinMaxLen64;
    return L <= 160 ? 160 : L <= 235 ? 235 : L <= 395 ? 395 : kLinMaxLen;
}

size_t lin_inside_smem_bytes(int Lmax, bool fp64) {
    return fp64 ? lin_layout<double>(Lmax).total : lin_layout<float>(Lmax).total;
}

}  // namespace cf
