// cf_latency.cu -- fold kernels for batches that do not fill the device: one
// sequence on one 512-thread CTA, or on the 4 or 8 256-thread CTAs of a
// thread-block cluster.
//
// Such a fold is bound by its longest serial chain, not by throughput: on each
// diagonal the step's barrier waits for the cell that folds the most terms one
// after another.  The grouped kernels let one thread find, evaluate and fold a
// cell's interior loops; here these are three things:
//
//   E  a warp a cell: the lanes take a row (l1) each, find its candidates,
//      evaluate their terms and store them, in the order they are folded, in a
//      buffer -- a diagonal ahead of their use, beside the chains;
//   F  a lane a cell: folds the stored terms, nothing else on its path;
//   A  a lane a cell: the bifurcation chains, as in the grouped kernels;
//   X  one warp: a step of the exterior recurrence (F5, F5o), which the grouped
//      kernels run alone after (before) the diagonals.
//
// All four of a step read only what earlier steps wrote; warps claim F and A
// chunks (the long chains) first, then E cells.  Terms, order and rounding are
// the grouped kernels', so tables are bitwise theirs.
#include "cf_group.cuh"

namespace cf {
namespace {

constexpr int kTermRows = kWindowMax;

// Interior-loop terms of two diagonals: terms[parity][k][cell], counts[parity][cell]
struct TermBuf {
    float* terms;
    int* counts;
    int stride;
    __device__ __forceinline__ float* at(int diag, int cell) const {
        return terms + (size_t)((diag & 1) * kTermRows) * stride + cell;
    }
    __device__ __forceinline__ int& count(int diag, int cell) const { return counts[(diag & 1) * stride + cell]; }
};
__device__ __forceinline__ TermBuf term_buf(float* at, int L) {
    TermBuf B;
    B.stride = (int)pad32(L);
    B.terms = at;
    B.counts = reinterpret_cast<int*>(at + (size_t)2 * kTermRows * B.stride);
    return B;
}

// Fast_LogPlusEquals for serial chains: both cubics that a unit bin of d can
// need, and the boundary between them, in one round trip to shared memory.
// (lse32's two dependent look-ups are fewer instructions, and some 30 cycles
// more on a chain's path.)
struct ChainTables {
    float4 below[16], above[16];   // unit bin of d: the cubics below / from the boundary inside it
    float edge[16];                // that boundary, or FLT_MAX
};
__device__ __forceinline__ void load_chain_tables(ChainTables* C, const PolyTables* pt) {
    for (int k = threadIdx.x; k < kLseBins; k += blockDim.x) {
        const float2 bin = pt->lse_bin[k];
        const int seg = __float_as_int(bin.y) / (int)sizeof(float4);
        C->below[k] = pt->lse[seg];
        C->above[k] = pt->lse[min(seg + 1, 7)];
        C->edge[k] = bin.x;
    }
}
struct Lse32Chain {
    using Real = float;
    const ChainTables* c;
    static __device__ __forceinline__ float neg() { return CF_NEG32; }
    static __device__ __forceinline__ float half() { return CF_HALF32; }
    static __device__ __forceinline__ float add(float x, float y) { return __fadd_rn(x, y); }
    __device__ __forceinline__ float plus(float a, float x) const {
        const float d = fabsf(__fsub_rn(a, x));   // = larger - smaller, the same rounding
        // floor(d): 2^23 + d rounded towards zero (any bin from 16 on, as in unit_bin)
        const int k = __float_as_int(__fadd_rz(d, 8388608.0f)) & 15;
        const float4 lo = c->below[k], hi = c->above[k];
        const bool up = d >= c->edge[k];
        const float4 q = make_float4(up ? hi.x : lo.x, up ? hi.y : lo.y, up ? hi.z : lo.z, up ? hi.w : lo.w);
        const float r = __fadd_rn(fminf(a, x), cubic(q, d));
        return d >= LSE_TMAX ? fmaxf(a, x) : r;
    }
};

// Terms p[0], p[stride], ... in global memory.
struct Stored {
    static constexpr bool kTwo = false;
    const float* p;
    int stride;
    __device__ __forceinline__ void next(const float*& x, const float*&) {
        x = p;
        p += stride;
    }
};
// Terms in shared memory, the same for every lane.
struct Listed {
    static constexpr bool kTwo = false;
    const float* p;
    __device__ __forceinline__ void next(const float*& x, const float*&) { x = p++; }
};
// Sums of two operands, of successive terms one diagonal apart in two
// triangular tables: the offsets' steps shrink by one from term to term where
// the span grows, and grow by one (negative: towards zero) where it falls --
// the same change.
struct TriPair {
    static constexpr bool kTwo = true;
    const float *a, *b;
    int oa, da, ob, db;
    __device__ __forceinline__ void next(const float*& x, const float*& y) {
        x = a + oa;
        y = b + ob;
        oa += da--;
        ob += db--;
    }
};

// acc (+) terms 0 .. n - 1 of src in order: blocks of eight, operands in
// registers two blocks ahead; the last one is filled up with the semiring's
// zero, which leaves acc as it is.  (Cycles a term at 801 nt: 134.  Operands 16
// to 32 terms ahead in shared memory 140; following the sum in plain floating
// point beside the chain, to have each d's cubics at hand before d, 115 to 160,
// 10 % off a whole fold for twice the instructions; both not kept.)
template <class S, class Src>
__device__ __forceinline__ float fold_chain(const S& sr, float acc, int n, Src src) {
    constexpr int U = 8;
    if (n <= 0) return acc;
    float x[U], y[U], cur[U];
    auto load = [&](int k) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float *px = nullptr, *py = nullptr;
            src.next(px, py);
            if (k + u < n) {
                x[u] = *px;
                if constexpr (Src::kTwo) y[u] = *py;
            }
        }
    };
    auto make = [&](int k, float (&v)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float t = x[u];
            if constexpr (Src::kTwo) t = __fadd_rn(t, y[u]);
            v[u] = k + u < n ? t : CF_NEG32;
        }
    };
    load(0);
    make(0, cur);
    load(U);
    for (int k = 0; k < n; k += U) {
        float nxt[U];
        make(k + U, nxt);
        load(k + 2 * U);
#pragma unroll
        for (int u = 0; u < U; ++u) acc = sr.plus(acc, cur[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = nxt[u];
    }
    return acc;
}

// Evaluates a cell's candidates (window_list) 32 at a time, four loads a lane
// in flight, and stores their terms in order.  (A row a lane, in place, cost
// 8,000 cycles a cell at 400 nt, this 5,000.)
template <class Val, class Term>
__device__ __forceinline__ int eval_terms(uint32_t msk, int l1, uint16_t* list, float* out, int stride, int lane, Val val,
                                          Term term) {
    const int total = window_list(msk, l1, list, lane);
    for (int k0 = lane; k0 < total; k0 += 128) {
        int c[4];
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = list[min(k0 + 32 * u, total - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = val(c[u] & 31, c[u] >> 5);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + 32 * u < total) out[(size_t)(k0 + 32 * u) * stride] = term(c[u] & 31, c[u] >> 5, v[u]);
    }
    __syncwarp();
    return total;
}

// E of inside cell (i, j): the terms of inside_B, rows l1 ascending.
template <class S>
__device__ __forceinline__ void inside_E(const SmemTabs<float>* __restrict__ tb, const SeqV& Q, const InTabs<float>& T,
                                         int i, int j, const TermBuf& B, int cell, uint16_t* list, int lane) {
    const ParamView<float> P{tb->blob};
    const int m = T.m, d = j - i;
    const int si = Q.s[i], sj1 = Q.s[j + 1], si1 = Q.s[i + 1], sj = Q.s[j];
    const float jB = tb->jB(si, sj1, si1, sj);
    // row l1: q from lo(l1) to j
    auto lo = [&](int l1) { return i + 2 + l1 > l1 + j - CMAX ? i + 2 + l1 : l1 + j - CMAX; };
    const uint32_t msk = lane <= (d < CMAX ? d : CMAX) ? Q.window(i + lane + 1, lo(lane), j - lo(lane) + 1) : 0u;
    const int total = eval_terms(
        msk, lane, list, B.at(d, cell), B.stride, lane,
        [&](int l1, int bit) { return T.FC[tri_off(lo(l1) + bit - 2 - i - l1, m) + i + l1 + 1]; },
        [&](int l1, int bit, float v) {
            const int p = i + l1, q = lo(l1) + bit, l2 = j - q;
            float e;
            if (l1 == 0 && l2 == 0) {
                e = S::add(P.bp(si1, sj), P.stack(si, sj1, si1, sj));
            } else {
                const int sq = Q.s[q], sa = Q.s[p + 1];
                const float jB2 = tb->jB(sq, sa, Q.s[q + 1], Q.s[p]);
                e = S::add(S::add(S::add(P.cs(l1, l2), P.bp(sa, sq)), jB), jB2);
                if (l1 < 2) {
                    const float sn = l1 == 0 ? (l2 == 1 ? P.b01(sj) : 0.0f)
                                             : (l2 == 0 ? P.b01(si1) : (l2 == 1 ? P.i11(si1, sj) : 0.0f));
                    e = S::add(e, sn);
                }
            }
            return S::add(e, v);
        });
    if (lane == 0) B.count(d, cell) = total;
}

// F of inside cell (i, j): FC (inside_B).
template <class S>
__device__ __forceinline__ void inside_F(const S& sr, const SmemTabs<float>* __restrict__ tb, const SeqV& Q,
                                         const InTabs<float>& T, int i, int j, float fm2, const TermBuf& B, int cell) {
    const ParamView<float> P{tb->blob};
    const int d = j - i;
    const float jB = tb->jB(Q.s[i], Q.s[j + 1], Q.s[i + 1], Q.s[j]);
    float acc = sr.plus(CF_NEG32, S::add(jB, P.hp(d <= DHP ? d : DHP)));
    const float* t = B.at(d, cell);
    acc = fold_chain(sr, acc, B.count(d, cell), Stored{t, B.stride});
    if (fm2 > CF_HALF32) {
        const float jA = junctionA<S>(P, Q.L, Q, i, j);
        acc = sr.plus(acc, S::add(S::add(S::add(fm2, jA), P.mp()), P.mb()));
    }
    T.FC[tri_off(d, T.m) + i] = acc;
}

// A of inside cell (i, j): FM2 (returned), FM1, FM (inside_A).
template <class S>
__device__ __forceinline__ float inside_A_lat(const S& sr, const SmemTabs<float>* __restrict__ tb, const SeqV& Q,
                                              const InTabs<float>& T, int i, int j) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m, d = j - i, at = tri_off(d, m) + i;
    const float NEG = CF_NEG32, HALF = CF_HALF32;
    if (i == 0 || j == L) {
        T.FC[at] = NEG;
        T.FM1[at] = NEG;
        T.FM[at] = NEG;
        return NEG;
    }
    if (!Q.pairable(i, j + 1)) T.FC[at] = NEG;
    float fm2 = NEG, fm1 = NEG, fm = NEG;
    if (i + 2 <= j) {
        // the terms that need no chain first, so that their loads are under way
        const float fin = T.FC[T.at(i + 1, j - 1)], ext = T.FM1[T.at(i + 1, j)], prev = T.FM[T.at(i, j - 1)];
        // splits k = i + 1 .. j - 1: FM1[i][k] (span 1 up), FM[k][j] (span d - 1 down)
        fm2 = fold_chain(sr, NEG, d - 1,
                         TriPair{T.FM1, T.FM, tri_off(1, m) + i, m - 1, tri_off(d - 1, m) + i + 1, d - 1 - m});
        if (Q.pairable(i + 1, j) && fin > HALF) {
            const float jAji = junctionA_rev<S>(P, L, Q, i, j);
            fm1 = sr.plus(fm1, S::add(S::add(S::add(fin, jAji), P.mp()), P.bp(Q.s[i + 1], Q.s[j])));
        }
        if (ext > HALF) fm1 = sr.plus(fm1, S::add(ext, P.mu()));
        if (fm2 > HALF) fm = sr.plus(fm, fm2);
        if (prev > HALF) fm = sr.plus(fm, S::add(prev, P.mu()));
        if (fm1 > HALF) fm = sr.plus(fm, fm1);
    }
    T.FM1[at] = fm1;
    T.FM[at] = fm;
    return fm2;
}

// Up to kXChunk terms of an exterior sum at once: evaluated by the lanes, all
// of their loads in flight together, closed up in order in xs, folded by every
// lane.
constexpr int kXChunk = 256;
template <class S, class Term>
__device__ __forceinline__ float exterior_sum(const S& sr, float acc, int n, float* xs, int lane, Term term) {
    for (int c0 = 0; c0 < n; c0 += kXChunk) {
        int len = 0;
        float v[kXChunk / 32];
        bool ok[kXChunk / 32];
#pragma unroll
        for (int u = 0; u < kXChunk / 32; ++u) {
            const int k = c0 + 32 * u + lane;
            ok[u] = k < n && term(k, v[u]);
        }
#pragma unroll
        for (int u = 0; u < kXChunk / 32; ++u) {
            const unsigned bits = __ballot_sync(0xffffffffu, ok[u]);
            if (ok[u]) xs[len + __popc(bits & ((1u << lane) - 1u))] = v[u];
            len += __popc(bits);
        }
        __syncwarp();
        acc = fold_chain(sr, acc, len, Listed{xs});
        __syncwarp();
    }
    return acc;
}

template <class S, class Team>
__device__ __forceinline__ void inside_lat(const S& sr, SmemFold<float>* sm, const FoldArgs& A, const Team& tm,
                                           const TermBuf& B, float* xs, uint16_t* list) {
    const SeqV Q = seq_v(sm, 0);
    const InView<float> V = in_view<float>(A, sm->ws[0], Q.L);
    const ParamView<float> P{sm->tabs.blob};
    const int L = Q.L;
    if (tm.rank() == 0) build_plist(Q, V.PLs);
    if (threadIdx.x == 0) sm->step_ctr[0] = sm->step_ctr[1] = 0;
    if (tm.rank() == 0 && threadIdx.x == 0) V.T.F5[0] = 0.0f;
    tm.sync();
    auto cells = [&](int d) { return d >= 0 && d <= L - 2 ? V.PLs.poff[d + 1] - V.PLs.poff[d] : 0; };
    for (int t = 0; t <= L + 1; ++t) {
        const int nB = cells(t - 1), cF = (nB + 31) >> 5, nA = max(0, L + 1 - t), cA = (nA + 31) >> 5, nE = cells(t);
        const int oB = nB ? V.PLs.poff[t - 1] : 0, oE = nE ? V.PLs.poff[t] : 0;
        run_items(sm, tm, t, 1 + cF + cA + nE, [&](int q, int lane) {
            if (q == 0) {   // F5[t]: FC of spans up to t - 2
                if (t < 1 || t > L) return;
                float acc = S::add(V.T.F5[t - 1], P.eu());
                acc = exterior_sum(sr, acc, t, xs, lane, [&](int k, float& v) {
                    if (!Q.pairable(k + 1, t)) return false;
                    const float fcin = V.T.FC[V.T.at(k + 1, t - 1)], f5k = V.T.F5[k];
                    if (!(fcin > CF_HALF32) || !(f5k > CF_HALF32)) return false;
                    const float jA = junctionA_rev<S>(P, L, Q, k, t);
                    v = S::add(S::add(S::add(S::add(f5k, fcin), P.ep()), P.bp(Q.s[k + 1], Q.s[t])), jA);
                    return true;
                });
                if (lane == 0) V.T.F5[t] = acc;
            } else if (q <= cF) {
                const int r = (q - 1) * 32 + lane;
                if (r >= nB) return;
                const int i = V.PLs.pl[oB + r];
                inside_F(sr, &sm->tabs, Q, V.T, i, i + t - 1, V.FB[((t - 1) & 1) * V.fbs + i], B, r);
            } else if (q <= cF + cA) {
                const int i = (q - 1 - cF) * 32 + lane;
                if (i >= nA) return;
                V.FB[(t & 1) * V.fbs + i] = inside_A_lat(sr, &sm->tabs, Q, V.T, i, i + t);
            } else {
                const int r = q - 1 - cF - cA, i = V.PLs.pl[oE + r];
                inside_E<S>(&sm->tabs, Q, V.T, i, i + t, B, r, list, lane);
            }
        });
    }
}

// E of outside cell (a, b): the sources of outside_B, rows l1 descending; the
// stacking source, folded last, after the others (and the count's bit 16).
__device__ __forceinline__ void outside_E(const SmemTabs<float>* __restrict__ tb, const SeqV& Q, const OutTabs& T, int a,
                                          int b, const TermBuf& B, int cell, uint16_t* list, int lane) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m, t = b - a;
    const int sa = Q.s[a], sb1 = Q.s[b + 1], sb2 = Q.s[b + 2];
    const float bp_ab = P.bp(sa, sb1);
    const float jB2 = tb->jB(sb1, sa, sb2, Q.s[a - 1]);
    const int l1max = (a - 2 < CMAX) ? a - 2 : CMAX;
    const int r1 = CMAX - lane;   // this lane's row: l1 descending
    const int jmax = (b + 1 + CMAX - r1 < L - 1) ? b + 1 + CMAX - r1 : L - 1;
    uint32_t msk = r1 >= 0 && r1 <= l1max ? Q.window(a - 1 - r1, b + 2, jmax - b) : 0u;
    const bool stacks = r1 == 0 && (msk & 1u);
    if (r1 == 0) msk &= ~1u;
    float* out = B.at(t, cell);
    auto val = [&](int l1, int bit) { return T.FCo[tri_off(b + 2 + bit - a + l1, m) + a - 1 - l1]; };
    auto term = [&](int l1, int bit, float v) {
        if (!(v > CF_HALF32)) return CF_NEG32;   // folds as nothing, as the source that is passed over
        const int i = a - 1 - l1, j = b + 1 + bit, l2 = bit, sj = Q.s[j], si = Q.s[i], si1 = Q.s[i + 1];
        float e;
        if (l1 == 0 && l2 == 0) {
            e = __fadd_rn(P.bp(si1, sj), P.stack(si, Q.s[j + 1], si1, sj));
        } else {
            const float jBij = tb->jB(si, Q.s[j + 1], si1, sj);
            e = __fadd_rn(__fadd_rn(__fadd_rn(P.cs(l1, l2), bp_ab), jBij), jB2);
            if (l1 < 2) {
                const float sn = l1 == 0 ? (l2 == 1 ? P.b01(sb2) : 0.0f)
                                         : (l2 == 0 ? P.b01(si1) : (l2 == 1 ? P.i11(si1, sb2) : 0.0f));
                e = __fadd_rn(e, sn);
            }
        }
        return __fadd_rn(v, e);
    };
    const int total = eval_terms(msk, r1, list, out, B.stride, lane, val, term);
    if (stacks) out[(size_t)total * B.stride] = term(0, 0, val(0, 0));
    const unsigned st = __ballot_sync(0xffffffffu, stacks);
    if (lane == 0) B.count(t, cell) = total | (st ? 1 << 16 : 0);
}

// F of outside cell (a, b): FCo (outside_B).
template <class S>
__device__ __forceinline__ void outside_F(const S& sr, const SmemTabs<float>* __restrict__ tb, const SeqV& Q,
                                          const OutTabs& T, int a, int b, const TermBuf& B, int cell) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, t = b - a;
    const float bp_ab = P.bp(Q.s[a], Q.s[b + 1]);
    float acc = CF_NEG32;
    const float f5k = T.F5[a - 1];
    const float jAji = junctionA_rev<S>(P, L, Q, a - 1, b + 1);
    if (f5k > CF_HALF32) {
        const float temp = __fadd_rn(__fadd_rn(__fadd_rn(T.F5o[b + 1], P.ep()), bp_ab), jAji);
        acc = sr.plus(acc, __fadd_rn(temp, f5k));
    }
    const float* x = B.at(t, cell);
    const int cnt = B.count(t, cell), n = cnt & 0xffff;
    acc = fold_chain(sr, acc, n, Stored{x, B.stride});
    if (a >= 2) {
        if (b + 1 < L) {
            const float v = T.FM1o[tri_off(t + 2, T.m) + a - 1];
            acc = sr.plus(acc, __fadd_rn(__fadd_rn(__fadd_rn(v, jAji), P.mp()), bp_ab));
        }
        if (cnt >> 16) acc = sr.plus(acc, x[(size_t)n * B.stride]);
    }
    T.FCo[tri_off(t, T.m) + a] = acc;
}

// A of outside cell (a, b): FMo, FM1o, FM2o (outside_A): two chains, of a - 1
// and of L - 1 - b terms.
template <class S>
__device__ __forceinline__ void outside_A_lat(const S& sr, const SmemTabs<float>* __restrict__ tb, const SeqV& Q,
                                              const OutTabs& T, int a, int b) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m, t = b - a, at = tri_off(t, m) + a;
    float fmo = CF_NEG32, fm1o = CF_NEG32;
    const bool fm_region = 0 < a && a + 2 <= b && b < L;
    if (fm_region) {
        const float up = b + 1 < L ? T.FMo[tri_off(t + 1, m) + a] : 0.0f;
        const float left = a >= 2 ? T.FM1o[tri_off(t + 1, m) + a - 1] : 0.0f;
        // FM2o[a - w][b] + FM1[a - w][a], w = a - 1 .. 1
        const int w1 = a - 1, w2 = L - 1 - b;
        float acc = fold_chain(sr, CF_NEG32, w1,
                               TriPair{T.FM2o, T.FM1, tri_off(t + w1, m) + a - w1, t + w1 - m, tri_off(w1, m) + a - w1,
                                       w1 - m});
        if (b + 1 < L) acc = sr.plus(acc, __fadd_rn(up, P.mu()));
        fmo = acc;
        // FM2o[a][b + w] + FM[b][b + w], w = L - 1 - b .. 1
        acc = CF_NEG32;
        if (a >= 2) acc = sr.plus(acc, __fadd_rn(left, P.mu()));
        acc = fold_chain(sr, acc, w2,
                         TriPair{T.FM2o, T.FM, tri_off(t + w2, m) + a, t + w2 - 1 - m, tri_off(w2, m) + b, w2 - 1 - m});
        fm1o = sr.plus(acc, fmo);
    }
    T.FMo[at] = fmo;
    T.FM1o[at] = fm1o;
    float fm2o = CF_NEG32;
    if (fm_region) fm2o = sr.plus(fm2o, fmo);
    if (0 < a && b < L && Q.pairable(a, b + 1)) {
        const float fco = T.FCo[at];
        if (fco > CF_HALF32) {
            const float jA = junctionA<S>(P, L, Q, a, b);
            fm2o = sr.plus(fm2o, __fadd_rn(__fadd_rn(__fadd_rn(fco, jA), P.mp()), P.mb()));
        }
    }
    T.FM2o[at] = fm2o;
}

template <class S, class Team>
__device__ __forceinline__ void outside_lat(const S& sr, SmemFold<float>* sm, const FoldArgs& A, const Team& tm,
                                            const TermBuf& B, float* xs, uint16_t* list) {
    const SeqV Q = seq_v(sm, 0);
    const int L = Q.L;
    const OutTabs T = out_tabs(A, sm->ws[0], L);
    const PairList PLs = plist_of(A, sm->ws[0], L);
    const ParamView<float> P{sm->tabs.blob};
    if (threadIdx.x == 0) sm->step_ctr[0] = sm->step_ctr[1] = 0;
    tm.sync();
    auto cells = [&](int d) { return d >= 0 && d <= L - 2 ? PLs.poff[d + 1] - PLs.poff[d] : 0; };
    for (int t = L; t >= 0; --t) {
        const int nB = cells(t - 1), cF = (nB + 31) >> 5, nA = L + 1 - t, cA = (nA + 31) >> 5, nE = cells(t - 2);
        const int oB = nB ? PLs.poff[t - 1] : 0, oE = nE ? PLs.poff[t - 2] : 0;
        run_items(sm, tm, t, 1 + cF + cA + nE, [&](int q, int lane) {
            if (q == 0) {   // F5o[t]
                float acc = 0.0f;
                if (t < L) {
                    acc = exterior_sum(sr, CF_NEG32, L - t - 1, xs, lane, [&](int k, float& v) {
                        const int j = L - k;   // L .. t + 2
                        if (!Q.pairable(t + 1, j)) return false;
                        const float fcin = T.FC[T.at(t + 1, j - 1)];
                        if (!(fcin > CF_HALF32)) return false;
                        const float jA = junctionA_rev<S>(P, L, Q, t, j);
                        const float temp = __fadd_rn(__fadd_rn(__fadd_rn(T.F5o[j], P.ep()), P.bp(Q.s[t + 1], Q.s[j])), jA);
                        v = __fadd_rn(temp, fcin);
                        return true;
                    });
                    acc = sr.plus(acc, __fadd_rn(T.F5o[t + 1], P.eu()));
                }
                if (lane == 0) T.F5o[t] = acc;
            } else if (q <= cF) {   // FCo of diagonal t - 1
                const int r = (q - 1) * 32 + lane;
                if (r >= nB) return;
                const int a = PLs.pl[oB + r];
                outside_F(sr, &sm->tabs, Q, T, a, a + t - 1, B, r);
            } else if (q <= cF + cA) {
                const int a = (q - 1 - cF) * 32 + lane;
                if (a < nA) outside_A_lat(sr, &sm->tabs, Q, T, a, a + t);
            } else {                // sources of diagonal t - 2: FCo of spans t and above
                const int r = q - 1 - cF - cA, a = PLs.pl[oE + r];
                outside_E(&sm->tabs, Q, T, a, a + t - 2, B, r, list, lane);
            }
        });
    }
}

// MEA decode's table (mea_cell) with the bifurcations of a cell in kMeaParts
// ascending ranges of k, a warp each: a part keeps the first k of its largest
// sum, and the parts join in order by the same strict '>', so the cell keeps
// the candidate a serial scan keeps.  (One thread a cell: 11.7 of 143 ms at
// 801 nt, waiting for its loads.)
constexpr int kMeaParts = 8;
template <class Team>
__device__ __forceinline__ void mea_lat(SmemFold<float>* sm, const FoldArgs& A, const Team& tm, const TermBuf& B) {
    const SeqV Q = seq_v(sm, 0);
    const int L = Q.L, m = L + 1, lane = threadIdx.x & 31;
    const Arena32 ar = arena32(L);
    float* base = A.ws + sm->ws[0];
    const float *POST = base + ar.FMo, *up = base + ar.up;
    float* score = base + ar.FM2o;
    int* tb = reinterpret_cast<int*>(base + ar.FM);
    const float two_g = __fmul_rn(2.0f, A.gamma);
    for (int i = 1 + tm.tid(); i <= L; i += tm.nthreads()) base[ar.up + i] = mea_unpaired(POST, L, two_g, i);
    for (int t = tm.tid(); t < L; t += tm.nthreads()) A.structs[sm->soff[0] + t] = '.';
    tm.sync();
    float* pv = B.terms;   // [part][i]: largest sum, its k
    int* pk = reinterpret_cast<int*>(B.terms + kMeaParts * (B.stride + 32));
    const int ps = B.stride + 32;
    for (int d = 0; d <= L; ++d) {
        const int chunks = (L + 1 - d + 31) >> 5, len = (d - 1 + kMeaParts - 1) / kMeaParts;
        if (d >= 2) {
            for (int u = tm.tid() >> 5; u < chunks * kMeaParts; u += tm.nthreads() >> 5) {
                const int part = u % kMeaParts, i = (u / kMeaParts) * 32 + lane;
                if (i + d > L) continue;
                float best = -3.402823466e38f;
                int arg = 0;
                const int s0 = 1 + part * len, s1 = min(d, s0 + len);
#pragma unroll 8
                for (int s = s0; s < s1; ++s) {
                    const float v = __fadd_rn(score[tri_off(s, m) + i], score[tri_off(d - s, m) + i + s]);
                    if (v > best) { best = v; arg = i + s + 4; }
                }
                pv[part * ps + i] = best;
                pk[part * ps + i] = arg;
            }
            tm.sync();
        }
        for (int i = tm.tid(); i + d <= L; i += tm.nthreads()) {
            const int j = i + d, c = tri_off(d, m) + i;
            if (d == 0) {
                score[c] = 0.0f;
                tb[c] = 0;
                continue;
            }
            float best = -1.0f;
            int arg = -1;
            float v = __fadd_rn(up[i + 1], score[tri_off(d - 1, m) + i + 1]);
            if (v > best) { best = v; arg = 1; }
            v = __fadd_rn(up[j], score[tri_off(d - 1, m) + i]);
            if (v > best) { best = v; arg = 2; }
            if (d >= 2) {
                if (Q.pairable(i + 1, j)) {
                    v = __fadd_rn(POST[tri_off(d - 1, m) + i + 1], score[tri_off(d - 2, m) + i + 1]);
                    if (v > best) { best = v; arg = 3; }
                }
#pragma unroll
                for (int p = 0; p < kMeaParts; ++p) {
                    v = pv[p * ps + i];
                    if (v > best) { best = v; arg = pk[p * ps + i]; }
                }
            }
            score[c] = best;
            tb[c] = arg;
        }
        tm.sync();
    }
    if (tm.rank() == 0 && threadIdx.x == 0) {
        int* qi = reinterpret_cast<int*>(base + ar.queue);
        mea_traceback(tb, L, qi, qi + 2 * L + 4, A.structs + sm->soff[0], A.status);
    }
}

// MODE 0: MEA, 1: BPP, 2: the inside with the accurate log-sum-exp alone
// (logZ, and the tables the sampler draws from).
template <int MODE, class Team>
__device__ __forceinline__ void fold_lat(const FoldArgs& A, const Team& tm, int gi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    __shared__ ChainTables chain;
    __shared__ float xs[kXChunk];
    __shared__ uint16_t lists[kLatThreads / 32][kTermRows];
    uint16_t* list = lists[threadIdx.x >> 5];
    setup_group(sm, A, A.blob32, gi);
    const int L = sm->L[0];
    float* ws = A.ws + sm->ws[0];
    if constexpr (MODE == 2) {
        inside_lat(LseAcc32{}, sm, A, tm, term_buf(ws + pad32(arena32_inside_words(L)), L), xs, list);
        if (A.logz != nullptr && tm.rank() == 0 && threadIdx.x == 0)
            A.logz[sm->idx[0]] = in_view<float>(A, sm->ws[0], L).T.F5[L];
    } else {
        load_chain_tables(&chain, &sm->poly);
        __syncthreads();
        const Lse32Chain sr{&chain};
        const TermBuf B = term_buf(ws + arena32(L).total, L);
        inside_lat(sr, sm, A, tm, B, xs, list);
        outside_lat(sr, sm, A, tm, B, xs, list);
        if constexpr (MODE == 0) {
            FoldArgs Ap = A;
            Ap.post_out = nullptr;
            Ap.logz = nullptr;
            posterior_group(sm, Ap, tm);
            mea_lat(sm, A, tm, B);
        } else {
            posterior_group(sm, A, tm);
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(kLatThreads, 1) k_fold_lat32(FoldArgs A) {
    fold_lat<MODE>(A, CtaTeam{}, blockIdx.x);
}
template <int MODE>
__global__ void __launch_bounds__(kFoldThreads, 2) k_fold_cluster32(FoldArgs A) {
    const int c = cluster_nctas();
    fold_lat<MODE>(A, ClusterTeam{cluster_ctarank(), c}, (int)blockIdx.x / c);
}

}  // namespace

LatKernels lat_kernels(bool cluster) {
    if (cluster) return {k_fold_cluster32<0>, k_fold_cluster32<1>, k_fold_cluster32<2>};
    return {k_fold_lat32<0>, k_fold_lat32<1>, k_fold_lat32<2>};
}
int64_t lat_term_words(int L) { return 2 * (kTermRows + 1) * pad32(L); }

}  // namespace cf
