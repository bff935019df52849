// cf_outside.cuh -- outside pass and posterior in float32.
//
// The reference (gpu_contrafold/cpu.py:680-819) computes the outside tables
// and the posterior by SCATTERING from each source cell into its children,
// sources visited i ascending / j descending (outside) and i descending / j
// ascending (posterior).  Float log-sum-exp and float += are not associative,
// so the value of a target depends on the order its contributions arrive.
// Here each target GATHERS its contributions, enumerating its sources in
// exactly the order the reference's scatter reaches it, with each
// contribution computed by the same operations -- a parallel formulation
// with bitwise the reference's results.  The derivation of each order is next
// to the code.
//
// Outside cells run in two phases per diagonal t (descending):
//   phase A (every cell): FMo, FM1o (read FM2o of larger spans, FMo / FM1o of
//           span t+1) and FM2o (reads the cell's own FMo and FCo);
//   phase B (pairable cells): FCo (reads FCo of spans >= t+2, FM1o of span t+2).
// A step runs A(t) and B(t-1); FCo(t) was produced one step earlier.
#pragma once

#include "cf_inside.cuh"
#include "cf_seq.cuh"

namespace cf {

struct OutTabs {
    CF_TAB(const float) FC;
    CF_TAB(const float) FM;
    CF_TAB(const float) FM1;
    CF_TAB(const float) F5;
    CF_TAB(float) FCo;
    CF_TAB(float) FMo;
    CF_TAB(float) FM1o;
    CF_TAB(float) FM2o;
    CF_TAB(float) F5o;
    int m;
    __device__ __forceinline__ int at(int i, int j) const { return tri_off(j - i, m) + i; }
    // table sizes for checked builds (nothing otherwise)
    __device__ __forceinline__ void sized(int L) {
        CF_SIZE_TAB(FC, tri_size(L));
        CF_SIZE_TAB(FM, tri_size(L));
        CF_SIZE_TAB(FM1, tri_size(L));
        CF_SIZE_TAB(F5, L + 2);
        CF_SIZE_TAB(FCo, tri_size(L));
        CF_SIZE_TAB(FMo, tri_size(L));
        CF_SIZE_TAB(FM1o, tri_size(L));
        CF_SIZE_TAB(FM2o, tri_size(L));
        CF_SIZE_TAB(F5o, L + 2);
        (void)L;
    }
};

// F5o (cpu.py:684-699) by one warp, k = L-1 .. 0.  Target k receives, in the
// reference's order, the pair terms of iterations j = L .. k+2 and then the
// unpaired term F5o[k+1] + eu of iteration j = k+1.
template <class QV>
__device__ __forceinline__ void exterior_outside_warp(const Lse32& sr, const SmemTabs<float>* __restrict__ tb,
                                                      const QV& Q, const OutTabs& T) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, lane = threadIdx.x & 31;
    if (lane == 0) T.F5o[L] = 0.0f;
    __syncwarp();
    for (int k = L - 1; k >= 0; --k) {
        float acc = CF_NEG32;
        for (int j0 = L; j0 >= k + 2; j0 -= 32) {
            const int j = j0 - lane;
            bool ok = false;
            float term = 0.0f;
            if (j >= k + 2 && Q.pairable(k + 1, j)) {
                const float fcin = T.FC[T.at(k + 1, j - 1)];
                if (fcin > CF_HALF32) {
                    const float jA = junctionA_rev<Lse32>(P, L, Q, k, j);
                    const float temp = __fadd_rn(__fadd_rn(__fadd_rn(T.F5o[j], P.ep()), P.bp(Q.s[k + 1], Q.s[j])), jA);
                    term = __fadd_rn(temp, fcin);
                    ok = true;
                }
            }
            unsigned mask = __ballot_sync(0xffffffffu, ok);
            while (mask) {
                const int t = __ffs(mask) - 1;
                mask &= mask - 1;
                acc = sr.plus(acc, __shfl_sync(0xffffffffu, term, t));
            }
        }
        acc = sr.plus(acc, __fadd_rn(T.F5o[k + 1], P.eu()));
        if (lane == 0) T.F5o[k] = acc;
        __syncwarp();
    }
}

// Phase A of outside cell (a, b), 0 <= a <= b <= L: FMo, FM1o, FM2o.
//
// FMo[a][b]: FM2o distribution of sources (i, b), i = 1 .. a-1 ascending, k = a
// (cpu.py:753-758); then block 1 of source (a, b+1): FMo[a][b] (+)= FMo[a][b+1]
// + mu (cpu.py:705).  FM1o[a][b]: block 2 of source (a-1, b): FM1o[a-1][b] + mu
// (cpu.py:715); FM2o distribution of sources (a, j), j = L-1 .. b+1, k = b
// (cpu.py:756); block 1 of source (a, b): (+)= FMo[a][b] (cpu.py:706).
// FM2o[a][b]: cpu.py:702-704, 746-751, FCo[a][b] from phase B.
//
// The FMo chain (a-1 terms) and the FM1o chain (L-1-b terms) run back to back
// in a single loop of (a-1) + (L-1-b) = L-2-t iterations, which is the same for
// every cell of diagonal t -- lanes of a warp working on one diagonal stay
// converged.
__device__ __forceinline__ void outside_A(const Lse32& sr, const SmemTabs<float>* __restrict__ tb,
                                                 const SeqV& Q, const OutTabs& T, int a, int b) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m, t = b - a;
    const int at = tri_off(t, m) + a;
    const bool fm_region = (0 < a) && (a + 2 <= b) && (b < L);
    float fmo = CF_NEG32, fm1o = CF_NEG32;
    if (fm_region) {
        const int n1 = a - 1, n2 = L - 1 - b, K = n1 + n2;
        const float* fmo_next = T.FMo + (tri_off(t + 1, m) + a);   // FMo[a][b + 1]
        float first = CF_NEG32;   // FM1o[a - 1][b] opens the FM1o chain
        if (a >= 2) first = sr.plus(first, __fadd_rn(T.FM1o[tri_off(t + 1, m) + a - 1], P.mu()));
        float acc = CF_NEG32, acc1 = CF_NEG32;
        // terms k < n1: FM2o[a-w][b], FM1[a-w][a] with w = n1-k; then
        // FM2o[a][b+w], FM[b][b+w] with w = n2-(k-n1).  Every lane of a warp
        // changes over at another k: it does so by selections (a branch, taken by
        // one lane after the other, cost 65 instead of 45 instructions a term; 10,000 x
        // 200 nt MEA 256 -> 246 ms).  One index for both FM and FM1, which lies fm1 cells on.
        const int fm1 = (int)(static_cast<const float*>(T.FM1) - static_cast<const float*>(T.FM));
        int x = tri_off(t + n1, m) + a - n1, y = fm1 + tri_off(n1, m) + a - n1, dx = n1 + t - m, dy = n1 - m;
        const int x2 = tri_off(t + n2, m) + a, y2 = tri_off(n2, m) + b;
        int kl = 0;
        prefetched_chain<float>(
            K,
            [&](const float*& px, const float*& py) {
                const bool over = kl == n1;
                x = over ? x2 : x;
                y = over ? y2 : y;
                dx = over ? n2 - 1 + t - m : dx;
                dy = over ? n2 - 1 - m : dy;
                px = T.FM2o + x;
#ifdef CF_CHECK
                py = y >= fm1 ? T.FM1 + (y - fm1) : T.FM + y;
#else
                py = T.FM + y;
#endif
                x += dx--;
                y += dy--;
                ++kl;
            },
            [&](int k, float vx, float vy) {
                acc1 = k == n1 ? acc : acc1;
                acc = k == n1 ? first : acc;
                // unguarded fold: a sentinel operand makes the term <= NEG, which
                // Fast_LogPlusEquals discards (it returns the larger argument)
                acc = sr.plus(acc, __fadd_rn(vx, vy));
            });
        if (n2 == 0) {
            acc1 = acc;
            acc = first;
        }
        fmo = b + 1 < L ? sr.plus(acc1, __fadd_rn(*fmo_next, P.mu())) : acc1;
        fm1o = sr.plus(acc, fmo);
    }
    T.FMo[at] = fmo;
    T.FM1o[at] = fm1o;
    float fm2o = CF_NEG32;
    if (fm_region) fm2o = sr.plus(fm2o, fmo);
    if (0 < a && b < L && Q.pairable(a, b + 1)) {
        const float fco = T.FCo[at];
        if (fco > CF_HALF32) {
            const float jA = junctionA<Lse32>(P, L, Q, a, b);
            fm2o = sr.plus(fm2o, __fadd_rn(__fadd_rn(__fadd_rn(fco, jA), P.mp()), P.mb()));
        }
    }
    T.FM2o[at] = fm2o;
}

// Phase B of a pairable outside cell (a, b) (pair (a, b+1)): FCo[a][b].
//  1. exterior term of the F5o phase, k = a-1, j = b+1 (cpu.py:695-699);
//  2. sources (i, j) = (a-1-l1, b+1+l2) of the main loop, i ascending
//     (l1 = 30 .. 0) and j descending; a source contributes through its
//     single-branch loop (block 3, cpu.py:717-745) iff pairable(i, j+1), so
//     each row walks the partner mask of position i over j+1 = b+2 ..
//     b+2+(30-l1), highest bit first.  Source (a-1, b+1) first contributes
//     through FM1o (block 2, cpu.py:708-714), then through block 3.
// `lanes`: the lanes evaluating cells together, walked together as in
// inside_B, four rows at a time from the largest l1max among them.
__device__ __forceinline__ void outside_B(const Lse32& sr, const SmemTabs<float>* __restrict__ tb,
                                          const SeqV& Q, const OutTabs& T, int a, int b, unsigned lanes) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m, t = b - a;
    const int sa = Q.s[a], sb1 = Q.s[b + 1];
    const float bp_ab = P.bp(sa, sb1);
    float acc = CF_NEG32;
    {
        const float f5k = T.F5[a - 1];
        if (f5k > CF_HALF32) {
            const float jA = junctionA_rev<Lse32>(P, L, Q, a - 1, b + 1);
            const float temp = __fadd_rn(__fadd_rn(__fadd_rn(T.F5o[b + 1], P.ep()), bp_ab), jA);
            acc = sr.plus(acc, __fadd_rn(temp, f5k));
        }
    }
    // jB of the inner pair (p+1, q) = (a, b+1): hc[s[q]][s[p+1]] + tm[s[q]][s[p+1]][s[q+1]][s[p]]
    const float jB2 = tb->jB(sb1, sa, Q.s[b + 2], Q.s[a - 1]);
    const int l1max = (a - 2 < CMAX) ? a - 2 : CMAX;   // i = a-1-l1 >= 1
    // row l1: sources (i, j) = (a - 1 - l1, b + 1 + l2), l1 + l2 <= 30, the
    // partner bits (zero beyond L) with l2 = 30 - l1 at bit 31.  FCo[i][j] has
    // span x = t + 2 + l1 + l2.  The last two sources of the rows 1 and 0 have an
    // extra term and are folded on their own (the others': as in inside_B).
    const int sb2 = Q.s[b + 2];
    const uint32_t* pb = Q.PB + ((b + 2) >> 5);
    const uint8_t* codep = Q.s.p + a - 1;
    const uint8_t* codeq = Q.s.p + b + 1;
    const float* cs = tb->blob + CF_OFF_CS;
    auto row = [&](int l1) -> uint32_t {
        if (l1 > l1max) return 0u;
        const int c = Q.pc[a - 1 - l1];
        const uint32_t* w = pb + (c & 3) * Q.W;
        const uint32_t x = __funnelshift_r(w[0], w[1], (b + 2) & 31) << (l1 + 1);
        return c < 4 ? x : 0u;
    };
    struct Cand {
        float e, v;
    };
    auto cand = [&](int l1, int l2) -> Cand {
        const int x = t + 2 + l1 + l2;
        const float v = T.FCo[((x * (2 * m + 1 - x)) >> 1) + a - 1 - l1];
        return {__fadd_rn(__fadd_rn(__fadd_rn(cs[l1 * 31 + l2], bp_ab), tb->jb[codep[-l1] * 25 + codeq[l2]].jB), jB2), v};
    };
    auto fold = [&](float v, float e, bool has) {
        const float r = sr.plus(acc, __fadd_rn(v, e));
        acc = has && v > CF_HALF32 ? r : acc;
    };
    const int lm = __reduce_max_sync(lanes, l1max);
    uint32_t near = 0u;
    for (int part = lm < 1 ? lm : 1; part >= 0; --part) {   // the rows lm .. 1, then row 0
        near = row(part) >> (part + 1);
        queue_rows<Cand>(
            lanes, part == 0 ? 1 : lm,
            [&](int k) -> uint32_t {
                const int l1 = part == 0 ? k : lm - k;
                const uint32_t x = row(l1);
                return l1 == part ? x & ~(6u << part) : x;   // l1 = part: bits part + 1 and part + 2 are l2 = 0 and 1
            },
            [&](int k, int u) {
                const int l1 = part == 0 ? k : lm - k;
                return cand(l1, 30 - l1 - u);
            },
            [&](const Cand& c, bool has) { fold(c.v, c.e, has); });
        if (near & 2u) {
            const Cand c = cand(part, 1);
            fold(c.v, __fadd_rn(c.e, part == 0 ? P.b01(sb2) : P.i11(Q.s[a - 1], sb2)), true);
        }
        if (part == 1 && near & 1u) {
            const Cand c = cand(1, 0);
            fold(c.v, __fadd_rn(c.e, P.b01(Q.s[a - 1])), true);
        }
    }
    if (l1max >= 0) {
        if (b + 1 < L) {
            const float v = T.FM1o[tri_off(t + 2, m) + a - 1];
            const float jAji = junctionA_rev<Lse32>(P, L, Q, a - 1, b + 1);
            acc = sr.plus(acc, __fadd_rn(__fadd_rn(__fadd_rn(v, jAji), P.mp()), bp_ab));
        }
        if (near & 1u) {   // the stacking source (a - 1, b + 1)
            const float v = T.FCo[tri_off(t + 2, m) + a - 1];
            if (v > CF_HALF32)
                acc = sr.plus(acc, __fadd_rn(v, __fadd_rn(bp_ab, P.stack(Q.s[a - 1], sb2, sa, sb1))));
        }
    }
    T.FCo[tri_off(t, m) + a] = acc;
}

// Posterior of the pair (a, b), 1 <= a < b <= L, pairable (cpu.py:760-819).
// The reference adds fexp32 terms into POST[a][b] from sources (i, j) =
// (a-1-l1, b+l2) visited i descending (l1 = 0 ..), j ascending (l2 = 0 ..),
// each iff pairable(i, j+1) and its outside value is live; source (a-1, b)
// adds its multiloop (FM1o) term right after its stacking term; the exterior
// term comes last.  Returns the clipped value.
// `lanes`: the lanes evaluating pairs together, walked together as in
// inside_B.
__device__ __forceinline__ float posterior_pair(const SmemTabs<float>* __restrict__ tb, const PolyTables* pt,
                                                const SeqV& Q, const OutTabs& T, float Z, int a, int b,
                                                unsigned lanes) {
    const ParamView<float> P{tb->blob};
    const int L = Q.L, m = T.m;
    const float fcin = T.FC[tri_off(b - 1 - a, m) + a];
    const bool live = fcin > CF_HALF32;
    const int sa = Q.s[a], sb = Q.s[b];
    const float bp_ab = P.bp(sa, sb);
    // jB of the inner pair (p+1, q) = (a, b)
    const float jB2 = tb->jB(sb, sa, Q.s[b + 1], Q.s[a - 1]);
    float post = 0.0f;
    const int l1max = live ? ((a - 2 < CMAX) ? a - 2 : CMAX) : -1;   // i = a-1-l1 >= 1
    // row l1: sources (i, j) = (a - 1 - l1, b + l2), l1 + l2 <= 30, the partner
    // bits (zero beyond L) with l2 = 0 at bit 31.  FCo[i][j] has span
    // x = b - a + 1 + l1 + l2.  The first two sources of the rows 0 and 1 have an
    // extra term and are added on their own (the others': as in inside_B).
    const int sb1 = Q.s[b + 1];
    const uint32_t* pb = Q.PB + ((b + 1) >> 5);
    const uint8_t* codep = Q.s.p + a - 1;
    const uint8_t* codeq = Q.s.p + b;
    const float* cs = tb->blob + CF_OFF_CS;
    auto row = [&](int l1) -> uint32_t {
        if (l1 > l1max) return 0u;
        const int c = Q.pc[a - 1 - l1];
        const uint32_t* w = pb + (c & 3) * Q.W;
        const uint32_t x = __brev(__funnelshift_r(w[0], w[1], (b + 1) & 31)) & (uint32_t)((int)0x80000000 >> (CMAX - l1));
        return c < 4 ? x : 0u;
    };
    struct Cand {
        float v, jB, cs;
    };
    auto cand = [&](int l1, int l2) -> Cand {
        const int x = b - a + 1 + l1 + l2;
        return {T.FCo[((x * (2 * m + 1 - x)) >> 1) + a - 1 - l1], tb->jb[codep[-l1] * 25 + codeq[l2]].jB, cs[l1 * 31 + l2]};
    };
    auto term = [&](const Cand& c) {
        return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fsub_rn(c.v, Z), c.jB), c.cs), fcin), bp_ab), jB2);
    };
    auto add = [&](const Cand& c, float e, bool has) {
        has = has && __fsub_rn(c.v, Z) > CF_HALF32;
        float x = fexp32_below(pt, e);
        if (has && e >= 0.0f) x = fexp32(pt, e);
        const float sum = __fadd_rn(post, x);
        post = has ? sum : post;
    };
    const int lm = __reduce_max_sync(lanes, l1max);
    for (int part = 0; part < 2 && part <= lm; ++part) {   // row 0, then the other rows
        const uint32_t near = row(part);
        if (part == 0) {   // the stacking source (a-1, b) and its multiloop term
            if (near & 0x80000000u) {
                const float out = __fsub_rn(T.FCo[tri_off(b - a + 1, m) + a - 1], Z);
                if (out > CF_HALF32)
                    post = __fadd_rn(post, fexp32(pt, __fadd_rn(__fadd_rn(__fadd_rn(out, bp_ab), P.stack(Q.s[a - 1], sb1, sa, sb)), fcin)));
            }
            if (l1max >= 0 && b < L) {
                const float v = T.FM1o[tri_off(b - a + 1, m) + a - 1];
                if (v > CF_HALF32) {
                    const float jAji = junctionA_rev<Lse32>(P, L, Q, a - 1, b);
                    const float x = __fsub_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(v, fcin), jAji), P.mp()), bp_ab), Z);
                    post = __fadd_rn(post, fexp32(pt, x));
                }
            }
        } else if (near & 0x80000000u) {
            const Cand c = cand(1, 0);
            add(c, __fadd_rn(term(c), P.b01(Q.s[a - 1])), true);
        }
        if (near & 0x40000000u) {
            const Cand c = cand(part, 1);
            add(c, __fadd_rn(term(c), part == 0 ? P.b01(sb1) : P.i11(Q.s[a - 1], sb1)), true);
        }
        queue_rows<Cand>(
            lanes, part == 0 ? 1 : lm, [&](int k) { return row(part + k) & (k == 0 ? 0x3fffffffu : ~0u); },
            [&](int k, int l2) { return cand(part + k, l2); },
            [&](const Cand& c, bool has) { add(c, term(c), has); });
    }
    if (!live) return 0.0f;
    const float outside = __fsub_rn(T.F5o[b], Z);
    const float f5k = T.F5[a - 1];
    if (outside > CF_HALF32 && f5k > CF_HALF32) {
        const float jA = junctionA_rev<Lse32>(P, L, Q, a - 1, b);
        const float x = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(outside, f5k), fcin), P.ep()), bp_ab), jA);
        post = __fadd_rn(post, fexp32(pt, x));
    }
    if (post < 0.0f) post = 0.0f;
    else if (post > 1.0f) post = 1.0f;
    return post;
}

}  // namespace cf
