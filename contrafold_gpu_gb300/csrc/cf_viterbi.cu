// cf_viterbi.cu -- Viterbi: max-plus inside in FP64, then the reference's EPS
// first-match traceback (cpu.py:302-501).
//
// A maximum does not depend on the order of its candidates, so nothing of a
// cell is serial: per diagonal one warp takes the interior loops of a pairable
// cell (candidates listed, 32 evaluated at a time, a butterfly), a warp takes a
// sixth of the multiloop splits of 32 cells, one the exterior recurrence's next
// step, and after a barrier a thread a cell joins them.  Each candidate is the
// reference's sum, rounded as there, so tables are its tables.
//
// The FP64 pipe bounds the fold of a full device (two adds or compares a cycle
// and SM: 81 % busy on 1,216 x 200 nt while 23 % of the issue slots are used),
// so what need not be an FP64 add is none: maxima compare ordered integers (see
// key), and cs + bp, a candidate's first sum, comes from a table.  That leaves
// a window candidate three adds of six operations and a split one of two.
#include "cf_group.cuh"

namespace cf {
namespace {

constexpr int kVitParts = 6;   // of a cell's splits; their maxima lie in the traceback stack's place
constexpr int kVitWarps = kFoldThreads / 32;

// Doubles as integers in the same order (and back).
__device__ __forceinline__ long long key(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double unkey(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ long long warp_max(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// cs(l1, l2) + bp of the six pairs, the first sum of a window candidate
struct LoopScores {
    double v[6][kWindowMax];
};
// slot of (l1, l2), rows l1 ascending; and the pair (x, y)'s number
__device__ __forceinline__ int loop_slot(int l1, int l2) { return l1 * (CMAX + 1) - ((l1 * (l1 - 1)) >> 1) + l2; }
__device__ __forceinline__ int pair_number(int x, int y) {
    constexpr unsigned long long N = 0ull << (4 * 3) | 1ull << (4 * 12) | 2ull << (4 * 6) | 3ull << (4 * 9) |
                                     4ull << (4 * 11) | 5ull << (4 * 14);   // AU UA CG GC GU UG
    return (int)(N >> (4 * (x * 4 + y))) & 7;
}
__device__ __forceinline__ void load_loop_scores(LoopScores* t, const SmemTabs<double>* tb) {
    const ParamView<double> P{tb->blob};
    const int x[6] = {0, 3, 1, 2, 2, 3}, y[6] = {3, 0, 2, 1, 3, 2};
    for (int k = threadIdx.x; k < 6 * (CMAX + 1) * (CMAX + 1); k += blockDim.x) {
        const int l1 = k / 6 / (CMAX + 1), l2 = k / 6 % (CMAX + 1);
        if (l1 + l2 <= CMAX) {
            double bp = 0.0;
#pragma unroll
            for (int n = 0; n < 6; ++n)
                if (n == k % 6) bp = P.bp(x[n], y[n]);
            t->v[k % 6][loop_slot(l1, l2)] = __dadd_rn(P.cs(l1, l2), bp);
        }
    }
}

// Largest interior-loop candidate of cell (i, j) (inside_B's terms).
__device__ __forceinline__ long long window_max(const SmemTabs<double>* __restrict__ tb, const LoopScores* __restrict__ ls,
                                                const SeqV& Q, const InTabs<double>& T, int i, int j, uint16_t* list,
                                                int lane) {
    const ParamView<double> P{tb->blob};
    const int m = T.m, d = j - i;
    const int si = Q.s[i], sj1 = Q.s[j + 1], si1 = Q.s[i + 1], sj = Q.s[j];
    const double jB = tb->jB(si, sj1, si1, sj);
    // row l1: q from j - C(l1) to j
    const int C0 = d - 2 < CMAX ? d - 2 : CMAX;
    const uint32_t msk = lane <= C0 ? Q.window(i + lane + 1, j - C0 + lane, C0 - lane + 1) : 0u;
    const int total = window_list(msk, lane, list, lane);
    long long best = key(CF_NEG64);
    for (int k0 = lane; k0 < total; k0 += 128) {
        int c[4];
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = list[min(k0 + 32 * u, total - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int l1 = c[u] & 31, l2 = C0 - l1 - (c[u] >> 5);
            v[u] = T.FC[tri_off(d - 2 - l1 - l2, m) + i + l1 + 1];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int l1 = c[u] & 31, l2 = C0 - l1 - (c[u] >> 5);
            const int cq = Q.s.pair(j - l2), cp = Q.s.pair(i + l1);   // (s[q], s[q + 1]), (s[p], s[p + 1])
            const int sq = (cq * 205) >> 10, sa = cp - 5 * ((cp * 205) >> 10);
            double e;
            if (l1 + l2 == 0) {
                e = __dadd_rn(P.bp(si1, sj), P.stack(si, sj1, si1, sj));
            } else {
                e = __dadd_rn(__dadd_rn(ls->v[pair_number(sa, sq)][loop_slot(l1, l2)], jB), tb->jb[cq * 25 + cp].jB);
                if (l1 < 2 && l2 < 2)   // 1-nt bulges and 1x1 (the zero that other loops add changes no maximum)
                    e = __dadd_rn(e, l1 == 0 ? P.b01(sj) : l2 == 0 ? P.b01(si1) : P.i11(si1, sj));
            }
            best = max(best, key(__dadd_rn(e, v[u])));
        }
    }
    __syncwarp();
    return warp_max(best);
}

// Warp 0's traceback: a state's candidates in the reference's order, 32 at a
// time; the first that matches the state's value within EPS is taken.
__device__ void viterbi_traceback(const SmemTabs<double>* tb, const SeqV& Q, const InTabs<double>& T, int* st, char* out,
                                  int* status, int lane) {
    const ParamView<double> P{tb->blob};
    const int L = Q.L;
    const double EPS = 1e-6, HALF = CF_HALF64;
    const int cap = 4 * L + 16;
    int *st_t = st, *st_i = st + cap, *st_j = st + 2 * cap;
    int sp = 0;
    bool full = false;
    auto push = [&](int t, int i, int j) {
        if (sp >= cap) {
            full = true;
            return;
        }
        if (lane == 0) {
            st_t[sp] = t;
            st_i[sp] = i;
            st_j[sp] = j;
        }
        ++sp;
    };
    auto pair = [&](int a, int b) {
        if (lane == 0) {
            out[a - 1] = '(';
            out[b - 1] = ')';
        }
    };
    // first k in [lo, hi) whose candidate matches, or -1
    auto first = [&](int lo, int hi, auto match) {
        for (int k0 = lo; k0 < hi; k0 += 32) {
            const int k = k0 + lane;
            const unsigned hit = __ballot_sync(0xffffffffu, k < hi && match(k));
            if (hit) return k0 + __ffs(hit) - 1;
        }
        return -1;
    };
    push(0, 0, L);
    while (sp > 0 && !full) {
        --sp;
        __syncwarp();
        const int typ = st_t[sp], i = st_i[sp], j = st_j[sp];
        __syncwarp();
        auto near = [&](double v, double val) { return fabs(__dadd_rn(v, -val)) <= EPS; };
        if (typ == 0) {
            if (j == 0) continue;
            const double val = T.F5[j], prev = T.F5[j - 1];
            if (prev > HALF && near(__dadd_rn(prev, P.eu()), val)) {
                push(0, 0, j - 1);
                continue;
            }
            const int k = first(0, j, [&](int k) {
                if (!Q.pairable(k + 1, j)) return false;
                const double fcin = T.FC[T.at(k + 1, j - 1)], f5k = T.F5[k];
                if (!(fcin > HALF) || !(f5k > HALF)) return false;
                const double jA = junctionA_rev<Max64>(P, L, Q, k, j);
                return near(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(f5k, fcin), P.ep()), P.bp(Q.s[k + 1], Q.s[j])), jA), val);
            });
            if (k >= 0) {
                pair(k + 1, j);
                push(1, k + 1, j - 1);
                push(0, 0, k);
            }
        } else if (typ == 1) {
            const double val = T.FC[T.at(i, j)];
            const int si = Q.s[i], sj1 = Q.s[j + 1], si1 = Q.s[i + 1], sj = Q.s[j];
            const double jB = tb->jB(si, sj1, si1, sj);
            const int d = j - i;
            if (near(__dadd_rn(jB, P.hp(d <= DHP ? d : DHP)), val)) continue;
            bool done = false;
            const int pmax = (i + CMAX < j) ? i + CMAX : j;
            for (int p = i; p <= pmax && !done; ++p) {   // a row of the window: q = j - lane
                const int l1 = p - i, q = j - lane, l2 = lane;
                const int qmin = p + 2 > l1 + j - CMAX ? p + 2 : l1 + j - CMAX;
                bool hit = false;
                if (q >= qmin && Q.pairable(p + 1, q)) {
                    const double inner = T.FC[T.at(p + 1, q - 1)];
                    if (inner > HALF) {
                        double e;
                        if (l1 == 0 && l2 == 0) {
                            e = __dadd_rn(P.bp(si1, sj), P.stack(si, sj1, si1, sj));
                        } else {
                            const double jB2 = tb->jB(Q.s[q], Q.s[p + 1], Q.s[q + 1], Q.s[p]);
                            double snuc = 0.0;
                            if (l1 == 0 && l2 == 1) snuc = P.b01(sj);
                            else if (l1 == 1 && l2 == 0) snuc = P.b01(si1);
                            else if (l1 == 1 && l2 == 1) snuc = P.i11(si1, sj);
                            e = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(P.cs(l1, l2), P.bp(Q.s[p + 1], Q.s[q])), jB), jB2), snuc);
                        }
                        hit = near(__dadd_rn(e, inner), val);
                    }
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                if (hits) {
                    const int b = j - (__ffs(hits) - 1);
                    pair(p + 1, b);
                    push(1, p + 1, b - 1);
                    done = true;
                }
            }
            if (done) continue;
            const double jA = junctionA<Max64>(P, L, Q, i, j);
            const int k = first(i + 1, j, [&](int k) {
                const double f1 = T.FM1[T.at(i, k)], fm = T.FM[T.at(k, j)];
                return f1 > HALF && fm > HALF &&
                       near(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(f1, fm), jA), P.mp()), P.mb()), val);
            });
            if (k >= 0) {
                push(3, i, k);
                push(2, k, j);
            }
        } else if (typ == 2) {
            const double val = T.FM[T.at(i, j)];
            const int k = first(i + 1, j, [&](int k) {
                const double f1 = T.FM1[T.at(i, k)], fm = T.FM[T.at(k, j)];
                return f1 > HALF && fm > HALF && near(__dadd_rn(f1, fm), val);
            });
            if (k >= 0) {
                push(3, i, k);
                push(2, k, j);
                continue;
            }
            const double prev = T.FM[T.at(i, j - 1)], f1 = T.FM1[T.at(i, j)];
            if (prev > HALF && near(__dadd_rn(prev, P.mu()), val)) push(2, i, j - 1);
            else if (f1 > HALF && near(f1, val)) push(3, i, j);
        } else {
            const double val = T.FM1[T.at(i, j)];
            if (Q.pairable(i + 1, j)) {
                const double fin = T.FC[T.at(i + 1, j - 1)];
                if (fin > HALF) {
                    const double jAji = junctionA_rev<Max64>(P, L, Q, i, j);
                    if (near(__dadd_rn(__dadd_rn(__dadd_rn(fin, jAji), P.mp()), P.bp(Q.s[i + 1], Q.s[j])), val)) {
                        pair(i + 1, j);
                        push(1, i + 1, j - 1);
                        continue;
                    }
                }
            }
            const double ext = T.FM1[T.at(i + 1, j)];
            if (ext > HALF && near(__dadd_rn(ext, P.mu()), val)) push(3, i + 1, j);
        }
    }
    if (full && lane == 0) atomicExch(status, CF_EDEVICE);
}

// A sequence's tables; parts ([kVitParts][L + 4]) lie in the traceback stack's
// place, wmax ([i]) in the step buffers, both keys.
struct VitSeq {
    SeqV Q;
    InView<double> V;
    int* stack;
    long long *parts, *wmax;
};
__device__ __forceinline__ VitSeq vit_seq(SmemFold<double>* sm, const FoldArgs& A, int g) {
    VitSeq X;
    X.Q = seq_v(sm, g);
    X.V = in_view<double>(A, sm->ws[g], X.Q.L);
    X.stack = reinterpret_cast<int*>(A.ws + sm->ws[g] + arena64(X.Q.L).stack);
    X.parts = reinterpret_cast<long long*>(X.stack);
    X.wmax = reinterpret_cast<long long*>(X.V.FB);
    return X;
}
__device__ __forceinline__ int vit_pairs(const VitSeq& X, int d) {   // pairable cells of diagonal d
    return d <= X.Q.L - 2 ? X.V.PLs.poff[d + 1] - X.V.PLs.poff[d] : 0;
}
__device__ __forceinline__ int vit_splits(int L, int d) {            // items of its splits
    return d >= 2 ? kVitParts * ((max(0, L - 1 - d) + 31) >> 5) : 0;
}

// F5[d]: FC of spans up to d - 2
__device__ __forceinline__ void vit_exterior(const SmemTabs<double>* tb, const VitSeq& X, int d, int lane) {
    const ParamView<double> P{tb->blob};
    const SeqV& Q = X.Q;
    const InTabs<double>& T = X.V.T;
    if (d < 1) return;
    long long best = key(CF_NEG64);
    for (int k = lane; k < d; k += 32) {
        if (!Q.pairable(k + 1, d)) continue;
        const double fcin = T.FC[T.at(k + 1, d - 1)], f5k = T.F5[k];
        if (!(fcin > CF_HALF64) || !(f5k > CF_HALF64)) continue;
        const double jA = junctionA_rev<Max64>(P, Q.L, Q, k, d);
        best = max(best, key(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(f5k, fcin), P.ep()), P.bp(Q.s[k + 1], Q.s[d])), jA)));
    }
    best = max(warp_max(best), key(__dadd_rn(T.F5[d - 1], P.eu())));
    if (lane == 0) T.F5[d] = unkey(best);
}

// Item u of the splits of diagonal d: a part of 32 inner cells'.
__device__ __forceinline__ void vit_split(const VitSeq& X, int d, int u, int lane) {
    const InTabs<double>& T = X.V.T;
    const int L = X.Q.L, m = T.m, part = u % kVitParts, i = 1 + (u / kVitParts) * 32 + lane;
    if (i > max(0, L - 1 - d)) return;
    constexpr int N = kVitParts, H = N * (N - 1) / 2;
    int s = 1 + part;
    int o1 = tri_off(s, m) + i, o2 = tri_off(d - s, m) + i + s;
    int d1 = N * m - N * s - H, d2 = N * (d - s) - N * m - N * N + H + N;   // see cf_linear.cu, dot_tri
    long long best = key(CF_NEG64);
#pragma unroll 4
    for (; s < d; s += N) {
        best = max(best, key(__dadd_rn(T.FM1[o1], T.FM[o2])));
        o1 += d1;
        d1 -= N * N;
        o2 += d2;
        d2 -= N * N;
    }
    X.parts[part * (L + 4) + i] = best;
}

// Joins the items of cell (i, i + d).
__device__ __forceinline__ void vit_join(const SmemTabs<double>* tb, const VitSeq& X, int d, int i) {
    const ParamView<double> P{tb->blob};
    const SeqV& Q = X.Q;
    const InTabs<double>& T = X.V.T;
    const double NEG = CF_NEG64, HALF = CF_HALF64;
    const int L = Q.L, ps = L + 4, j = i + d, at = tri_off(d, T.m) + i;
    double fc = NEG, fm1 = NEG, fm = NEG;
    if (i > 0 && j < L) {
        long long k2 = key(NEG);
        if (d >= 2) {
#pragma unroll
            for (int p = 0; p < kVitParts; ++p) k2 = max(k2, X.parts[p * ps + i]);
        }
        const double fm2 = unkey(k2);
        if (Q.pairable(i, j + 1)) {
            const double jB = tb->jB(Q.s[i], Q.s[j + 1], Q.s[i + 1], Q.s[j]);
            fc = unkey(max(key(__dadd_rn(jB, P.hp(d <= DHP ? d : DHP))), X.wmax[i]));
            if (fm2 > HALF)
                fc = fmax(fc, __dadd_rn(__dadd_rn(__dadd_rn(fm2, junctionA<Max64>(P, L, Q, i, j)), P.mp()), P.mb()));
        }
        if (d >= 2) {
            const double fin = T.FC[T.at(i + 1, j - 1)], ext = T.FM1[T.at(i + 1, j)], prev = T.FM[T.at(i, j - 1)];
            if (Q.pairable(i + 1, j) && fin > HALF)
                fm1 = __dadd_rn(__dadd_rn(__dadd_rn(fin, junctionA_rev<Max64>(P, L, Q, i, j)), P.mp()),
                                P.bp(Q.s[i + 1], Q.s[j]));
            if (ext > HALF) fm1 = fmax(fm1, __dadd_rn(ext, P.mu()));
            if (fm2 > HALF) fm = fm2;
            if (prev > HALF) fm = fmax(fm, __dadd_rn(prev, P.mu()));
            if (fm1 > HALF) fm = fmax(fm, fm1);
        }
    }
    T.FC[at] = fc;
    T.FM1[at] = fm1;
    T.FM[at] = fm;
}

// What a fold begins with: no pairs yet, the pair list, F5[0].
template <class Team>
__device__ __forceinline__ void vit_begin(SmemFold<double>* sm, const FoldArgs& A, const Team& tm, const VitSeq& X, int g) {
    if (tm.rank() == 0) build_plist(X.Q, X.V.PLs);
    if (tm.rank() == 0 && threadIdx.x == 0) X.V.T.F5[0] = 0.0;
    for (int t = tm.tid(); t < X.Q.L; t += tm.nthreads()) A.structs[sm->soff[g] + t] = '.';
}

struct VitShared {
    uint16_t lists[kVitWarps][kWindowMax];
    LoopScores ls;
};

template <class Team>
__device__ __forceinline__ void viterbi_fold(const FoldArgs& A, const Team& tm, int gi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<double>*>(smem_raw);
    __shared__ VitShared sh;
    uint16_t* list = sh.lists[threadIdx.x >> 5];
    setup_group(sm, A, A.blob64, gi);
    load_loop_scores(&sh.ls, &sm->tabs);
    const VitSeq X = vit_seq(sm, A, 0);
    const int L = X.Q.L;
    if (threadIdx.x == 0) sm->step_ctr[0] = sm->step_ctr[1] = 0;
    vit_begin(sm, A, tm, X, 0);
    tm.sync();
    for (int d = 0; d <= L; ++d) {
        const int nE = vit_pairs(X, d), oE = nE ? X.V.PLs.poff[d] : 0;
        run_items(sm, tm, d, 1 + nE + vit_splits(L, d), [&](int q, int lane) {
            if (q == 0) {
                vit_exterior(&sm->tabs, X, d, lane);
            } else if (q <= nE) {
                const int i = X.V.PLs.pl[oE + q - 1];
                const long long w = window_max(&sm->tabs, &sh.ls, X.Q, X.V.T, i, i + d, list, lane);
                if (lane == 0) X.wmax[i] = w;
            } else {
                vit_split(X, d, q - 1 - nE, lane);
            }
        });
        for (int i = tm.tid(); i + d <= L; i += tm.nthreads()) vit_join(&sm->tabs, X, d, i);
        tm.sync();
    }
    if (tm.rank() == 0 && threadIdx.x < 32)
        viterbi_traceback(&sm->tabs, X.Q, X.V.T, X.stack, A.structs + sm->soff[0], A.status, threadIdx.x);
}

// The same for a group of very short sequences on a CTA (rule: cf_engine.cu):
// alone, each has fewer items a diagonal than the CTA has warps.
__device__ __forceinline__ void viterbi_group(const FoldArgs& A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<double>*>(smem_raw);
    __shared__ VitShared sh;
    __shared__ int npair[2][kVitGroup];   // pairable cells of a diagonal, by its parity
    uint16_t* list = sh.lists[threadIdx.x >> 5];
    const CtaTeam tm;
    setup_group(sm, A, A.blob64);
    load_loop_scores(&sh.ls, &sm->tabs);
    const int ng = sm->n, tid = threadIdx.x;
    if (tid == 0) sm->step_ctr[0] = sm->step_ctr[1] = 0;
    for (int g = 0; g < ng; ++g) vit_begin(sm, A, tm, vit_seq(sm, A, g), g);
    __syncthreads();
    if (tid < ng) npair[0][tid] = vit_pairs(vit_seq(sm, A, tid), 0);
    __syncthreads();
    for (int d = 0; d <= sm->Lmax; ++d) {
        auto items = [&](int g) { return d > sm->L[g] ? 0 : 1 + npair[d & 1][g] + vit_splits(sm->L[g], d); };
        int total = 0, cells = 0;
        for (int g = 0; g < ng; ++g) {
            total += items(g);
            cells += max(0, sm->L[g] + 1 - d);
        }
        run_items(sm, tm, d, total, [&](int q, int lane) {
            int g = 0;
            for (int n; q >= (n = items(g)); ++g) q -= n;
            const VitSeq X = vit_seq(sm, A, g);
            const int nE = npair[d & 1][g];
            if (q == 0) {
                vit_exterior(&sm->tabs, X, d, lane);
            } else if (q <= nE) {
                const int i = X.V.PLs.pl[X.V.PLs.poff[d] + q - 1];
                const long long w = window_max(&sm->tabs, &sh.ls, X.Q, X.V.T, i, i + d, list, lane);
                if (lane == 0) X.wmax[i] = w;
            } else {
                vit_split(X, d, q - 1 - nE, lane);
            }
        });
        if (tid < ng) npair[(d + 1) & 1][tid] = vit_pairs(vit_seq(sm, A, tid), d + 1);
        for (int c = tid; c < cells; c += kFoldThreads) {
            int g = 0, i = c;
            for (int n; i >= (n = max(0, sm->L[g] + 1 - d)); ++g) i -= n;
            vit_join(&sm->tabs, vit_seq(sm, A, g), d, i);
        }
        __syncthreads();
    }
    for (int g = tid >> 5; g < ng; g += kVitWarps) {
        const VitSeq X = vit_seq(sm, A, g);
        viterbi_traceback(&sm->tabs, X.Q, X.V.T, X.stack, A.structs + sm->soff[g], A.status, tid & 31);
    }
}

}  // namespace

__global__ void __launch_bounds__(kFoldThreads, 3) k_viterbi64(FoldArgs A) { viterbi_fold(A, CtaTeam{}, blockIdx.x); }
__global__ void __launch_bounds__(kFoldThreads, 3) k_viterbi_group64(FoldArgs A) { viterbi_group(A); }
__global__ void __launch_bounds__(kFoldThreads, 2) k_viterbi_cluster64(FoldArgs A) {
    const int c = cluster_nctas();
    viterbi_fold(A, ClusterTeam{cluster_ctarank(), c}, (int)blockIdx.x / c);
}

}  // namespace cf
