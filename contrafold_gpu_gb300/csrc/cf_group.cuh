// cf_group.cuh -- what the kernels that fold a group of sequences on one CTA or
// one thread-block cluster share: shared-memory layout and set-up, teams of
// threads, arena views.
#pragma once

#include "cf_kernels.h"
#include "cf_mea.cuh"
#include "cf_outside.cuh"

namespace cf {

// ---------------------------------------------------------------------------
// Shared memory: parameter tables + group descriptors, then per sequence the
// codes (s, pc) and the four partner bit sets.
// ---------------------------------------------------------------------------
template <typename R>
struct SmemFold {
    SmemTabs<R> tabs;
    PolyTables poly;
    int L[kMaxGroup];
    int64_t ws[kMaxGroup];
    int64_t soff[kMaxGroup];
    int idx[kMaxGroup];
    int n;        // sequences in this group
    int gcap;     // sequences per CTA of the launch (sizes the dynamic region)
    int Lmax;
    int step_ctr[2];   // per-step work counters of step_items (by step parity)
};

__host__ __device__ __forceinline__ int code_stride(int Lmax) { return (Lmax + 2 + 15) & ~15; }

// Item index of this thread when one serial item per thread is dealt over the
// warps first: thread (w, lane) takes item w + lane * warps.  A bijection of
// [0, blockDim.x).
__device__ __forceinline__ int tb_index() {
    return (threadIdx.x >> 5) + (threadIdx.x & 31) * (int)(blockDim.x >> 5);
}

template <typename R>
__device__ __forceinline__ unsigned char* dyn_smem(SmemFold<R>* sm) {
    return reinterpret_cast<unsigned char*>(sm + 1);
}

template <typename R>
__device__ __forceinline__ SeqV seq_v(SmemFold<R>* sm, int g) {
    const int cs = code_stride(sm->Lmax), W = pb_words(sm->Lmax);
    unsigned char* base = dyn_smem(sm);
    const uint8_t* s = base + (2 * g) * cs;
    const int8_t* pc = reinterpret_cast<const int8_t*>(base + (2 * g + 1) * cs);
    const uint32_t* PB = reinterpret_cast<const uint32_t*>(base + 2 * sm->gcap * cs) + (size_t)g * 4 * W;
    return SeqV{Codes{s}, pc, PB, W, sm->L[g]};
}

// Build codes and partner bit sets of the group's sequences (descriptors
// already in shared memory).
template <typename R>
__device__ __forceinline__ void build_group_seqs(SmemFold<R>* sm, const FoldArgs& A) {
    const int cs = code_stride(sm->Lmax), W = pb_words(sm->Lmax);
    unsigned char* base = dyn_smem(sm);
    for (int g = 0; g < sm->n; ++g) {
        uint8_t* s = base + (2 * g) * cs;
        int8_t* pc = reinterpret_cast<int8_t*>(base + (2 * g + 1) * cs);
        uint32_t* PB = reinterpret_cast<uint32_t*>(base + 2 * sm->gcap * cs) + (size_t)g * 4 * W;
        build_seq(A.seqs, A.mask, sm->soff[g], sm->L[g], W, s, pc, PB);
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Teams: the threads that fold one group together.  CtaTeam is one CTA (the
// batched kernels, which take no other); ClusterTeam is the C CTAs of a
// thread-block cluster, on C SMs (the latency and the Viterbi kernels).  Work of a diagonal step
// is split over tid() / nthreads(); sync() separates steps (a cluster barrier
// with release / acquire semantics for ClusterTeam, so table cells written in
// global memory by one CTA are read by the others after it).  Every sync() is
// reached by all threads of the team: the loops around them run the same trip
// counts in every CTA (each CTA loads the same group descriptors), and
// rank-0-only work sits between two syncs, not around one.
// ---------------------------------------------------------------------------
struct CtaTeam {
    __device__ __forceinline__ int rank() const { return 0; }
    __device__ __forceinline__ int size() const { return 1; }
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int nthreads() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};

struct ClusterTeam {
    int r, c;   // rank of this CTA in the cluster, cluster size
    __device__ __forceinline__ int rank() const { return r; }
    __device__ __forceinline__ int size() const { return c; }
    __device__ __forceinline__ int tid() const { return r * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ int nthreads() const { return c * blockDim.x; }
    __device__ __forceinline__ void sync() const {
        asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
    }
};

__device__ __forceinline__ int cluster_ctarank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return (int)r;
}

__device__ __forceinline__ int cluster_nctas() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(r));
    return (int)r;
}

// Load tables, group descriptors, sequence codes and partner bit sets of
// group `gi` (default: this CTA's index).
template <typename R>
__device__ __forceinline__ void setup_group(SmemFold<R>* sm, const FoldArgs& A, const R* __restrict__ gblob,
                                            int gi = -1) {
    const int g0 = (gi < 0 ? (int)blockIdx.x : gi) * A.group;
    const int ng = min(A.group, A.n - g0);
    if (threadIdx.x == 0) {
        int lmax = 0;
        for (int g = 0; g < ng; ++g) {
            const SeqDesc D = A.descs[g0 + g];
            sm->L[g] = D.L;
            sm->ws[g] = D.ws_off;
            sm->soff[g] = D.seq_off;
            sm->idx[g] = D.idx;
            lmax = max(lmax, D.L);
        }
        sm->n = ng;
        sm->gcap = A.group;
        sm->Lmax = lmax;
    }
    load_tabs(&sm->tabs, gblob);
    load_poly_tables(&sm->poly);
    __syncthreads();
    build_group_seqs(sm, A);
}

// ---------------------------------------------------------------------------
// Arena views
// ---------------------------------------------------------------------------
template <typename R>
struct InView {
    InTabs<R> T;
    R* FB;        // two FM2 step buffers of stride fbs
    int fbs;
    PairList PLs;
};

template <typename R>
__device__ __forceinline__ InView<R> in_view(const FoldArgs& A, int64_t ws_off, int L) {
    InView<R> V;
    if (sizeof(R) == 4) {
        const Arena32 a = arena32(L);
        float* base = A.ws + ws_off;
        V.T.FC = reinterpret_cast<R*>(base + a.FC);
        V.T.FM = reinterpret_cast<R*>(base + a.FM);
        V.T.FM1 = reinterpret_cast<R*>(base + a.FM1);
        V.T.F5 = reinterpret_cast<R*>(base + a.F5);
        V.FB = reinterpret_cast<R*>(base + a.FB);
        V.PLs = plist_at(base + a.PL, L);
    } else {
        const Arena64 a = arena64(L);
        double* base = reinterpret_cast<double*>(A.ws + ws_off);
        V.T.FC = reinterpret_cast<R*>(base + a.FC);
        V.T.FM = reinterpret_cast<R*>(base + a.FM);
        V.T.FM1 = reinterpret_cast<R*>(base + a.FM1);
        V.T.F5 = reinterpret_cast<R*>(base + a.F5);
        V.FB = reinterpret_cast<R*>(base + a.FB);
        V.PLs = plist_at(A.ws + ws_off + a.PL, L);
    }
    V.T.m = L + 1;
    V.T.sized(L);
    V.fbs = (int)pad32(L + 2);
    return V;
}

__device__ __forceinline__ OutTabs out_tabs(const FoldArgs& A, int64_t ws_off, int L) {
    const Arena32 a = arena32(L);
    float* base = A.ws + ws_off;
    OutTabs T;
    T.FC = base + a.FC; T.FM = base + a.FM; T.FM1 = base + a.FM1; T.F5 = base + a.F5;
    T.FCo = base + a.FCo; T.FMo = base + a.FMo; T.FM1o = base + a.FM1o; T.FM2o = base + a.FM2o;
    T.F5o = base + a.F5o;
    T.m = L + 1;
    T.sized(L);
    return T;
}

__device__ __forceinline__ PairList plist_of(const FoldArgs& A, int64_t ws_off, int L) {
    return plist_at(A.ws + ws_off + arena32(L).PL, L);
}

// Posterior of every pairable pair; POST goes to the FMo slot (triangular,
// zero elsewhere) and, for cf_bpp, densely into the caller's L x L matrix.
template <class Team = CtaTeam>
__device__ __forceinline__ void posterior_group(SmemFold<float>* sm, const FoldArgs& A, const Team tm = Team{}) {
    for (int g = 0; g < sm->n; ++g) {
        const int L = sm->L[g];
        float* POST = out_tabs(A, sm->ws[g], L).FMo;
        const int64_t tot = tri_size(L);
        for (int64_t c = tm.tid(); c < tot; c += tm.nthreads()) POST[c] = 0.0f;
        if (A.post_out) {
            float* dense = A.post_out + A.post_offs[sm->idx[g]];
            for (int64_t c = tm.tid(); c < (int64_t)L * L; c += tm.nthreads()) dense[c] = 0.0f;
        }
    }
    tm.sync();
    for (int g = 0; g < sm->n; ++g) {
        const SeqV Q = seq_v(sm, g);
        const int L = Q.L, m = L + 1;
        const OutTabs T = out_tabs(A, sm->ws[g], L);
        const PairList PLs = plist_of(A, sm->ws[g], L);
        const float Z = T.F5[L];
        float* POST = T.FMo;
        float* dense = A.post_out ? A.post_out + A.post_offs[sm->idx[g]] : nullptr;
        // pairable FC cells (i, i+d) <-> pairs (a, b) = (i, i+d+1), in list
        // order, whole warps at a time (team thread k takes entries k, k + nthreads, ...)
        const int total = PLs.poff[L + 1];
        const int lane = threadIdx.x & 31;
        for (int c0 = tm.tid() - lane; c0 < total; c0 += tm.nthreads()) {
            const int c = c0 + lane;
            const unsigned lanes = __ballot_sync(0xffffffffu, c < total);
            if (c >= total) continue;
            const int d = plist_diag(PLs, L, c);
            const int a = PLs.pl[c], b = a + d + 1;
            const float v = posterior_pair(&sm->tabs, &sm->poly, Q, T, Z, a, b, lanes);
            POST[tri_off(d + 1, m) + a] = v;
            if (dense != nullptr) dense[(int64_t)(a - 1) * L + (b - 1)] = v;
        }
    }
    tm.sync();
    if (A.logz != nullptr && tm.rank() == 0)
        for (int g = threadIdx.x; g < sm->n; g += blockDim.x) {
            const OutTabs T = out_tabs(A, sm->ws[g], sm->L[g]);
            A.logz[sm->idx[g]] = T.F5[sm->L[g]];
        }
}

// Walk diagonals d = d_begin .. d_end (step +1) over all sequences of the
// group; call f(g, i, i + d) for every cell.  One barrier per diagonal.
template <typename R, class Team, typename F>
__device__ __forceinline__ void wavefront(SmemFold<R>* sm, const Team& tm, int d_begin, int d_end, int step, F f) {
    const int ng = sm->n;
    for (int d = d_begin; step > 0 ? d <= d_end : d >= d_end; d += step) {
        int total = 0;
        for (int g = 0; g < ng; ++g) total += max(0, sm->L[g] + 1 - d);
        for (int c = tm.tid(); c < total; c += tm.nthreads()) {
            int g = 0, r = c;
            while (true) {
                const int cnt = max(0, sm->L[g] + 1 - d);
                if (r < cnt) break;
                r -= cnt;
                ++g;
            }
            f(g, r, r + d);
        }
        tm.sync();
    }
}

// MEA decode (cpu.py:823-895): unpaired weights, gamma-weighted max-plus DP
// with the reference's strict-'>' candidate order, BFS traceback.
template <class Team = CtaTeam>
__device__ __forceinline__ void mea_group(SmemFold<float>* sm, const FoldArgs& A, const Team tm = Team{}) {
    const float two_g = __fmul_rn(2.0f, A.gamma);
    for (int g = 0; g < sm->n; ++g) {
        const int L = sm->L[g];
        const Arena32 ar = arena32(L);
        float* base = A.ws + sm->ws[g];
        for (int i = 1 + tm.tid(); i <= L; i += tm.nthreads()) base[ar.up + i] = mea_unpaired(base + ar.FMo, L, two_g, i);
    }
    tm.sync();
    wavefront(sm, tm, 0, sm->Lmax, +1, [&](int g, int i, int j) {
        const SeqV Q = seq_v(sm, g);
        const Arena32 ar = arena32(Q.L);
        float* base = A.ws + sm->ws[g];
        mea_cell(Q, base + ar.FMo, base + ar.up, base + ar.FM2o, reinterpret_cast<int*>(base + ar.FM), Q.L, i, j);
    });
    for (int g = 0; g < sm->n; ++g) {
        const int L = sm->L[g];
        char* out = A.structs + sm->soff[g];
        for (int t = tm.tid(); t < L; t += tm.nthreads()) out[t] = '.';
    }
    tm.sync();
    // one traceback per thread, dealt over the warps first (lane 0 of every
    // warp, then lane 1, ...): lanes of one warp with different tracebacks
    // would run them one after another
    if (tm.rank() == 0)
        for (int g = tb_index(); g < sm->n; g += blockDim.x) {
            const int L = sm->L[g];
            const Arena32 ar = arena32(L);
            float* base = A.ws + sm->ws[g];
            int* qi = reinterpret_cast<int*>(base + ar.queue);
            mea_traceback(reinterpret_cast<const int*>(base + ar.FM), L, qi, qi + 2 * L + 4, A.structs + sm->soff[g],
                          A.status);
        }
    tm.sync();
}

// ---------------------------------------------------------------------------
// One sequence on a team, warps taking items of unlike kinds (cf_latency.cu,
// cf_viterbi.cu)
// ---------------------------------------------------------------------------
constexpr int kWindowMax = (CMAX + 1) * (CMAX + 2) / 2;   // interior loops of one cell at most

__device__ __forceinline__ int warp_exclusive(int v, int lane, int& total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// The candidates of a cell in the order of its rows: every lane lists its
// row's (mask msk, packed l1 | bit << 5, highest bit first) behind the rows
// before it.  Returns how many.
__device__ __forceinline__ int window_list(uint32_t msk, int l1, uint16_t* list, int lane) {
    int total;
    int at = warp_exclusive(__popc(msk), lane, total);
    while (msk) {
        const int bit = 31 - __clz(msk);
        msk ^= 1u << bit;
        list[at++] = (uint16_t)(l1 | bit << 5);
    }
    __syncwarp();
    return total;
}

// Claims the items of one step: item() runs for every index of this CTA's share
template <typename R, class Team, class Item>
__device__ __forceinline__ void run_items(SmemFold<R>* sm, const Team& tm, int step, int total, Item item) {
    int* ctr = &sm->step_ctr[step & 1];
    if (threadIdx.x == 0) sm->step_ctr[(step & 1) ^ 1] = 0;
    const int lane = threadIdx.x & 31;
    for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(ctr, 1);
        q = __shfl_sync(0xffffffffu, q, 0) * tm.size() + tm.rank();
        if (q >= total) break;
        item(q, lane);
    }
    tm.sync();
}

}  // namespace cf
