// cf_fold.cu -- fold kernels: inside (FP32 / FP64), outside, posterior, MEA
// decode.
//
// Scheduling: a CTA owns a GROUP of sequences (group size 1 is the plain
// one-sequence-per-block path of gpu.py:508; larger groups are the batched
// path).  The CTA walks the DP diagonals of all its sequences in lock step;
// on each diagonal the threads take the cells of every sequence of the group
// (flattened), so short diagonals of several sequences fill the warps that one
// sequence alone would leave idle.  One barrier separates diagonals.  (Batches
// that leave most of the device idle: cf_latency.cu.)
#include "cf_group.cuh"
#include "cf_mea.cuh"

namespace cf {

// ---------------------------------------------------------------------------
// One pipelined step over the group: phase-B items (pairable cells of
// diagonal dB, from the pair lists) then phase-A items (every cell of
// diagonal dA).  The B block is padded to a multiple of 32 so that each warp
// holds one kind of item.  fB(g, i), fA(g, i) process one cell.
//
// Warps claim 32-item chunks from a shared counter (B chunks, the costlier
// window walks, come first), so a warp that drew cheap cells takes more and
// the step's barrier waits less for the slowest warp.  Step `t` uses counter
// t & 1 and clears the other one for step t + 1 (nobody uses it after the
// previous step's barrier); both start at zero (step_ctr_init).
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ void step_ctr_init(SmemFold<R>* sm) {
    if (threadIdx.x == 0) sm->step_ctr[0] = sm->step_ctr[1] = 0;
    __syncthreads();
}

template <typename R, class Team, typename GetPL, typename FB, typename FA>
__device__ __forceinline__ void step_items(SmemFold<R>* sm, const Team& tm, int t, int dB, int dA, GetPL getpl, FB fB, FA fA) {
    const int ng = sm->n;
    int NB = 0, NA = 0;
    for (int g = 0; g < ng; ++g) {
        const int L = sm->L[g];
        if (dB >= 0 && dB <= L - 2) {
            const PairList PLs = getpl(g);
            NB += PLs.poff[dB + 1] - PLs.poff[dB];
        }
        if (dA >= 0) NA += max(0, L + 1 - dA);
    }
    const int NB32 = (NB + 31) & ~31;
    const int total = NB32 + NA;
    int* ctr = &sm->step_ctr[t & 1];
    if (threadIdx.x == 0) sm->step_ctr[(t & 1) ^ 1] = 0;
    const int lane = threadIdx.x & 31;
    for (;;) {
        // the CTA's q-th chunk is chunk q * size + rank of the team's step
        int q = 0;
        if (lane == 0) q = atomicAdd(ctr, 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        const int base = (q * tm.size() + tm.rank()) * 32;
        if (base >= total) break;
        const int c = base + lane;
        if (c >= total) continue;   // only in the last A chunk (the B block is whole warps)
        if (c < NB32) {
            // B items fill whole warps (NB32 is a multiple of 32): the lanes
            // holding a cell walk it together (see inside_B)
            const unsigned lanes = __ballot_sync(0xffffffffu, c < NB);
            if (c >= NB) continue;
            int r = c, g = 0;
            for (;; ++g) {
                const int L = sm->L[g];
                if (dB <= L - 2) {
                    const PairList PLs = getpl(g);
                    const int o = PLs.poff[dB], cnt = PLs.poff[dB + 1] - o;
                    if (r < cnt) { fB(g, (int)PLs.pl[o + r], lanes); break; }
                    r -= cnt;
                }
            }
        } else {
            int r = c - NB32, g = 0;
            for (;; ++g) {
                const int cnt = max(0, sm->L[g] + 1 - dA);
                if (r < cnt) { fA(g, r); break; }
                r -= cnt;
            }
        }
    }
    tm.sync();
}

// ---------------------------------------------------------------------------
// Inside (any semiring): pair lists, FC/FM/FM1 wavefront, F5.
// ---------------------------------------------------------------------------
template <class S>
__device__ __forceinline__ S make_sr(const PolyTables* pt);
template <>
__device__ __forceinline__ Lse32 make_sr<Lse32>(const PolyTables* pt) { return Lse32{pt}; }
template <>
__device__ __forceinline__ LseAcc32 make_sr<LseAcc32>(const PolyTables*) { return LseAcc32{}; }
template <>
__device__ __forceinline__ Lse64 make_sr<Lse64>(const PolyTables*) { return Lse64{}; }

template <class S, class Team = CtaTeam>
__device__ __forceinline__ void inside_group(SmemFold<typename S::Real>* sm, const FoldArgs& A, const Team tm = Team{}) {
    using R = typename S::Real;
    const S sr = make_sr<S>(&sm->poly);
    if (tm.rank() == 0)
        for (int g = 0; g < sm->n; ++g) build_plist(seq_v(sm, g), in_view<R>(A, sm->ws[g], sm->L[g]).PLs);
    if (tm.size() > 1) tm.sync();   // the pair lists, for every CTA of the team
    auto getpl = [&](int g) { return in_view<R>(A, sm->ws[g], sm->L[g]).PLs; };
    step_ctr_init(sm);
    for (int t = 0; t <= sm->Lmax + 1; ++t) {
        step_items(
            sm, tm, t, t - 1, t <= sm->Lmax ? t : -1, getpl,
            [&](int g, int i, unsigned lanes) {   // phase B(t-1): FC of a pairable cell
                const SeqV Q = seq_v(sm, g);
                const InView<R> V = in_view<R>(A, sm->ws[g], Q.L);
                const R fm2 = V.FB[((t - 1) & 1) * V.fbs + i];
                inside_B<S>(sr, &sm->tabs, Q, V.T, i, i + t - 1, fm2, lanes);
            },
            [&](int g, int i) {   // phase A(t): FM2, FM1, FM
                const SeqV Q = seq_v(sm, g);
                const InView<R> V = in_view<R>(A, sm->ws[g], Q.L);
                V.FB[(t & 1) * V.fbs + i] = inside_A<S>(sr, &sm->tabs, Q, V.T, i, i + t);
            });
    }
    // exterior recurrence: one warp per sequence
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (tm.rank() == 0)
        for (int g = warp; g < sm->n; g += nwarps)
            exterior_warp<S>(sr, &sm->tabs, seq_v(sm, g), in_view<R>(A, sm->ws[g], sm->L[g]).T);
    tm.sync();
}

__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_inside32(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    inside_group<Lse32>(sm, A);
    if (A.logz != nullptr)
        for (int g = threadIdx.x; g < sm->n; g += blockDim.x)
            A.logz[sm->idx[g]] = in_view<float>(A, sm->ws[g], sm->L[g]).T.F5[sm->L[g]];
}

// Same recurrence with accurate float32 log-sum-exp: logZ_batch and the sampler.
__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_inside32acc(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    inside_group<LseAcc32>(sm, A);
    if (A.logz != nullptr)
        for (int g = threadIdx.x; g < sm->n; g += blockDim.x)
            A.logz[sm->idx[g]] = in_view<float>(A, sm->ws[g], sm->L[g]).T.F5[sm->L[g]];
}

__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_inside64(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<double>*>(smem_raw);
    setup_group(sm, A, A.blob64);
    inside_group<Lse64>(sm, A);
    for (int g = threadIdx.x; g < sm->n; g += blockDim.x)
        A.logz64[sm->idx[g]] = in_view<double>(A, sm->ws[g], sm->L[g]).T.F5[sm->L[g]];
}

// Sequences that the sum-of-products kernels left (fails[0] of them, descs
// indices fails[1 ..]; usually none), in the log domain.  How many there are is
// known here only, so each CTA takes as many of them together as the host's rule
// gives a batch of that size, A.group at most: as few waves as that allows, or
// two where lengths are mixed (GB300, the whole logZ call: 1,000 hairpins of 124
// nt 20.2 ms with one a CTA in turn, 9.8 so; 500 of 304 nt 46.4, 35.3).
template <class S>
__device__ __forceinline__ void inside_redo(const FoldArgs& A, const int* fails, bool mixed, const typename S::Real* blob,
                                            typename S::Real* out) {
    using R = typename S::Real;
    const int n = fails[0], slots = gridDim.x;
    if (n == 0) return;
    const int waves = (n + A.group * slots - 1) / (A.group * slots);
    const int group = mixed ? min(A.group, max(1, (n + slots) / (2 * slots))) : (n + waves * slots - 1) / (waves * slots);
    if ((int)blockIdx.x * group >= n) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<R>*>(smem_raw);
    load_tabs(&sm->tabs, blob);
    load_poly_tables(&sm->poly);
    for (int k = blockIdx.x * group; k < n; k += slots * group) {
        __syncthreads();
        if (threadIdx.x == 0) {
            sm->n = min(group, n - k);
            sm->gcap = A.group;
            sm->Lmax = 0;
            for (int g = 0; g < sm->n; ++g) {
                const SeqDesc D = A.descs[fails[1 + k + g]];
                sm->L[g] = D.L;
                sm->ws[g] = D.ws_off;
                sm->soff[g] = D.seq_off;
                sm->idx[g] = D.idx;
                sm->Lmax = max(sm->Lmax, D.L);
            }
        }
        __syncthreads();
        build_group_seqs(sm, A);
        inside_group<S>(sm, A);
        for (int g = threadIdx.x; g < sm->n; g += blockDim.x)
            out[sm->idx[g]] = in_view<R>(A, sm->ws[g], sm->L[g]).T.F5[sm->L[g]];
    }
}
__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_inside_redo32(FoldArgs A, const int* fails, bool mixed) {
    inside_redo<LseAcc32>(A, fails, mixed, A.blob32, A.logz);
}
__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_inside_redo64(FoldArgs A, const int* fails, bool mixed) {
    inside_redo<Lse64>(A, fails, mixed, A.blob64, A.logz64);
}

// ---------------------------------------------------------------------------
// Outside + posterior + MEA (FP32)
// ---------------------------------------------------------------------------
template <class Team = CtaTeam>
__device__ __forceinline__ void outside_group(SmemFold<float>* sm, const FoldArgs& A, const Team tm = Team{}) {
    const Lse32 sr{&sm->poly};
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (tm.rank() == 0)
        for (int g = warp; g < sm->n; g += nwarps)
            exterior_outside_warp(sr, &sm->tabs, seq_v(sm, g), out_tabs(A, sm->ws[g], sm->L[g]));
    tm.sync();
    auto getpl = [&](int g) { return plist_of(A, sm->ws[g], sm->L[g]); };
    step_ctr_init(sm);
    for (int t = sm->Lmax; t >= 0; --t) {
        step_items(
            sm, tm, t, t - 1, t, getpl,
            [&](int g, int a, unsigned lanes) {   // phase B(t-1): FCo of a pairable cell
                const SeqV Q = seq_v(sm, g);
                outside_B(sr, &sm->tabs, Q, out_tabs(A, sm->ws[g], Q.L), a, a + t - 1, lanes);
            },
            [&](int g, int a) {   // phase A(t): FMo, FM1o, FM2o
                const SeqV Q = seq_v(sm, g);
                outside_A(sr, &sm->tabs, Q, out_tabs(A, sm->ws[g], Q.L), a, a + t);
            });
    }
}

__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_outside32(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    outside_group(sm, A);
}

__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_posterior32(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    posterior_group(sm, A);
}

// MEA decode (cpu.py:823-895): unpaired weights, gamma-weighted max-plus DP
// with the reference's strict-'>' candidate order, BFS traceback.
__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_mea32(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    mea_group(sm, A);
}

// ---------------------------------------------------------------------------
// Fused grouped fold: one launch runs inside -> outside -> posterior -> MEA
// decode (MODE 0) or posterior into the caller's matrices (MODE 1) for the
// CTA's group.  MODE 2 is MODE 0 built for the register budget of the other
// fold kernels (kFoldMinBlocks per SM instead of kFoldMinBlocksMea): on a
// device shared with them, a CTA of any of them fits the slot another frees
// (an 80-register CTA never fits where a 64-register one left).  Each CTA goes on to its next phase as soon as its own group
// is done, instead of every phase waiting for the slowest CTA of the grid.
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kFoldThreads, MODE == 0 ? kFoldMinBlocksMea : kFoldMinBlocks) k_fold_group32(FoldArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    setup_group(sm, A, A.blob32);
    if constexpr (MODE == 0 || MODE == 2) {
        inside_group<Lse32>(sm, A);
        outside_group(sm, A);
        __syncthreads();
        FoldArgs Ap = A;
        Ap.post_out = nullptr;
        Ap.logz = nullptr;
        posterior_group(sm, Ap);
        mea_group(sm, A);
    } else {
        inside_group<Lse32>(sm, A);
        outside_group(sm, A);
        __syncthreads();
        posterior_group(sm, A);
    }
}

// ---------------------------------------------------------------------------
// Persistent fused fold: each CTA takes one sequence at a time from a device
// work queue and runs inside -> outside -> posterior -> MEA decode (or the
// inside alone for logZ) before taking the next.  Only one or two sequences
// per SM are in flight, so the DP tables that every diagonal step re-reads
// stay resident in L2; the CTA's arena slot is reused across sequences.
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kFoldThreads, kFoldMinBlocks) k_fold_cta(FoldArgs A, int* counter, int64_t slot_words) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto* sm = reinterpret_cast<SmemFold<float>*>(smem_raw);
    __shared__ int item_s;
    load_tabs(&sm->tabs, A.blob32);
    load_poly_tables(&sm->poly);
    const int64_t slot = (int64_t)blockIdx.x * slot_words;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int item = atomicAdd(counter, 1);
            item_s = item;
            if (item < A.n) {
                const SeqDesc D = A.descs[item];
                sm->L[0] = D.L;
                sm->ws[0] = slot;
                sm->soff[0] = D.seq_off;
                sm->idx[0] = D.idx;
                sm->n = 1;
                sm->gcap = 1;
                sm->Lmax = D.L;
            }
        }
        __syncthreads();
        if (item_s >= A.n) break;
        build_group_seqs(sm, A);
        if constexpr (MODE == kCtaLogZ) {
            inside_group<LseAcc32>(sm, A);
            if (threadIdx.x == 0) A.logz[sm->idx[0]] = in_view<float>(A, sm->ws[0], sm->L[0]).T.F5[sm->L[0]];
            continue;
        }
        inside_group<Lse32>(sm, A);
        outside_group(sm, A);
        __syncthreads();
        posterior_group(sm, A);
        if constexpr (MODE == kCtaMea) mea_group(sm, A);
    }
}

template __global__ void k_fold_cta<kCtaLogZ>(FoldArgs, int*, int64_t);
template __global__ void k_fold_cta<kCtaMea>(FoldArgs, int*, int64_t);
template __global__ void k_fold_cta<kCtaBpp>(FoldArgs, int*, int64_t);

const void* cta_kernel(int mode) {
    switch (mode) {
        case kCtaLogZ: return (const void*)k_fold_cta<kCtaLogZ>;
        case kCtaMea: return (const void*)k_fold_cta<kCtaMea>;
        default: return (const void*)k_fold_cta<kCtaBpp>;
    }
}

// ---------------------------------------------------------------------------
FoldKernels fold_kernels() {
    return {k_inside32, k_inside32acc, k_outside32, k_posterior32, k_mea32,
            k_fold_group32<0>, k_fold_group32<1>, k_fold_group32<2>};
}

size_t fold_smem_bytes(int Lmax, int group, bool fp64) {
    const size_t head = fp64 ? sizeof(SmemFold<double>) : sizeof(SmemFold<float>);
    return head + 2 * (size_t)code_stride(Lmax) * group + (size_t)group * 4 * pb_words(Lmax) * 4;
}

}  // namespace cf
