// cf_kernels.h -- kernel entry points and launch arguments (host + device).
#pragma once

#include <cstddef>
#include <cstdint>

#include "cf_device.cuh"

namespace cf {

constexpr int kFoldThreads = 256;       // threads per fold CTA
#ifndef CF_FOLD_MIN_BLOCKS
#define CF_FOLD_MIN_BLOCKS 3
#endif
constexpr int kFoldMinBlocks = CF_FOLD_MIN_BLOCKS;   // resident CTAs per SM the register budget targets
// ... and for the fused grouped MEA kernel alone (GB300, 10,000 x 200 nt MEA:
// 3, 4, 5 -> 250, 236, 250 ms, with the chain depth best for each)
#ifndef CF_FOLD_MIN_BLOCKS_MEA
#define CF_FOLD_MIN_BLOCKS_MEA 4
#endif
constexpr int kFoldMinBlocksMea = CF_FOLD_MIN_BLOCKS_MEA;
constexpr int kLatThreads = 512;    // threads of the one-CTA latency kernels (cf_latency.cu)
constexpr int kMaxGroup = 32;       // sequences per CTA on the batched path

struct FoldArgs {
    const SeqDesc* descs;      // [n], grouped: CTA b owns descs[b*group .. b*group+group)
    int n;
    int group;
    const uint8_t* seqs;       // ASCII
    const uint8_t* mask;       // nullable
    const float* blob32;
    const double* blob64;
    float* ws;                 // arena base
    float* logz;               // [batch] or null
    double* logz64;            // [batch] or null
    char* structs;             // dot-brackets at seq_off
    float* post_out;           // dense L*L per sequence or null
    const int64_t* post_offs;  // indexed by SeqDesc::idx
    float gamma;
    int* status;               // device status word (CF_OK or an error code)
};

// FP32 grouped kernels, kFoldThreads threads per CTA (cf_fold.cu)
using FoldKernel = void (*)(FoldArgs);
struct FoldKernels {
    FoldKernel inside, inside_acc, outside, posterior, mea;
    FoldKernel fused_mea, fused_bpp;   // k_fold_group32: all phases of MEA / BPP in one launch
    FoldKernel fused_mea_shared;       // fused MEA at the other kernels' register budget (shared device)
};
FoldKernels fold_kernels();
// Latency kernels (cf_latency.cu): one sequence on one CTA of kLatThreads, or
// on the 4 or kClusterCtas CTAs of a cluster, of kFoldThreads each.  They need
// lat_term_words(L) words behind the sequence's arena.
constexpr int kClusterCtas = 8;   // the largest portable cluster
struct LatKernels {
    FoldKernel mea, bpp, inside_acc;
};
LatKernels lat_kernels(bool cluster);   // kLatThreads threads; kFoldThreads in a cluster's CTAs
int64_t lat_term_words(int L);
constexpr int kLatStaticSmem = 18 * 1024;   // at most, beside the grouped kernels' dynamic shared memory
__global__ void k_inside64(FoldArgs A);
// Viterbi (cf_viterbi.cu): one sequence a CTA, up to kVitGroup, or one a cluster
__global__ void k_viterbi64(FoldArgs A);
__global__ void k_viterbi_group64(FoldArgs A);
__global__ void k_viterbi_cluster64(FoldArgs A);
constexpr int kVitGroup = 8;
constexpr int kVitStaticSmem = 32 * 1024;   // at most, beside fold_smem_bytes
// log-domain logZ of the sequences listed in fails (cf_linear.h), A.group at most on a CTA (cf_fold.cu)
__global__ void k_inside_redo32(FoldArgs A, const int* fails, bool mixed);
__global__ void k_inside_redo64(FoldArgs A, const int* fails, bool mixed);

size_t fold_smem_bytes(int Lmax, int group, bool fp64);

// Plain path: the reference's launch shape (cf_plain.cu), one sequence per CTA.
__global__ void k_plain_inside32(FoldArgs A);
__global__ void k_plain_outside32(FoldArgs A);
__global__ void k_plain_posterior32(FoldArgs A);
__global__ void k_plain_mea32(FoldArgs A);
size_t plain_smem_bytes(int Lmax);

// Adjoint (cf_adjoint.cu): inside with a soft unpaired bonus (FM2 kept on
// every ckpt-th diagonal), then the outside with the expected counts folded in.
// list (nullable): only the descs it names (cf_linear.h).
__global__ void k_adj_inside(FoldArgs A, const float* bonus, int ckpt, const int* list);
__global__ void k_adj_outside(FoldArgs A, const float* bonus, int ckpt, double* counts_out, double* unpaired_out,
                              const int* list);
size_t adj_smem_bytes(int Lmax);
int64_t adj_arena_words(int L, int ckpt);
int adj_auto_checkpoint(int L);

// Persistent fused per-sequence kernel (one CTA per sequence at a time).
enum { kCtaLogZ = 0, kCtaMea = 1, kCtaBpp = 2 };
template <int MODE>
__global__ void k_fold_cta(FoldArgs A, int* counter, int64_t slot_words);
const void* cta_kernel(int mode);

}  // namespace cf
