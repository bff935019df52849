// cf_linear.h -- the partition function as plain sums of products (cf_linear.cu):
// entry points, launch arguments and the weight tables they read.
#pragma once

#include <cstddef>
#include <cstdint>

#include "cf_device.cuh"

namespace cf {

// Longest sequence of the sum-of-products kernels.  float32 logZ of longer
// sequences stays with the log-domain kernels: their result carries the
// rounding bias of float32 log-sum-exp chains (measured on GB300 against 64
// bits, relative: 1e-6 at 128 nt, 5e-6 at 300, 1e-5 at 500, 4e-5 to 9e-5 at
// 1,000), and a sum without it would move the established values by more than
// 2e-5 there.
constexpr int kLinMaxLen = 512;
constexpr int kLinMaxLen64 = 416;   // double: what one CTA's shared memory holds (225 KB)
constexpr int kLinMaxLenGrad = 400;  // the gradient kernel's rings and sums (226 KB)
constexpr int kLinOutThreads = 512;
constexpr int kLinSmemMax = 232448;  // shared memory one CTA can have on sm_103a

// Every position costs a factor kLinScale, taken out of log Z again at the
// end: random sequences gain 0.02 to 0.13 nats a position, so scaled values
// stay near 1 (exactly representable, so no rounding in its powers' base).
#define CF_LIN_SCALE 0.9375
#define CF_LIN_LOG_SCALE (-0.064538521137571171672923915683993)   // log(15/16)

// Exponentials of the tied scores, made once per parameter set on the host
// (engine: cf_engine_set_params).
template <typename R>
struct LinWeights {
    // interior loops by total length t = l1 + l2: csf[t * 32 + l1] = cs(l1, t - l1),
    // zero where the cell takes the term itself (t < 2, and 1x1); read 16 bytes at a time
    alignas(16) R csf[31 * 32];
    R stack[625];     // bp is not part of it
    R close[625];     // hc + tm: the pair's own loop junction
    R bp[25], hc[25], dl[125], dr[125], i11[25];
    R hp[32];
    R b01[8];
    R mb, mu, mp, eu, ep, cs01, cs10, cs11;
};
void lin_weights(const double* blob, LinWeights<float>* w);
void lin_weights(const double* blob, LinWeights<double>* w);

struct LinArgs {
    const SeqDesc* descs;      // CTA b takes descs[first + b]
    int first;
    const uint8_t* seqs;
    const uint8_t* mask;       // nullable
    const void* weights;       // LinWeights<R>
    float* ws;                 // arena base
    void* logz;                // R[batch], written at SeqDesc::idx
    const float* bonus;        // gradients: unpaired bonus of each position, nullable
    double* counts;            // [batch][CF_BLOB_LEN]
    double* unpaired;          // at SeqDesc::seq_off
    int* fails;                // [0] count, [1 ..] indices into descs whose values left the range
};
struct LinKernel {
    void (*fn)(LinArgs);
    int threads;
};
// the inside of sequences of up to L nt; train: with bonuses, and the tables the derivatives need
LinKernel lin_inside_kernel(int L, bool fp64, bool train, bool narrow);   // narrow: 256 threads at most
int lin_class_end(int L, bool fp64);   // sequences up to this length share the launch of an L-nt one
size_t lin_inside_smem_bytes(int Lmax, bool fp64);
// gradients: the derivatives, after lin_inside_kernel(train)
__global__ void k_lin_outside32(LinArgs A);
size_t lin_outside_smem_bytes(int Lmax);

}  // namespace cf
