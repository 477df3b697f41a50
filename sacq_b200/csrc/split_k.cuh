// Interface of the cluster split-K tensor-core kernel (linear_split_k.cu).
#pragma once

#include <stdint.h>

#include "common.cuh"

namespace sacq {

constexpr int kSplitMaxLayers = 4;    // sibling layers of one launch

// What the weight operand of a call is:
enum SplitMode {
  kSplitHiLo = 0,   // e4m3 high and low halves of the codewords, e4m3 activations; one scale per row
  kSplitHalf = 1,   // fp16(codeword x scale), activations widened to fp16: grouped scales, INT8 activations
  kSplitHalf2 = 2,  // the same product as two fp16 numbers, exactly: its 16 significant bits are 11 and 5
  kSplitInt8 = 3,   // the INT8 recipe's weight bytes, int8 activations, int32 sums
  kSplitFp8 = 4     // the FP8 recipe's weight bytes, e4m3 activations
};

// How one call is cut up: token tiles of `tok` tokens, clusters of `split` CTAs with `parts` slices of K each.
struct SplitChoice {
  int tok = 0, tiles = 0, split = 0, parts = 1, act_stages = 0, max_slices = 0, max_groups = 0;
  int box_shift = 2;            // logarithm of the 16-byte index slices per box
  bool own_recv = false;        // whether the partial sums of a cluster have shared memory of their own
  double us = 1e30;             // modelled time
};

// Fills sacq_layer::split_tok, once, when the layer is made.
void split_k_init(sacq_layer* L);
// Whether shared memory leaves the call the tiles that the model wants.  A CTA holds the packed indices of its whole slice
// of K, so deep layers have room for narrow tiles only, each of which expands the weights again.
bool split_k_tiles_fit(const sacq_layer* L, int64_t M, SplitMode mode);

// The best cut for M tokens (at most kSplitMaxM); false if the kernel cannot run the layer in that form.
constexpr int64_t kSplitMaxM = 1 << 19;
bool split_k_choose(const sacq_layer* L, int64_t M, SplitMode mode, SplitChoice* out);

// The same for several layers in one launch; false if they are not of one geometry.
bool split_k_choose_multi(const sacq_layer* const* layers, int n, int64_t M, SplitMode mode, SplitChoice* out);

// n layers of one geometry (n = 1: the plain launch) on one set of activations: bytes [M, K], or for kSplitHalf
// and kSplitHalf2 the activations already widened to fp16 [M, K].  row_scale: the recipes' per-row weight scales [N] (n = 1).
int launch_split_k(const sacq_layer* const* layers, int n, const void* act, const float* scale, int64_t M, void* const* ys,
                   const int64_t* ldys, SplitMode mode, const SplitChoice& c, cudaStream_t s, const void* residual = nullptr,
                   int64_t ldr = 0, const BcastDst* bc = nullptr, const float* row_scale = nullptr, const void* x = nullptr,
                   int64_t x_pitch = 0);
// Whether the CTAs of a kSplitHiLo call cut up like that can quantize the tokens themselves (launch_split_k with x: bf16 rows
// that are 16-byte aligned, instead of act and scale): their rows fit shared memory.
bool split_k_quantizes(const sacq_layer* L, const SplitChoice& c);
int64_t split_k_ctas(const sacq_layer* L, const SplitChoice& c);
// Whether the layer's codebook fits the kernel's shared memory (else it is gathered from L2).
bool split_k_codebook_in_smem(const sacq_layer* L);
// Whether the quantizer in front of a call of M tokens should be the one that shares SMs with this kernel (act_quant.cu).
// Not where the codebook is gathered through L1, which the quantizer's carve-out would take from the SM (65,536 entries,
// 2048 -> 6144 at 16 tokens 11.3 / 14.4 us), not for wide layers of several waves (2048 -> 6144 at 700 27.5 / 27.6; 2048 -> 2048
// 13.7 / 12.2), and not where the chip has room for the CTAs of two GEMMs and the quantizer's beside each other (INT8, 2048 -> 1024,
// d = 4, at 40 tokens 9.6 / 9.9; at the edge, 2048 -> 1536 INT8 at 64 with 2 x 48 + 64 CTAs, 7.8 / 7.6 in a graph, but 7.7 / 8.2
// eager), which deep layers with their longer rows need not wait for (6144 -> 1536 at 64, as many CTAs, 10.4 / 9.5).
Beside split_k_beside(const sacq_layer* L, int64_t M, const SplitChoice& c);
void split_k_release(sacq_layer* L);

}  // namespace sacq
