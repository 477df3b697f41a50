// Tensor-core path of layers with GROUPED scales, and of INT8 activations on any layer, from a few dozen
// tokens up to the batched sizes:
//   y[m,n] = bf16( s[m] * (sum_k q[m,k] * cb[idx[n,k/d], k%d] * scale[n, k/G]) + bias[n] )
//
// The layouts the reference deployed (dim-4 vectors, one scale per 64 weights, 5- to 11-bit
// indices; gr00t_libero/acceleration/presets/FROZEN_DECODE_SELECTION.json) change their scale inside
// the K loop, so it has to be folded into the weight operand, and codeword x scale has 16 significant
// bits.  The split-K kernel (linear_split_k.cu, fp16 forms) multiplies fp16(codeword x scale) -- 11
// significant bits, finer than the bf16 rounding of the reference's own reconstruction -- or, at few
// tokens, that product as two fp16 numbers and so exactly, by the activation bytes widened to fp16
// (exact) in a pre-pass into the caller's workspace.
//
// Replaces, for M above a few dozen rows, the reference's per-forward decode kernel plus 8-bit
// GEMM on these layouts (perrow_int8_fused_decode_r1.py:12-88, perrow_a8_candidate_r3.py:56-69).
#include "common.cuh"
#include "split_k.cuh"
#include "widen.cuh"

namespace sacq {

namespace {

constexpr int64_t kSlabTokens = 1024;   // tokens widened per launch: bounds the fp16 scratch

SplitMode form_of(bool exact) { return exact ? kSplitHalf2 : kSplitHalf; }

}  // namespace

int64_t large_m_grouped_slab(void) { return kSlabTokens; }

// The kernels that this one takes over from at few tokens multiply exact weights: the index-unpacking kernel up to 32, 47
// or 95 tokens, the CUDA-core and fp16 warp-MMA kernels of INT8 activations up to 47, and any number of tokens where the
// codebook does not fit shared memory.  There it splits its weights into two fp16 numbers (2048 -> 2048 at 47 tokens,
// INT8, d = 4: 8.4 us with 11 bits, 9.9 exact, 60 on the CUDA-core kernel; 2048 -> 6144 at 32, e4m3: 10.7 / 11.7 / 22.8).
// Beyond, weights of 11 bits, finer than the bf16 reconstruction.  A kernel chosen by its selector has one form at
// every size.
bool large_m_grouped_exact(const sacq_layer* L, int64_t M, bool int8) {
  if (!split_k_codebook_in_smem(L)) return true;
  if (int8) return M < 48;
  if (L->force_kernel == 7) return false;
  return M < (L->order_rows >= 32 * (int64_t)L->num_sms ? 33 : L->order_rows >= 2048 ? 48 : 96);
}

bool large_m_grouped_supported(const sacq_layer* L) { return L->d.index_bits >= 1 && L->split_tok[kSplitHalf] > 0; }

// Whether the persistent kernel for grouped scales takes a call that shared memory leaves this one narrow tiles for, or none:
// from where the weights need not be exact, if it is modelled to be faster by a margin (its model was fitted to shallower
// layers: K = 28,672, 4,096 rows, d = 4, 11-bit, group 64 at 1,000 tokens: modelled 0.5 ms, measured 0.82).
bool large_m_grouped_cedes(const sacq_layer* L, int64_t M, bool int8) {
  const bool exact = large_m_grouped_exact(L, M, int8);
  if (exact || split_k_tiles_fit(L, M, form_of(exact)) || !large_m_tmem_grouped_supported(L)) return false;
  if (!large_m_grouped_supported(L)) return true;
  const int64_t rows = M < kSlabTokens ? M : kSlabTokens;
  SplitChoice c;
  return !split_k_choose(L, rows, form_of(exact), &c) || 1.6 * large_m_tmem_grouped_us(L, M) < c.us * (double)M / (double)rows;
}

// Workspace behind the counter region: the fp16 activations of one token slab.
int64_t large_m_grouped_workspace_bytes(const sacq_layer* L, int64_t M) {
  const int64_t rows = M < kSlabTokens ? M : kSlabTokens;
  return (rows * L->d.in_features * 2 + 255) & ~(int64_t)255;
}

int launch_large_m_grouped(const sacq_layer* L, const void* q, const float* scale, int64_t M, void* y, int64_t ldy,
                           void* ws, int64_t ws_bytes, cudaStream_t s, const void* residual, int64_t ldr,
                           ActForm form, bool exact, const BcastDst* bc, const SplitChoice* cut) {
  if (!large_m_grouped_supported(L))
    return set_error(SACQ_ERR_UNSUPPORTED, "grouped tensor-core kernel cannot run this layer geometry");
  if (M <= 0 || L->d.out_features == 0) return SACQ_OK;
  if (reinterpret_cast<uintptr_t>(q) % 8 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "quantized activations must be 8-byte aligned");
  if (form == kActHalf) {
    SplitChoice c;
    const SplitMode mode = form_of(exact);
    if (M > kSlabTokens || (cut == nullptr && !split_k_choose(L, M, mode, &c)))
      return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld exceeds a slab", (long long)M);
    return launch_split_k(&L, 1, q, scale, M, &y, &ldy, mode, cut != nullptr ? *cut : c, s, residual, ldr, bc);
  }
  const int64_t need = large_m_grouped_workspace_bytes(L, M);
  if (ws == nullptr || ws_bytes < need)
    return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed behind the counter region, %lld given",
                     (long long)need, (long long)ws_bytes);
  if (reinterpret_cast<uintptr_t>(ws) % 256 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  const int64_t K = L->d.in_features;
  const SplitMode mode = form_of(exact);
  for (int64_t m0 = 0; m0 < M; m0 += kSlabTokens) {
    const int64_t rows = (M - m0) < kSlabTokens ? (M - m0) : kSlabTokens;
    if (int rc = launch_widen(static_cast<const uint8_t*>(q) + m0 * K, rows, K, form == kActInt8, ws, s)) return rc;
    SplitChoice c;
    if (cut != nullptr && M <= kSlabTokens) c = *cut;
    else if (!split_k_choose(L, rows, mode, &c)) return set_error(SACQ_ERR_UNSUPPORTED, "grouped tensor-core kernel: no tile fits");
    BcastDst slab{};
    for (int i = 0; bc != nullptr && i < bc->n; ++i) slab.ptr[slab.n++] = static_cast<uint16_t*>(bc->ptr[i]) + m0 * ldy;
    void* y_slab = static_cast<uint16_t*>(y) + m0 * ldy;
    const int rc = launch_split_k(&L, 1, ws, scale + m0, rows, &y_slab, &ldy, mode, c, s,
                                  residual ? static_cast<const uint16_t*>(residual) + m0 * ldr : nullptr, ldr,
                                  bc ? &slab : nullptr);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}

// Sibling layers of one geometry: the shared activations are widened once and the GEMMs run as one launch,
// byte-identical to separate calls.  SACQ_ERR_UNSUPPORTED (nothing launched) when they cannot share one.
int launch_large_m_grouped_multi(const sacq_layer* const* layers, int n, const void* q, const float* scale, int64_t M,
                                 void* const* ys, const int64_t* ldys, void* ws, int64_t ws_bytes, cudaStream_t s) {
  if (n < 2 || n > kSplitMaxLayers || M <= 0 || M > kSlabTokens || reinterpret_cast<uintptr_t>(q) % 8 != 0)
    return SACQ_ERR_UNSUPPORTED;
  const bool exact = large_m_grouped_exact(layers[0], M, false);
  for (int l = 0; l < n; ++l)
    if (!large_m_grouped_supported(layers[l]) || large_m_grouped_exact(layers[l], M, false) != exact) return SACQ_ERR_UNSUPPORTED;
  if (ws == nullptr || ws_bytes < large_m_grouped_workspace_bytes(layers[0], M) || reinterpret_cast<uintptr_t>(ws) % 256 != 0)
    return SACQ_ERR_UNSUPPORTED;
  SplitChoice c;
  if (!split_k_choose_multi(layers, n, M, form_of(exact), &c)) return SACQ_ERR_UNSUPPORTED;
  if (int rc = launch_widen(q, M, layers[0]->d.in_features, false, ws, s)) return rc;
  return launch_split_k(layers, n, ws, scale, M, ys, ldys, form_of(exact), c, s);
}

}  // namespace sacq
