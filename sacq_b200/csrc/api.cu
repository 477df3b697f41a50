// C ABI of libsacq_b200: layer handles, argument checking, kernel selection.
// The kernels live in dequant.cu, act_quant.cu, linear_small_m.cu, linear_large_m.cu.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>

#include "common.cuh"
#include "host/internal.h"
#include "split_k.cuh"

static_assert(sizeof(sacq_layer_desc) == 88, "sacq_layer_desc layout is part of the ABI");

namespace sacq {

namespace {
thread_local char g_error[512] = "";
std::atomic<long long> g_launches{0};
constexpr int64_t kCounterBytes = 64 * 1024;  // 16384 row-block arrival counters
}  // namespace

int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return set_error(SACQ_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
}

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

namespace {

// Runs `fn` with the layer's device current, restoring the caller's device afterwards.
struct DeviceGuard {
  int prev = -1;
  bool ok = true;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
    if (prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
  }
  ~DeviceGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

int check_layer(const sacq_layer_t* L) {
  if (L == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "layer handle is null");
  return SACQ_OK;
}

// Rows per launch of the small-M kernel so that its arrival counters fit their region.
int64_t small_m_slab_rows(const sacq_layer* L) {
  const int64_t row_blocks = (L->d.out_features + 31) / 32;
  int64_t chunks = (kCounterBytes / (int64_t)sizeof(int)) / (row_blocks > 0 ? row_blocks : 1);
  if (chunks < 1) chunks = 1;
  return chunks * 16;
}

// Rows of a layer in whole row tiles of the split-K kernel.
int64_t tiled_rows(const sacq_layer* L) { return (L->d.out_features + 127) / 128 * 128; }

// Rows from which the grouped split-K kernel takes over from the index-unpacking warp-MMA kernel, which walks the
// weights once per 48 tokens and multiplies exact weights (quantizer + GEMM, d = 4, 10-bit, group 64: 2048x6144 19.0 / 10.1 us
// at 32 rows; 2048x2048 9.2 / 7.8 and 6144x2048 20.5 / 12.8 at 47, there with weights of 11 bits, which up to 47 rows would be
// less than before; the smallest lose a tenth, 1024x1024 5.4 / 6.0).  With exact weights, a forward and a call on quantized
// activations, which this kernel has to widen, in a graph as shares of the other kernel's time:
//  * on the widest layers from the ninth row on, if they have many vectors (d = 4, at 9 / 16 rows: 2048x6144 0.91 / 0.89 and
//    0.96 / 0.94, 3072x5632 0.73 / 0.72 and 0.77 / 0.78; 2048x5000 0.95 / 0.91 and 0.99 / 0.98, but eager 0.99 / 0.96 and 1.03 / 1.02;
//    3072x4736, fewer row tiles, 0.97 / 0.96 and 1.20 / 1.20; below nine rows gains and losses are even);
//  * on 4,096 rows from the second chunk on (at 17 / 32: 1024x4096 0.66 / 0.73 and 0.77 / 0.75, 3072x4096 0.81 / 0.78 and 0.95 / 0.91,
//    d = 8 0.84 / 0.81 and 0.99 / 0.96; at 16 eager 1024x4096 6.2 / 7.6 us, the other one being a single launch);
//  * on deep layers from the third on (at 32 / 33: 6144x2048 0.93 / 0.76 and 1.14 / 0.91, 4096x2048 0.93 / 0.77 and 1.11 / 0.91).
//    Codebooks of up to 32 entries gain as much, but the tests hold the other kernel's bytes on them;
//  * not on smaller ones (2048x2048 at 41 9.2 / 10.0 us, 4096x1024 9.2 / 10.5).
int64_t grouped_min_m(const sacq_layer* L) {
  // ... or from the CUDA-core kernel, at any number (2048x2048, 65,536 entries, group 128: 127 / 11 us at 17 rows)
  if (L->small_m_warps == 0) return 1;
  const int64_t rows = tiled_rows(L);
  if (rows >= 44 * 128) return L->d.in_features * rows / L->d.vector_dim >= (3 << 20) ? 9 : 17;
  if (L->d.out_features >= 4096) return 17;
  return L->d.in_features >= 4096 && L->d.in_features * L->d.out_features >= (8 << 20) && L->d.index_bits > 5 ? 33 : 48;
}
// From how many tokens the persistent kernel with the weights in tensor memory takes over; its 128-row tiles need that many
// to fill the device.  The split-K kernel expands a wide layer again for every second 384-token tile, from about 700 tokens
// on in a second wave (1024x4096 at 1,000 tokens 23.5 / 12.6 us, 2048x6144 39 / 24).  It keeps them up to 960 all the same:
// the two sum in different orders, and up to there the tokens of a request get the same bytes alone and in a batch of
// three (the price: 2048x6144 at 700 tokens 30.6 / 19.4).  Below 1,024 of K they do sum alike, but there sibling layers gain by the
// split-K kernel's shared launch what one layer loses (768x4096 at 560 9.7 / 9.1, two of them 11.2 / 16.2).  A codebook that is
// gathered from L2 makes an expansion twice as dear (2048x6144 at 400 30.4 / 28.7).  Narrower layers lose nothing (2048x2048
// at 1,000 17.6 / 16.3, 6144x1536 30 / 37).
int64_t tmem_min_m(const sacq_layer* L) {
  if (L->d.out_features < 4096) return 1024;
  return split_k_codebook_in_smem(L) ? 960 : 384;
}

// From how many tokens a split-K kernel, which walks the weights once, beats a small-M kernel, which walks them
// once per 16-token chunk: from the second chunk on wide or deep layers, from the third on all but the smallest.
// A codebook in L2 leaves the small-M kernel 2 warps' gathers in flight per scheduler: the split-K kernel wins from one
// token on (65,536 entries, 2048x6144: 17.4 / 11.3 us at 16 tokens; 6144x2048 13.4 / 11.1 at one, 13.7 / 11.5 at 16;
// 2048x2048 7.2 / 7.0 and 7.6 / 7.1), on the smallest layers from the second chunk on (2048x1024 6.4 / 7.2 at 16 and
// 7.6 / 7.2 at 32, 1024x1024 5.5 / 5.8 and 6.4 / 5.8).
// Dim-8 layers of 4,096 rows and more, shares of the small-M kernel's time in a graph / eager:
//  * 12 M weights: from one token on (2048x6144 0.93 / 0.93 at one, 0.90 / 0.94 at 16; 3072x4096 0.95 / 0.96 and 0.94 / 0.90; 4096x4096
//    0.93 / 0.89 and 0.89 / 0.85; 2048x8192 0.80 / 0.82 and 0.70 / 0.75).  2048x5120 gains as much (0.92 / 0.93), but the tests hold the
//    small-M kernel's bytes on 5,992 rows of 2,048, a row tile below the line; 1536x6144 is even (1.00 / 0.99 and 0.95 / 0.98);
//  * at most 1,024 of K: from where the split-K kernel alone quantizes in the same launch (1024x4096 eager 7.5 / 5.5 us at eight; at one
//    token 5.6 / 5.4 on one host, 6.5 / 7.1 on another).
// Narrower deep layers keep the small-M kernel (6144x2048 8.0 / 8.3 at eight), and so do dim-4 vectors, whose bytes up to 16
// tokens the tests hold (2048x6144 8.8 / 7.8).
bool split_wins(const sacq_layer* L, int64_t M) {
  const int64_t work = L->d.in_features * L->d.out_features;
  if (!split_k_codebook_in_smem(L)) return M > 16 || work > (2 << 20) || L->d.out_features >= 4096;
  if (L->d.out_features >= 4096 && L->d.vector_dim == 8 &&
      (L->d.in_features * tiled_rows(L) >= (12 << 20) || (L->d.in_features <= 1024 && M > L->small_m_warps)))
    return true;
  return (M > 16 && (L->d.out_features >= 4096 || work >= (8 << 20))) || M > 32;
}

// Whether the persistent kernel takes a call that shared memory leaves the split-K kernel narrow tiles for: if it is
// modelled to be faster.
bool large_m_cedes(const sacq_layer* L, int64_t M) {
  SplitChoice c;
  return !split_k_tiles_fit(L, M, kSplitHiLo) && large_m_tmem_supported(L) &&
         (!split_k_choose(L, M, kSplitHiLo, &c) || large_m_tmem_us(L, M) < c.us);
}

int pick_kernel(const sacq_layer* L, int64_t M) {
  if (is_shard(L)) {                                   // whether a kernel can run a layer does not depend on its width
    const sacq_layer whole = whole_layer(L);
    return pick_kernel(&whole, M);
  }
  if (L->force_kernel == 7) return large_m_grouped_supported(L) ? 3 : SACQ_ERR_UNSUPPORTED;
  if (L->force_kernel >= 12) return large_m_tmem_grouped_supported(L) ? 5 : SACQ_ERR_UNSUPPORTED;
  if (L->force_kernel >= 8) return large_m_tmem_supported(L) ? 4 : SACQ_ERR_UNSUPPORTED;
  if (L->force_kernel == 1 || L->force_kernel >= 3)
    return small_m_supported(L) ? 1 : SACQ_ERR_UNSUPPORTED;
  if (L->force_kernel == 2) return large_m_supported(L) ? 2 : SACQ_ERR_UNSUPPORTED;
  // A shape rule, not a backend switch.  The tensor-core kernels sum in an order that depends on K alone (the staged warp-MMA
  // kernel on its tile class too, see make_plan), so the row shards of a split layer reproduce the whole layer bit for bit
  // where they run the same kernel.  Thresholds depend on the width, hence the whole layer's.
  if (large_m_tmem_supported(L) && M >= tmem_min_m(L)) return 4;
  // Below, quantizer + GEMM of the small-M and the split-K kernel at 17 tokens: 1024x4096 10.9 / 6.8 us,
  // 6144x2048 15.4 / 11.5, 2048x6144 15.5 / 8.9; at 33: 1024x1024 7.3 / 5.7, 2048x2048 9.2 / 8.8, 4096x1024
  // 9.5 / 9.2, 2048x1024 even.
  if (large_m_supported(L)) {
    if (split_wins(L, M)) return large_m_cedes(L, M) ? 4 : 2;
  } else if (large_m_tmem_supported(L)) {              // a layer too deep for the split-K kernel
    if (M >= (L->d.out_features >= 32 * (int64_t)L->num_sms ? 17 : 49)) return 4;
  } else if (large_m_tmem_grouped_supported(L) && M >= large_m_tmem_grouped_min_m(L)) {
    return 5;                                          // grouped scales, odd index widths: weights in tensor memory
  } else if (M >= grouped_min_m(L)) {
    if (large_m_grouped_cedes(L, M, false)) return 5;
    if (large_m_grouped_supported(L)) return 3;        // ... K split over clusters
  }
  return small_m_supported(L) ? 1 : SACQ_ERR_UNSUPPORTED;
}

}  // namespace
}  // namespace sacq

using namespace sacq;

extern "C" {

SACQ_API int sacq_abi_version(void) { return SACQ_ABI_VERSION; }
SACQ_API const char* sacq_last_error(void) { return g_error; }
SACQ_API int64_t sacq_launch_count(void) { return (int64_t)g_launches.load(std::memory_order_relaxed); }
SACQ_API int64_t sacq_workspace_counter_bytes(void) { return kCounterBytes; }

SACQ_API int sacq_layer_create(const sacq_layer_desc* desc, sacq_layer_t** out_layer) {
  if (desc == nullptr || out_layer == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  *out_layer = nullptr;
  if (desc->struct_size != sizeof(sacq_layer_desc))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "sacq_layer_desc.struct_size is %u, this library expects %zu",
                     desc->struct_size, sizeof(sacq_layer_desc));
  const sacq_layer_desc& d = *desc;
  if (d.out_features < 0 || d.in_features <= 0 || d.vector_dim <= 0 || d.group_size <= 0 || d.codebook_size <= 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "non-positive geometry (N=%lld K=%lld d=%d G=%d C=%d)",
                     (long long)d.out_features, (long long)d.in_features, d.vector_dim, d.group_size,
                     d.codebook_size);
  if (d.in_features % d.group_size != 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "in_features=%lld is not a multiple of group_size=%d",
                     (long long)d.in_features, d.group_size);
  if (d.group_size % d.vector_dim != 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "group_size=%d is not a multiple of vector_dim=%d", d.group_size,
                     d.vector_dim);
  if (d.index_bits < 1 || d.index_bits > 24)
    return set_error(SACQ_ERR_UNSUPPORTED, "index_bits=%d outside [1, 24]", d.index_bits);
  if (d.index_bits < 31 && (int64_t)d.codebook_size > (1LL << d.index_bits))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "codebook_size=%d does not fit index_bits=%d", d.codebook_size,
                     d.index_bits);
  if (d.in_features > (1 << 24) || d.out_features > (1 << 24))
    return set_error(SACQ_ERR_UNSUPPORTED, "features above 2^24 are not supported");
  const int64_t vpr = d.in_features / d.vector_dim;
  const int64_t expect = (d.out_features * vpr * d.index_bits + 7) / 8;
  if (d.packed_bytes != expect)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "packed stream has %lld bytes, expected %lld",
                     (long long)d.packed_bytes, (long long)expect);
  if (d.codebook == nullptr || d.scales == nullptr || (d.packed == nullptr && expect > 0))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null device pointer in layer description");
  if (reinterpret_cast<uintptr_t>(d.packed) % 16 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "packed stream must be 16-byte aligned");
  if (reinterpret_cast<uintptr_t>(d.codebook) % 16 != 0 || reinterpret_cast<uintptr_t>(d.scales) % 2 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "codebook must be 16-byte aligned");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0)
    return set_error(SACQ_ERR_CUDA, "no CUDA device is available; this library has no CPU path");
  if (d.device < 0 || d.device >= ndev)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "device %d out of range (%d devices)", d.device, ndev);

  DeviceGuard guard(d.device);
  if (!guard.ok) return set_error(SACQ_ERR_CUDA, "cannot make device %d current", d.device);
  sacq_layer* L = new (std::nothrow) sacq_layer();
  if (L == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "out of host memory");
  memset(L, 0, sizeof(*L));
  L->d = d;
  L->vectors_per_row = vpr;
  L->num_groups = d.in_features / d.group_size;
  L->row_bits = vpr * d.index_bits;
  L->rows_16b_aligned = (L->row_bits % 128) == 0;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, d.device) != cudaSuccess) {
    delete L;
    return set_error(SACQ_ERR_CUDA, "cudaGetDeviceProperties failed");
  }
  if (prop.major != 10) {
    delete L;
    return set_error(SACQ_ERR_UNSUPPORTED, "device %d is sm_%d%d; this library is built for sm_100a only", d.device,
                     prop.major, prop.minor);
  }
  L->num_sms = prop.multiProcessorCount;
  L->cb_entries = (d.codebook_size + 1) & ~1;
  L->order_rows = d.out_features;
  split_k_init(L);
  L->small_m_warps = small_m_staged_warps(L, 1);
  const int64_t count = (int64_t)L->cb_entries * d.vector_dim;
  // one allocation for all that is derived from the layer (each of its own costs a layer's making milliseconds)
  auto up = [](int64_t v) { return (v + 255) & ~(int64_t)255; };
  const int64_t hilo_at = up(count * 2), mul_at = hilo_at + up(count * 2), status_at = mul_at + up(d.out_features * 4);
  cudaError_t e = cudaMalloc(&L->derived, (size_t)(status_at + 256));
  if (e == cudaSuccess) {
    L->cb_f16 = reinterpret_cast<__half*>(L->derived);
    L->cb_hilo = L->derived + hilo_at;
    L->row_mul = reinterpret_cast<float*>(L->derived + mul_at);
    L->d_status = reinterpret_cast<int*>(L->derived + status_at);
    e = cudaMemset(L->d_status, 0, sizeof(int));
  }
  if (e != cudaSuccess) {
    sacq_layer_destroy(L);
    return cuda_fail(e, "allocating derived codebook tables");
  }
  L->resident_bytes = status_at + 256;
  const int rc = launch_build_tables(L, nullptr);
  if (rc != SACQ_OK) {
    sacq_layer_destroy(L);
    return rc;
  }
  *out_layer = L;
  return SACQ_OK;
}

SACQ_API int sacq_layer_destroy(sacq_layer_t* L) {
  if (L == nullptr) return SACQ_OK;
  DeviceGuard guard(L->d.device);
  large_m_release(L);
  split_k_release(L);
  if (L->derived) cudaFree(L->derived);
  delete L;
  return SACQ_OK;
}

SACQ_API int64_t sacq_layer_resident_bytes(const sacq_layer_t* L) { return L ? L->resident_bytes : 0; }

SACQ_API int sacq_dequant_bf16(const sacq_layer_t* L, void* w_out, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (w_out == nullptr && L->d.out_features > 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "w_out is null");
  DeviceGuard guard(L->d.device);
  return launch_dequant_bf16(L, w_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_weight_row_scale(const sacq_layer_t* L, float* sw_out, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (sw_out == nullptr && L->d.out_features > 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "sw_out is null");
  DeviceGuard guard(L->d.device);
  return launch_weight_row_scale(L, sw_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_decode_weight_fp8(const sacq_layer_t* L, const float* sw, void* wq_out, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if ((sw == nullptr || wq_out == nullptr) && L->d.out_features > 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  DeviceGuard guard(L->d.device);
  return launch_decode_weight_fp8(L, sw, wq_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_quant_act_fp8(const void* x_bf16, int64_t x_pitch, int64_t M, int64_t K, void* q_out, float* scale_out,
                       void* stream) {
  if (M < 0 || K < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "negative size (M=%lld K=%lld)", (long long)M,
                                       (long long)K);
  if (M == 0) return SACQ_OK;
  if (x_pitch < K) return set_error(SACQ_ERR_INVALID_ARGUMENT, "row pitch %lld smaller than K=%lld",
                                    (long long)x_pitch, (long long)K);
  if (scale_out == nullptr || ((x_bf16 == nullptr || q_out == nullptr) && K > 0))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (K == 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "K must be positive");
  return launch_quant_act(x_bf16, x_pitch, M, K, false, false, q_out, scale_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_act_quant_fp8(int kind, const void* a_bf16, int64_t a_pitch, const void* b_bf16, int64_t b_pitch,
                                int64_t M, int64_t K, void* q_out, float* scale_out, void* stream) {
  if (kind != SACQ_ACT_SILU_MUL && kind != SACQ_ACT_GELU)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "unknown activation kind %d", kind);
  if (M < 0 || K < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "negative size (M=%lld K=%lld)", (long long)M,
                                       (long long)K);
  if (M == 0) return SACQ_OK;
  if (K == 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "K must be positive");
  if (a_bf16 == nullptr || q_out == nullptr || scale_out == nullptr || (kind == SACQ_ACT_SILU_MUL && b_bf16 == nullptr))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (a_pitch < K || (kind == SACQ_ACT_SILU_MUL && b_pitch < K))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "row pitch smaller than K=%lld", (long long)K);
  return launch_act_quant_fp8(kind, a_bf16, a_pitch, b_bf16, b_pitch, nullptr, M, K, q_out, scale_out,
                              static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_layernorm_quant_fp8(const void* x_bf16, int64_t x_pitch, const void* gamma_bf16, const void* beta_bf16,
                                      float eps, const void* mod_scale_bf16, const void* mod_shift_bf16, int64_t M,
                                      int64_t K, void* y_out_bf16, int64_t y_pitch, void* q_out, float* scale_out,
                                      void* stream) {
  if (M < 0 || K < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "negative size (M=%lld K=%lld)", (long long)M,
                                       (long long)K);
  if (M == 0) return SACQ_OK;
  if (K == 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "K must be positive");
  if (x_bf16 == nullptr || q_out == nullptr || scale_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if ((mod_scale_bf16 == nullptr) != (mod_shift_bf16 == nullptr))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "modulation needs both its scale and its shift vector");
  if (x_pitch < K || (y_out_bf16 != nullptr && y_pitch < K))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "row pitch smaller than K=%lld", (long long)K);
  if (!(eps >= 0.f)) return set_error(SACQ_ERR_INVALID_ARGUMENT, "eps must be non-negative");
  return launch_layernorm_quant_fp8(x_bf16, x_pitch, gamma_bf16, beta_bf16, eps, mod_scale_bf16, mod_shift_bf16, M, K,
                                    y_out_bf16, y_pitch, q_out, scale_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_modulate_quant_fp8(const void* x_bf16, int64_t x_pitch, const void* scale_vec_bf16,
                                     const void* shift_vec_bf16, int64_t M, int64_t K, void* q_out, float* scale_out,
                                     void* stream) {
  if (M < 0 || K < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "negative size (M=%lld K=%lld)", (long long)M,
                                       (long long)K);
  if (M == 0) return SACQ_OK;
  if (K == 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "K must be positive");
  if (x_bf16 == nullptr || scale_vec_bf16 == nullptr || shift_vec_bf16 == nullptr || q_out == nullptr ||
      scale_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (x_pitch < K) return set_error(SACQ_ERR_INVALID_ARGUMENT, "row pitch smaller than K=%lld", (long long)K);
  return launch_act_quant_fp8(2, x_bf16, x_pitch, scale_vec_bf16, 0, shift_vec_bf16, M, K, q_out, scale_out,
                              static_cast<cudaStream_t>(stream));
}

SACQ_API int sacq_layer_set_kernel(sacq_layer_t* L, int which) {
  if (int rc = check_layer(L)) return rc;
  if (which < 0 || which > 15) return set_error(SACQ_ERR_INVALID_ARGUMENT, "kernel selector %d not in 0..15", which);
  L->force_kernel = which;
  return SACQ_OK;
}

SACQ_API int sacq_layer_set_shard_of(sacq_layer_t* L, int64_t rows) {
  if (int rc = check_layer(L)) return rc;
  if (rows < L->d.out_features || rows > (1 << 24))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "a shard of %lld rows of a layer of %lld", (long long)L->d.out_features, (long long)rows);
  L->order_rows = rows;
  L->small_m_warps = small_m_staged_warps(L, 1);
  return SACQ_OK;
}

SACQ_API int sacq_layer_kernel_for(const sacq_layer_t* L, int64_t M) {
  if (int rc = check_layer(L)) return rc;
  const int k = pick_kernel(L, M);
  if (k < 0) return set_error(k, "no kernel can run this layer geometry");
  return k;
}

SACQ_API int64_t sacq_workspace_bytes(const sacq_layer_t* L, int64_t M) {
  if (L == nullptr || M < 0) return 0;
  const int k = pick_kernel(L, M);
  if (k == 3) return kCounterBytes + large_m_grouped_workspace_bytes(L, M);
  if (k == 5) return kCounterBytes + large_m_tmem_grouped_workspace_bytes(L, M);
  const int64_t slab = small_m_slab_rows(L);
  return small_m_workspace_bytes(L, M < slab ? M : slab);
}

namespace {
// Common body of sacq_linear_a8 and sacq_linear_a8_residual.
// form: what q holds (fp16 only where the chosen kernel takes it, see sacq_forward_call).
int linear_a8_impl(const sacq_layer_t* L, const void* q, const float* scale, int64_t M, const void* residual,
                   int64_t ldr, void* y_out, int64_t ldy, void* workspace, int64_t workspace_bytes, void* stream,
                   const BcastDst* bc = nullptr, ActForm form = kActE4M3, const SplitChoice* cut = nullptr) {
  if (int rc = check_layer(L)) return rc;
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0 || L->d.out_features == 0) return SACQ_OK;
  if (q == nullptr || scale == nullptr || y_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (ldy < L->d.out_features)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldy=%lld smaller than out_features=%lld", (long long)ldy,
                     (long long)L->d.out_features);
  if (residual != nullptr && ldr < L->d.out_features)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldr=%lld smaller than out_features=%lld", (long long)ldr,
                     (long long)L->d.out_features);
  DeviceGuard guard(L->d.device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int k = pick_kernel(L, M);
  if (k < 0) return set_error(k, "no kernel can run this layer geometry");
  if (k == 2) return launch_large_m(L, q, scale, M, y_out, ldy, s, residual, ldr, bc, cut);
  if (k == 4)
    return launch_large_m_tmem(L, q, scale, M, y_out, ldy, s, residual, ldr, bc,
                               L->force_kernel >= 9 ? L->force_kernel - 8 : 0);
  if (k == 3 || k == 5) {
    if (workspace == nullptr || workspace_bytes < kCounterBytes)
      return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed, %lld given",
                       (long long)sacq_workspace_bytes(L, M), (long long)workspace_bytes);
    if (k == 5)
      return launch_large_m_tmem_grouped(L, q, scale, M, y_out, ldy, static_cast<uint8_t*>(workspace) + kCounterBytes,
                                         workspace_bytes - kCounterBytes, s, residual, ldr, form, bc,
                                         L->force_kernel >= 13 ? L->force_kernel - 12 : 0);
    return launch_large_m_grouped(L, q, scale, M, y_out, ldy, static_cast<uint8_t*>(workspace) + kCounterBytes,
                                  workspace_bytes - kCounterBytes, s, residual, ldr, form, large_m_grouped_exact(L, M, false), bc, cut);
  }
  const int64_t slab = small_m_slab_rows(L);
  for (int64_t m0 = 0; m0 < M; m0 += slab) {
    const int64_t rows = (M - m0) < slab ? (M - m0) : slab;
    BcastDst slab_bc{};
    if (bc != nullptr) {
      slab_bc.n = bc->n;
      for (int i = 0; i < bc->n; ++i) slab_bc.ptr[i] = static_cast<uint16_t*>(bc->ptr[i]) + m0 * ldy;
    }
    const int rc = launch_small_m(L, static_cast<const uint8_t*>(q) + m0 * L->d.in_features, scale + m0, rows,
                                  static_cast<uint16_t*>(y_out) + m0 * ldy, ldy, workspace, workspace_bytes, s,
                                  residual ? static_cast<const uint16_t*>(residual) + m0 * ldr : nullptr, ldr, 0,
                                  bc ? &slab_bc : nullptr);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}
}  // namespace

namespace {
// INT8 activations run on the kernels that take them widened to fp16: the tensor-core kernels of grouped scales,
// which run on any layer, or at small M the fp16 warp-MMA kernel where the layer's geometry allows it (8-, 12-
// and 16-bit indices) and it is the faster one (quantizer + GEMM: 2048x2048 8.1 / 12.0 us at 16 tokens and
// 13.9 / 12.7 at 40, 1536x1536 8.9 / 10.6 at 40), else the CUDA-core kernel.
enum Int8Route { kInt8Small, kInt8Grouped, kInt8TmemGrouped };
Int8Route int8_route(const sacq_layer* L, int64_t M) {
  if (is_shard(L)) {
    const sacq_layer whole = whole_layer(L);
    return int8_route(&whole, M);
  }
  if (large_m_tmem_grouped_supported(L) && M >= large_m_tmem_grouped_min_m(L)) return kInt8TmemGrouped;
  if (large_m_grouped_cedes(L, M, true)) return kInt8TmemGrouped;
  if (!large_m_grouped_supported(L)) return kInt8Small;
  const bool warp_mma = small_m_int8_selector(L) == 5 && (split_k_codebook_in_smem(L) || L->d.out_features < 4096);
  const int64_t warp_mma_wins = !warp_mma ? 0 : L->d.out_features < 2048 && split_k_codebook_in_smem(L) ? 48 : 16;
  return M > warp_mma_wins ? kInt8Grouped : kInt8Small;
}
}  // namespace

SACQ_API int sacq_quant_act_int8(const void* x_bf16, int64_t x_pitch, int64_t M, int64_t K, void* q_out, float* scale_out,
                                 void* stream) {
  if (M < 0 || K < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "negative size (M=%lld K=%lld)", (long long)M,
                                       (long long)K);
  if (M == 0) return SACQ_OK;
  if (x_pitch < K) return set_error(SACQ_ERR_INVALID_ARGUMENT, "row pitch %lld smaller than K=%lld",
                                    (long long)x_pitch, (long long)K);
  if (scale_out == nullptr || ((x_bf16 == nullptr || q_out == nullptr) && K > 0))
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (K == 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "K must be positive");
  return launch_quant_act(x_bf16, x_pitch, M, K, true, false, q_out, scale_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int64_t sacq_workspace_bytes_int8(const sacq_layer_t* L, int64_t M) {
  if (L == nullptr || M < 0) return 0;
  const Int8Route r = int8_route(L, M);
  if (r == kInt8TmemGrouped) return kCounterBytes + large_m_tmem_grouped_workspace_bytes(L, M);
  if (r == kInt8Grouped) return kCounterBytes + large_m_grouped_workspace_bytes(L, M);
  sacq_layer view = *L;
  view.force_kernel = small_m_int8_selector(L);
  const int64_t slab = small_m_slab_rows(L);
  return small_m_workspace_bytes(&view, M < slab ? M : slab);
}

namespace {
int linear_a8i_impl(const sacq_layer_t* L, const void* q, const float* scale, int64_t M, void* y_out, int64_t ldy,
                    void* workspace, int64_t workspace_bytes, void* stream, ActForm form, const SplitChoice* cut = nullptr) {
  DeviceGuard guard(L->d.device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Int8Route r = int8_route(L, M);
  if (r != kInt8Small) {
    if (workspace == nullptr || workspace_bytes < kCounterBytes)
      return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed, %lld given",
                       (long long)sacq_workspace_bytes_int8(L, M), (long long)workspace_bytes);
    return (r == kInt8TmemGrouped)
               ? launch_large_m_tmem_grouped(L, q, scale, M, y_out, ldy, static_cast<uint8_t*>(workspace) + kCounterBytes,
                                             workspace_bytes - kCounterBytes, s, nullptr, 0, form)
               : launch_large_m_grouped(L, q, scale, M, y_out, ldy, static_cast<uint8_t*>(workspace) + kCounterBytes,
                                        workspace_bytes - kCounterBytes, s, nullptr, 0, form, large_m_grouped_exact(L, M, true), nullptr, cut);
  }
  if (!small_m_supported(L)) return set_error(SACQ_ERR_UNSUPPORTED, "no kernel can run this layer geometry");
  sacq_layer view = *L;
  view.force_kernel = small_m_int8_selector(L);
  const int64_t slab = small_m_slab_rows(L);
  for (int64_t m0 = 0; m0 < M; m0 += slab) {
    const int64_t rows = (M - m0) < slab ? (M - m0) : slab;
    const int rc = launch_small_m(&view, static_cast<const uint8_t*>(q) + m0 * L->d.in_features, scale + m0, rows,
                                  static_cast<uint16_t*>(y_out) + m0 * ldy, ldy, workspace, workspace_bytes, s, nullptr,
                                  0, 1);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}
}  // namespace

SACQ_API int sacq_linear_a8i(const sacq_layer_t* L, const void* q_int8, const float* scale, int64_t M, void* y_out,
                             int64_t ldy, void* workspace, int64_t workspace_bytes, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0 || L->d.out_features == 0) return SACQ_OK;
  if (q_int8 == nullptr || scale == nullptr || y_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (ldy < L->d.out_features)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldy=%lld smaller than out_features=%lld", (long long)ldy,
                     (long long)L->d.out_features);
  return linear_a8i_impl(L, q_int8, scale, M, y_out, ldy, workspace, workspace_bytes, stream, kActInt8);
}

SACQ_API int sacq_weight_row_scale_int8(const sacq_layer_t* L, float* sw_out, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (sw_out == nullptr && L->d.out_features > 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "sw_out is null");
  DeviceGuard guard(L->d.device);
  return launch_weight_row_scale(L, sw_out, static_cast<cudaStream_t>(stream), 127.0f);
}

SACQ_API int sacq_decode_weight_int8(const sacq_layer_t* L, const float* sw, void* wq_out, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if ((sw == nullptr || wq_out == nullptr) && L->d.out_features > 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  DeviceGuard guard(L->d.device);
  return launch_decode_weight_int8(L, sw, wq_out, static_cast<cudaStream_t>(stream));
}

SACQ_API int64_t sacq_workspace_bytes_w8a8(const sacq_layer_t* L, int64_t M) {
  if (L == nullptr || M < 0) return 0;
  // the leading counter region of every workspace stays untouched (and zero) for the kernels that use it
  return kCounterBytes + ((L->d.out_features * L->d.in_features + 255) & ~(int64_t)255);
}

namespace {
// Few tokens run as one kernel, whose expanders make the weight bytes on the way to the tensor cores; for more, making
// them once for all tiles and a dense GEMM is faster, except where the layer's own row tiles fill the chip and one token
// tile holds the call (quantizer included, 6144 -> 2048: 14.3 / 23.0 us at 16 tokens, 21.9 / 20.8 at 200; 2048 -> 6144:
// 16.7 / 17.0 at 200, 17.6 / 19.7 at 300, 27.7 / 21.1 at 400; with a codebook of 65,536 entries 20.2 / 20.1 at 200).
bool recipe_in_one(const sacq_layer* L, const void* q, const float* act_scale, const float* w_scale, int64_t M, void* y,
                   int64_t ldy, SplitMode mode, cudaStream_t s, int* rc) {
  SplitChoice c;
  const bool wide = L->order_rows >= 4096 && L->d.in_features >= 2048;
  if (M > (!wide ? 32 : split_k_codebook_in_smem(L) ? 320 : 200) || reinterpret_cast<uintptr_t>(q) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(L->d.codebook) % 16 != 0 ||
      (mode == kSplitInt8 && L->d.in_features * 127 * 127 > 2147483647LL) || !split_k_tiles_fit(L, M, mode) ||
      !split_k_choose(L, M, mode, &c))
    return false;
  *rc = launch_split_k(&L, 1, q, act_scale, M, &y, &ldy, mode, c, s, nullptr, 0, nullptr, w_scale);
  return true;
}
}  // namespace

SACQ_API int sacq_linear_w8a8_int8(const sacq_layer_t* L, const void* q_int8, const float* act_scale, const float* w_scale,
                                   int64_t M, void* y_out, int64_t ldy, void* workspace, int64_t workspace_bytes,
                                   void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0 || L->d.out_features == 0) return SACQ_OK;
  if (q_int8 == nullptr || act_scale == nullptr || w_scale == nullptr || y_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (ldy < L->d.out_features)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldy=%lld smaller than out_features=%lld", (long long)ldy,
                     (long long)L->d.out_features);
  if (!dense_i8_supported(L))
    return set_error(SACQ_ERR_UNSUPPORTED, "INT8 recipe needs in_features to be a multiple of 16");
  const int64_t need = sacq_workspace_bytes_w8a8(L, M);
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed, %lld given", (long long)need,
                     (long long)workspace_bytes);
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  DeviceGuard guard(L->d.device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // per call, as the reference does: packed stream -> int8 weight rows, then the dense integer GEMM
  int rc = SACQ_OK;
  if (recipe_in_one(L, q_int8, act_scale, w_scale, M, y_out, ldy, kSplitInt8, s, &rc)) return rc;
  void* wq = static_cast<uint8_t*>(workspace) + kCounterBytes;
  if ((rc = launch_decode_weight_int8(L, w_scale, wq, s)) != SACQ_OK) return rc;
  return launch_dense_i8(L, q_int8, act_scale, wq, w_scale, M, y_out, ldy, s);
}

SACQ_API int sacq_linear_w8a8_fp8(const sacq_layer_t* L, const void* q_e4m3, const float* act_scale, const float* w_scale,
                                  int64_t M, void* y_out, int64_t ldy, void* workspace, int64_t workspace_bytes,
                                  void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0 || L->d.out_features == 0) return SACQ_OK;
  if (q_e4m3 == nullptr || act_scale == nullptr || w_scale == nullptr || y_out == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  if (ldy < L->d.out_features)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldy=%lld smaller than out_features=%lld", (long long)ldy,
                     (long long)L->d.out_features);
  if (!dense_i8_supported(L))
    return set_error(SACQ_ERR_UNSUPPORTED, "FP8 recipe needs in_features to be a multiple of 16");
  const int64_t need = sacq_workspace_bytes_w8a8(L, M);
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed, %lld given", (long long)need,
                     (long long)workspace_bytes);
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  DeviceGuard guard(L->d.device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // per call, as the reference does: packed stream -> e4m3 weight rows, then the dense FP8 GEMM
  int rc = SACQ_OK;
  if (recipe_in_one(L, q_e4m3, act_scale, w_scale, M, y_out, ldy, kSplitFp8, s, &rc)) return rc;
  void* wq = static_cast<uint8_t*>(workspace) + kCounterBytes;
  if ((rc = launch_decode_weight_fp8(L, w_scale, wq, s)) != SACQ_OK) return rc;
  return launch_dense_i8(L, q_e4m3, act_scale, wq, w_scale, M, y_out, ldy, s, true);
}

SACQ_API int sacq_linear_a8(const sacq_layer_t* L, const void* q, const float* scale, int64_t M, void* y_out, int64_t ldy,
                   void* workspace, int64_t workspace_bytes, void* stream) {
  return linear_a8_impl(L, q, scale, M, nullptr, 0, y_out, ldy, workspace, workspace_bytes, stream);
}

SACQ_API int sacq_linear_a8_bcast(const sacq_layer_t* L, const void* q, const float* scale, int64_t M, void* y_out,
                                  void* const* peer_outs, int num_peers, int64_t ldy, void* workspace,
                                  int64_t workspace_bytes, void* stream) {
  if (num_peers < 0 || num_peers > kMaxBcast)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "num_peers=%d outside [0, %d]", num_peers, kMaxBcast);
  if (num_peers > 0 && peer_outs == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "peer_outs is null");
  BcastDst bc{};
  bc.n = num_peers;
  for (int i = 0; i < num_peers; ++i) {
    if (peer_outs[i] == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "peer output %d is null", i);
    bc.ptr[i] = peer_outs[i];
  }
  return linear_a8_impl(L, q, scale, M, nullptr, 0, y_out, ldy, workspace, workspace_bytes, stream, &bc);
}

// ---- buffers that other processes of the node can map (CUDA IPC) -------------------------
SACQ_API int sacq_peer_buffer_create(int device, int64_t bytes, void** dev_ptr, void* handle_out) {
  if (dev_ptr == nullptr || handle_out == nullptr || bytes <= 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument or non-positive size");
  DeviceGuard guard(device);
  if (!guard.ok) return set_error(SACQ_ERR_CUDA, "cannot make device %d current", device);
  void* p = nullptr;
  SACQ_CUDA_TRY(cudaMalloc(&p, (size_t)bytes));
  cudaIpcMemHandle_t h;
  const cudaError_t e = cudaIpcGetMemHandle(&h, p);
  if (e != cudaSuccess) {
    cudaFree(p);
    return cuda_fail(e, "cudaIpcGetMemHandle");
  }
  static_assert(sizeof(cudaIpcMemHandle_t) == SACQ_PEER_HANDLE_BYTES, "handle size");
  memcpy(handle_out, &h, sizeof(h));
  *dev_ptr = p;
  return SACQ_OK;
}

SACQ_API int sacq_peer_buffer_open(int device, const void* handle, void** dev_ptr) {
  if (dev_ptr == nullptr || handle == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  DeviceGuard guard(device);
  if (!guard.ok) return set_error(SACQ_ERR_CUDA, "cannot make device %d current", device);
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, sizeof(h));
  SACQ_CUDA_TRY(cudaIpcOpenMemHandle(dev_ptr, h, cudaIpcMemLazyEnablePeerAccess));
  return SACQ_OK;
}

SACQ_API int sacq_peer_buffer_close(int device, void* dev_ptr) {
  if (dev_ptr == nullptr) return SACQ_OK;
  DeviceGuard guard(device);
  SACQ_CUDA_TRY(cudaIpcCloseMemHandle(dev_ptr));
  return SACQ_OK;
}

SACQ_API int sacq_peer_buffer_destroy(int device, void* dev_ptr) {
  if (dev_ptr == nullptr) return SACQ_OK;
  DeviceGuard guard(device);
  SACQ_CUDA_TRY(cudaFree(dev_ptr));
  return SACQ_OK;
}

SACQ_API int sacq_linear_a8_residual(const sacq_layer_t* L, const void* q, const float* scale, int64_t M,
                                     const void* residual, int64_t ldr, void* y_out, int64_t ldy, void* workspace,
                                     int64_t workspace_bytes, void* stream) {
  if (residual == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "residual is null");
  return linear_a8_impl(L, q, scale, M, residual, ldr, y_out, ldy, workspace, workspace_bytes, stream);
}

SACQ_API int sacq_linear_a8_multi(const sacq_layer_t* const* layers, int num_layers, const void* q, const float* scale,
                                  int64_t M, void* const* y_outs, const int64_t* ldys, void* workspace,
                                  int64_t workspace_bytes, void* stream) {
  if (layers == nullptr || y_outs == nullptr || ldys == nullptr || num_layers <= 0)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument or no layers");
  for (int l = 0; l < num_layers; ++l) {
    if (int rc = check_layer(layers[l])) return rc;
    if (layers[l]->d.in_features != layers[0]->d.in_features)
      return set_error(SACQ_ERR_INVALID_ARGUMENT, "layers that share an input must have the same in_features");
    if (layers[l]->d.device != layers[0]->d.device)
      return set_error(SACQ_ERR_INVALID_ARGUMENT, "layers that share an input must be on one device");
    if (y_outs[l] == nullptr && layers[l]->d.out_features > 0 && M > 0)
      return set_error(SACQ_ERR_INVALID_ARGUMENT, "null output for layer %d", l);
    if (ldys[l] < layers[l]->d.out_features)
      return set_error(SACQ_ERR_INVALID_ARGUMENT, "ldy=%lld smaller than out_features=%lld", (long long)ldys[l],
                       (long long)layers[l]->d.out_features);
  }
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0) return SACQ_OK;
  if (q == nullptr || scale == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  {
    // one launch when every layer would use the staged small-M kernel on a common geometry
    bool small = num_layers >= 2;
    for (int l = 0; l < num_layers && small; ++l) small = pick_kernel(layers[l], M) == 1;
    if (small) {
      DeviceGuard guard(layers[0]->d.device);
      const int rc = launch_small_m_multi(layers, num_layers, q, scale, M, y_outs, ldys,
                                          static_cast<cudaStream_t>(stream));
      if (rc != SACQ_ERR_UNSUPPORTED) return rc;
    }
    // ... or the FP8 tensor-core kernel (blockIdx.z = layer)
    bool large = num_layers >= 2;
    for (int l = 0; l < num_layers && large; ++l) large = pick_kernel(layers[l], M) == 2;
    if (large) {
      DeviceGuard guard(layers[0]->d.device);
      const int rc = launch_large_m_multi(layers, num_layers, q, scale, M, y_outs, ldys,
                                          static_cast<cudaStream_t>(stream));
      if (rc != SACQ_ERR_UNSUPPORTED) return rc;
    }
    // ... or its fp16 form for grouped scales
    bool grouped = num_layers >= 2 && workspace != nullptr && workspace_bytes > kCounterBytes;
    for (int l = 0; l < num_layers && grouped; ++l) grouped = pick_kernel(layers[l], M) == 3;
    if (grouped) {
      DeviceGuard guard(layers[0]->d.device);
      const int rc = launch_large_m_grouped_multi(layers, num_layers, q, scale, M, y_outs, ldys,
                                                  static_cast<uint8_t*>(workspace) + kCounterBytes,
                                                  workspace_bytes - kCounterBytes, static_cast<cudaStream_t>(stream));
      if (rc != SACQ_ERR_UNSUPPORTED) return rc;
    }
  }
  for (int l = 0; l < num_layers; ++l) {
    const int rc = sacq_linear_a8(layers[l], q, scale, M, y_outs[l], ldys[l], workspace, workspace_bytes, stream);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}

namespace {
// Whether a forward on a staged warp-MMA kernel quantizes its activations in the GEMM's own CTAs.  It saves a launch, which
// costs the host 2 us of the 7 that an eager call of these sizes takes, and costs the GPU 0.3 to 1.3 us: each CTA's own
// pass over the tokens (2048x2048, d = 4, 16 tokens 6.5 us against 5.4; 2048x1024 at one 4.5 / 4.2).  A captured call
// pays for the GPU's time only and keeps the quantizer as a launch of its own; the bytes are the same.  On layers that
// keep the GPU busy anyway it is a loss in eager calls too (2048x6144 8.9 against 8.4 at one token, 6144x2048 10.7 / 8.4 at 8).
bool eager(cudaStream_t s) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &status) != cudaSuccess) {   // the default stream beside another thread's capture
    cudaGetLastError();
    return false;
  }
  return status == cudaStreamCaptureStatusNone;
}
bool quantizes_in_gemm(const sacq_layer* L, int64_t M, cudaStream_t s) {
  return L->d.in_features * L->d.out_features <= (4 << 20) && M * L->d.in_features <= (32 << 10) && M <= small_m_staged_warps(L, M) && eager(s);
}
// The same for the split-K kernel, whose expander warps quantize the tokens, a warp each, once their rows have landed in shared
// memory.  Its CTAs enter long before the wait for the kernel in front ends, if the last call's leave them SMs: then the GPU loses
// little or nothing (graph / eager, quantizer by itself against this: 1024 -> 4096 5.2 / 8.3 against 5.0 / 5.5 us at 8 tokens,
// 5.5 / 8.1 against 6.1 / 6.6 at 24; codebook in L2, 2048 -> 2048 at 4 6.5 / 8.3 against 5.9 / 6.2).  CTAs that wait for SMs have
// it ahead of them on top of their expansions: up to 16 tokens as long as a launch takes the host (2048 -> 6144 at 4
// 7.0 / 8.2 against 7.5 / 7.8, 16 7.1 / 8.2 against 7.9 / 8.3; in L2 11.3 / 11.5 against 10.8 / 10.8), not beyond (24, 256 codewords,
// 7.1 / 8.2 against 8.8 / 9.1).  Every CTA reads the whole rows of its tokens: not 32 of 2,048 (256 codewords, 2048 -> 1024 at 64
// 6.5 / 7.7 against 8.0 / 8.3; 16 to a tile at 40 6.5 / 7.7 against 6.5 / 6.9).
bool quantizes_in_split(const sacq_layer* L, int64_t M, cudaStream_t s, const SplitChoice& c) {
  if (M > 64 || c.tok * L->d.in_features > (48 << 10) || !split_k_quantizes(L, c)) return false;
  const bool early = 2 * split_k_ctas(L, c) <= L->num_sms, few = M <= 16;
  return (few && (early || !split_k_codebook_in_smem(L))) || ((few || early) && eager(s));
}

// Quantizer + GEMM of one call, in one launch where the GEMM can quantize for itself (own_quantizer = false allows it).
// Where the GEMM takes fp16 activations, the quantizer writes them as fp16 into the workspace: one launch less than
// quantizing to bytes and widening those (2 us of host time and as much of the GPU's at small sizes), the same values.
int forward_impl(const sacq_layer_t* L, const void* x_bf16, int64_t x_pitch, int64_t M, int int8, const void* residual,
                 int64_t ldr, void* q_scratch, float* scale_scratch, void* y_out, int64_t ldy, void* workspace,
                 int64_t workspace_bytes, void* stream, bool own_quantizer) {
  if (int rc = check_layer(L)) return rc;
  if (M == 0) return SACQ_OK;
  const int64_t K = L->d.in_features;
  Beside beside = kBesideNone;                        // the quantizer runs beside the split-K kernel
  SplitChoice c;                                      // how that kernel's call is cut up: searched once (0.2 to 0.4 us)
  const SplitChoice* cut = nullptr;
  int64_t slab = 0;                                   // tokens up to which the GEMM takes fp16 activations in one piece
  int64_t need = 0;
  const bool rows_ok = M > 0 && L->d.out_features > 0 && K % 8 == 0 && x_bf16 != nullptr &&
                       reinterpret_cast<uintptr_t>(x_bf16) % 16 == 0 && x_pitch % 8 == 0 && x_pitch >= K && y_out != nullptr &&
                       ldy >= L->d.out_features;
  if (rows_ok) {
    const Int8Route r = int8 ? int8_route(L, M) : kInt8Small;
    const int k = int8 ? 0 : pick_kernel(L, M);
    if (k == 1 && !own_quantizer && quantizes_in_gemm(L, M, static_cast<cudaStream_t>(stream))) {
      DeviceGuard guard(L->d.device);
      return launch_small_m(L, q_scratch, scale_scratch, M, y_out, ldy, workspace, workspace_bytes,
                            static_cast<cudaStream_t>(stream), residual, ldr, 0, nullptr, x_bf16, x_pitch);
    }
    if (k == 2 || k == 3 || r == kInt8Grouped) {
      const SplitMode mode = k == 2 ? kSplitHiLo : large_m_grouped_exact(L, M, int8 != 0) ? kSplitHalf2 : kSplitHalf;
      if (M <= 1024 && split_k_choose(L, M, mode, &c)) {
        cut = &c;
        if (k == 2 && !own_quantizer && (residual == nullptr || ldr >= L->d.out_features) &&
            quantizes_in_split(L, M, static_cast<cudaStream_t>(stream), c)) {
          DeviceGuard guard(L->d.device);
          return launch_split_k(&L, 1, nullptr, nullptr, M, &y_out, &ldy, kSplitHiLo, c, static_cast<cudaStream_t>(stream), residual, ldr,
                                nullptr, nullptr, x_bf16, x_pitch);
        }
        // a projection with a residual follows attention, not a GEMM: nothing to share an SM with (prefill block at 300 tokens 90.7 / 91.2 us)
        if (residual == nullptr) beside = split_k_beside(L, M, c);
      }
    }
    if (r == kInt8TmemGrouped || k == 5) {
      slab = large_m_tmem_grouped_slab();
      need = large_m_tmem_grouped_workspace_bytes(L, M);
    } else if (r == kInt8Grouped || k == 3) {
      slab = large_m_grouped_slab();
      need = large_m_grouped_workspace_bytes(L, M);
    }
  }
  const bool wide = rows_ok && M <= slab && workspace != nullptr && scale_scratch != nullptr &&
                    reinterpret_cast<uintptr_t>(workspace) % 256 == 0 && workspace_bytes >= kCounterBytes + need;
  if (wide) {
    DeviceGuard guard(L->d.device);
    void* a16 = static_cast<uint8_t*>(workspace) + kCounterBytes;
    if (int rc = launch_quant_act(x_bf16, x_pitch, M, K, int8 != 0, true, a16, scale_scratch, static_cast<cudaStream_t>(stream), beside))
      return rc;
    if (int8) return linear_a8i_impl(L, a16, scale_scratch, M, y_out, ldy, workspace, workspace_bytes, stream, kActHalf, cut);
    return linear_a8_impl(L, a16, scale_scratch, M, residual, ldr, y_out, ldy, workspace, workspace_bytes, stream, nullptr,
                          kActHalf, cut);
  }
  const int rc = beside != kBesideNone && q_scratch != nullptr && scale_scratch != nullptr
                     ? launch_quant_act(x_bf16, x_pitch, M, K, int8 != 0, false, q_scratch, scale_scratch, static_cast<cudaStream_t>(stream), beside)
                 : int8 ? sacq_quant_act_int8(x_bf16, x_pitch, M, K, q_scratch, scale_scratch, stream)
                        : sacq_quant_act_fp8(x_bf16, x_pitch, M, K, q_scratch, scale_scratch, stream);
  if (rc != SACQ_OK) return rc;
  if (int8) return sacq_linear_a8i(L, q_scratch, scale_scratch, M, y_out, ldy, workspace, workspace_bytes, stream);
  return linear_a8_impl(L, q_scratch, scale_scratch, M, residual, ldr, y_out, ldy, workspace, workspace_bytes, stream, nullptr,
                        kActE4M3, cut);
}

// Whether the kernel of a call with M tokens may store its result straight into pinned host memory: one whose stores
// are whole segments of a token's row (the split-K kernel 256 bytes per warp, the staged warp-MMA kernels 16 to 96).
bool stores_reach_host(const sacq_layer* L, int64_t M) {
  const int k = pick_kernel(L, M);
  return k == 2 || k == 3 || (k == 1 && small_m_staged_warps(L, M) > 0);
}
}  // namespace

int sacq_forward_call(const sacq_layer_t* L, const void* x_bf16, int64_t x_pitch, int64_t M, int int8, const void* residual,
                      int64_t ldr, void* q_scratch, float* scale_scratch, void* y_out, int64_t ldy, void* workspace,
                      int64_t workspace_bytes, void* stream) {
  return forward_impl(L, x_bf16, x_pitch, M, int8, residual, ldr, q_scratch, scale_scratch, y_out, ldy, workspace,
                      workspace_bytes, stream, false);
}

SACQ_API int sacq_linear_bf16(const sacq_layer_t* L, const void* x_bf16, int64_t x_pitch, int64_t M, void* q_scratch,
                     float* scale_scratch, void* y_out, int64_t ldy, void* workspace, int64_t workspace_bytes,
                     void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (M == 0) return SACQ_OK;
  // the two calls it stands for: its caller finds the quantized activations in its scratch
  const int rc = sacq_quant_act_fp8(x_bf16, x_pitch, M, L->d.in_features, q_scratch, scale_scratch, stream);
  return rc != SACQ_OK ? rc
                       : linear_a8_impl(L, q_scratch, scale_scratch, M, nullptr, 0, y_out, ldy, workspace, workspace_bytes, stream);
}

// Layout of the device scratch of sacq_linear_bf16_host: workspace first (its counter
// region leads), then scale, x, q, y, each 256-byte aligned.
namespace {
struct HostForwardLayout {
  int64_t ws, scale, x, q, y, total;
};
HostForwardLayout host_forward_layout(const sacq_layer* L, int64_t M) {
  auto up = [](int64_t v) { return (v + 255) & ~(int64_t)255; };
  HostForwardLayout h;
  h.ws = 0;
  h.scale = up(sacq_workspace_bytes(L, M));
  h.x = h.scale + up(M * 4);
  h.q = h.x + up(M * L->d.in_features * 2);
  h.y = h.q + up(M * L->d.in_features);
  h.total = h.y + up(M * L->d.out_features * 2);
  return h;
}

// Transfers up to this size bypass the copy engine when the host buffer is pinned: the
// quantizer reads the activations straight from host memory and a copy kernel pushes the
// result back (each copy-engine hand-over on a stream costs more than the transfer itself).
constexpr int64_t kDirectHostIoBytes = 1 << 20;

// Device alias of a pinned (page-locked, mapped) host pointer, or null.
void* pinned_alias(const void* host) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}
}  // namespace

SACQ_API int64_t sacq_host_forward_scratch_bytes(const sacq_layer_t* L, int64_t M) {
  if (L == nullptr || M < 0) return 0;
  return host_forward_layout(L, M).total;
}

SACQ_API int sacq_linear_bf16_host(const sacq_layer_t* L, const void* x_host, int64_t M, void* y_host,
                                   void* dev_scratch, int64_t dev_scratch_bytes, void* stream) {
  if (int rc = check_layer(L)) return rc;
  if (M < 0) return set_error(SACQ_ERR_INVALID_ARGUMENT, "M=%lld is negative", (long long)M);
  if (M == 0 || L->d.out_features == 0) return SACQ_OK;
  if (x_host == nullptr || y_host == nullptr || dev_scratch == nullptr)
    return set_error(SACQ_ERR_INVALID_ARGUMENT, "null argument");
  const HostForwardLayout h = host_forward_layout(L, M);
  if (dev_scratch_bytes < h.total)
    return set_error(SACQ_ERR_WORKSPACE, "device scratch of %lld bytes needed, %lld given", (long long)h.total,
                     (long long)dev_scratch_bytes);
  if (reinterpret_cast<uintptr_t>(dev_scratch) % 256 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "device scratch must be 256-byte aligned");
  DeviceGuard guard(L->d.device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint8_t* base = static_cast<uint8_t*>(dev_scratch);
  const int64_t K = L->d.in_features, N = L->d.out_features;
  const void* x_dev = base + h.x;
  void* x_alias = M * K * 2 <= kDirectHostIoBytes && reinterpret_cast<uintptr_t>(x_host) % 16 == 0
                      ? pinned_alias(x_host) : nullptr;
  if (x_alias != nullptr)
    x_dev = x_alias;                                   // the quantizer reads the pinned buffer itself
  else
    SACQ_CUDA_TRY(cudaMemcpyAsync(base + h.x, x_host, (size_t)(M * K * 2), cudaMemcpyHostToDevice, s));
  void* y_alias = M * N * 2 <= kDirectHostIoBytes && reinterpret_cast<uintptr_t>(y_host) % 16 == 0
                      ? pinned_alias(y_host) : nullptr;
  // rows of whole 128-byte lines: the GEMM stores them to the host itself (another kernel that copies them out costs
  // the call 3 us; rows that share lines would cross the bus in pieces)
  const bool stores_out = y_alias != nullptr && N % 64 == 0 && reinterpret_cast<uintptr_t>(y_host) % 128 == 0 &&
                          stores_reach_host(L, M);
  // the quantizer keeps its own launch: it reads the host's rows once, not once per CTA of the GEMM
  const int rc = forward_impl(L, x_dev, K, M, 0, nullptr, 0, base + h.q, reinterpret_cast<float*>(base + h.scale),
                              stores_out ? y_alias : base + h.y, N, base + h.ws, h.scale, stream, true);
  if (rc != SACQ_OK || stores_out) return rc;
  if (y_alias != nullptr) return launch_copy_to_host(base + h.y, y_alias, M * N * 2, L->num_sms, s);
  SACQ_CUDA_TRY(cudaMemcpyAsync(y_host, base + h.y, (size_t)(M * N * 2), cudaMemcpyDeviceToHost, s));
  return SACQ_OK;
}

SACQ_API int sacq_layer_status(const sacq_layer_t* L, int* status_out) {
  if (int rc = check_layer(L)) return rc;
  if (status_out == nullptr) return set_error(SACQ_ERR_INVALID_ARGUMENT, "status_out is null");
  DeviceGuard guard(L->d.device);
  SACQ_CUDA_TRY(cudaMemcpy(status_out, L->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  return SACQ_OK;
}

}  // extern "C"
