// Tensor-core path of per-channel layers from a few dozen tokens up to the batched sizes: argument checks
// and launch of the split-K kernel (linear_split_k.cu), the tensor-map helpers every tensor-core kernel
// uses, and a layer's index-tile map.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "split_k.cuh"
#include "tmem_weights.cuh"
#include "umma.cuh"

namespace sacq {

struct LargeMPlan {
  CUtensorMap tmap_idx;         // index super-blocks (two 128-k blocks) x 128 weight rows
  bool have;
};

namespace {

constexpr int kBK = 128;          // e4m3 elements (= bytes) per K block: one 128B swizzle row

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver entry point is resolved through the runtime so the library carries no
// link-time dependency on libcuda (it must load on a machine without a driver).
EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

}  // namespace

// 2-D byte tensor [rows][row_bytes] with a [box_rows][box_bytes] box.
int encode_bytes_2d(CUtensorMap* map, const void* base, uint64_t row_bytes, uint64_t rows, uint64_t pitch_bytes,
                    uint32_t box_bytes, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return set_error(SACQ_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {row_bytes, rows};
  const cuuint64_t strides[1] = {pitch_bytes};
  const cuuint32_t box[2] = {box_bytes, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_error(SACQ_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return SACQ_OK;
}

namespace {

int sb_bytes_for(const sacq_layer* L) { return 2 * (kBK / L->d.vector_dim) * L->d.index_bits / 8; }

std::mutex g_plan_mutex;   // layers build their index tile map on first use, possibly from several host threads

}  // namespace

bool large_m_supported(const sacq_layer* L) {
  const sacq_layer_desc& d = L->d;
  if (d.index_bits != 8 && d.index_bits != 12 && d.index_bits != 16) return false;
  return d.in_features % (2 * kBK) == 0 && L->split_tok[kSplitHiLo] > 0;
}

void large_m_release(sacq_layer* L) {
  delete L->large_plan;
  L->large_plan = nullptr;
}

int large_m_index_map(const sacq_layer* Lc, const CUtensorMap** out) {
  sacq_layer* L = const_cast<sacq_layer*>(Lc);
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  if (L->large_plan == nullptr) L->large_plan = new LargeMPlan();
  if (!L->large_plan->have) {
    const uint64_t row_bytes = (uint64_t)(L->row_bits / 8);
    const int rc = encode_bytes_2d(&L->large_plan->tmap_idx, L->d.packed, row_bytes, (uint64_t)L->d.out_features, row_bytes,
                                   (uint32_t)sb_bytes_for(L), 128u, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc != SACQ_OK) return rc;
    L->large_plan->have = true;
  }
  *out = &L->large_plan->tmap_idx;
  return SACQ_OK;
}

namespace {

// A tile's width for `t` tokens: a multiple of 32, of 64 above 256 (two instructions).
int width_of(int64_t t) {
  const int64_t step = t > 256 ? 64 : 32;
  return (int)((t + step - 1) / step * step);
}

// The tiles of M tokens in tiles of `tok` and one of what is left, and the modelled time of the busiest worker.  The
// remainders go to the workers that have a whole tile less than the others, or, where that makes too many for them, to all.
double plan_of(const sacq_layer* L, int64_t M, TileTime tile_us, int tok, tmemw::TilePlan* p) {
  p->row_tiles = (int)((L->d.out_features + tmemw::kRows - 1) / tmemw::kRows);
  p->tok = tok;
  p->full = (int)(M / tok) * p->row_tiles;
  p->rem = width_of(M % tok);
  p->rem_m0 = (int)(M / tok * tok);
  p->rem_first = 0;
  const int tiles = p->full + (p->rem > 0 ? p->row_tiles : 0);
  p->workers = tiles < L->num_sms ? tiles : L->num_sms;
  const int rounds = p->full / p->workers, extra = p->full % p->workers;
  const double whole = (rounds + (extra > 0 ? 1 : 0)) * tile_us(L, tok);
  if (p->rem == 0) return whole;
  auto rems = [&](int on) { return (p->row_tiles + on - 1) / on * tile_us(L, p->rem); };
  const double few = rounds * tile_us(L, tok) + rems(p->workers - extra);
  if (rounds == 0 && p->full > 0 && few >= whole + rems(extra)) {     // as many workers as whole tiles
    p->workers = p->full;
    return whole + rems(p->workers);
  }
  const double all = whole + rems(p->workers);
  if (rounds > 0 && few >= all) return all;
  p->rem_first = extra;
  return few > whole ? few : whole;
}

}  // namespace

// 8,192 tokens of a 6,144-row layer, for instance, are 1,008 tiles of 384 and 48 of 128 on 148 SMs: 7 rounds, where a grid
// of equal tiles takes 8.
bool plan_tiles(const sacq_layer* L, int64_t M, TileTime tile_us, int tok_force, tmemw::TilePlan* p, double* us) {
  if (M / 32 + 1 > 0x7fffffff / ((L->d.out_features + tmemw::kRows) / tmemw::kRows)) return false;
  double best_us = 1e30;
  for (int t = tmemw::kMaxTok; t >= 32; t -= t > 256 ? 64 : 32) {
    if (tok_force > 0 && t != tok_force) continue;
    tmemw::TilePlan c;
    const double t_us = plan_of(L, M, tile_us, t, &c);
    if (t_us < best_us - 1e-9) {
      best_us = t_us;
      *p = c;
    }
  }
  if (us != nullptr) *us = best_us;
  // one activation copy size for both kinds of tile
  auto part_of = [](int t) { return t / (t > 256 ? 2 : 1); };
  p->box = part_of(p->full > 0 ? p->tok : p->rem);
  for (int a = part_of(p->rem); p->full > 0 && a > 0;) {
    const int r = p->box % a;
    p->box = a;
    a = r;
  }
  return true;
}

int tile_output(const sacq_layer* L, int64_t M, void* y, int64_t ldy, const void* residual, int64_t ldr, const BcastDst* bc,
                tmemw::TmemOut* out, CUtensorMap* ty, tmemw::BcastMaps* tb) {
  const sacq_layer_desc& d = L->d;
  out->y = static_cast<uint16_t*>(y);
  out->ldy = ldy;
  out->residual = static_cast<const uint16_t*>(residual);
  out->ldr = ldr;
  out->M = (int)M;
  out->N = (int)d.out_features;
  bool tma = residual == nullptr && reinterpret_cast<uintptr_t>(y) % 16 == 0 && (ldy * 2) % 16 == 0 && d.out_features >= 32;
  for (int i = 0; bc != nullptr && i < bc->n; ++i) {
    out->ybc[i] = static_cast<uint16_t*>(bc->ptr[i]);
    tma = tma && reinterpret_cast<uintptr_t>(bc->ptr[i]) % 16 == 0;
  }
  out->n_bc = bc != nullptr ? bc->n : 0;
  out->y_tma = tma ? 1 : 0;
  for (int i = tma ? -1 : out->n_bc; i < out->n_bc; ++i) {
    const int rc = encode_bytes_2d(i < 0 ? ty : &tb->m[i], i < 0 ? y : bc->ptr[i], (uint64_t)d.out_features * 2, (uint64_t)M,
                                   (uint64_t)ldy * 2, 64, 32, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}

int launch_large_m(const sacq_layer* L, const void* q, const float* scale, int64_t M, void* y, int64_t ldy,
                   cudaStream_t s, const void* residual, int64_t ldr, const BcastDst* bc, const SplitChoice* cut) {
  if (!large_m_supported(L)) return set_error(SACQ_ERR_UNSUPPORTED, "large-M kernel cannot run this layer geometry");
  if (M <= 0 || L->d.out_features == 0) return SACQ_OK;
  if (M > (1 << 30)) return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld too large", (long long)M);
  for (int64_t m0 = 0; m0 < M; m0 += kSplitMaxM) {
    const int64_t rows = M - m0 < kSplitMaxM ? M - m0 : kSplitMaxM;
    SplitChoice c;
    if (cut != nullptr) c = *cut;
    else if (!split_k_choose(L, rows, kSplitHiLo, &c)) return set_error(SACQ_ERR_UNSUPPORTED, "split-K kernel: no tile fits");
    BcastDst slab{};
    for (int i = 0; bc != nullptr && i < bc->n; ++i) slab.ptr[slab.n++] = static_cast<uint16_t*>(bc->ptr[i]) + m0 * ldy;
    void* y_slab = static_cast<uint16_t*>(y) + m0 * ldy;
    const int rc = launch_split_k(&L, 1, static_cast<const uint8_t*>(q) + m0 * L->d.in_features, scale + m0, rows, &y_slab,
                                  &ldy, kSplitHiLo, c, s, residual ? static_cast<const uint16_t*>(residual) + m0 * ldr : nullptr,
                                  ldr, bc ? &slab : nullptr);
    if (rc != SACQ_OK) return rc;
  }
  return SACQ_OK;
}

// Several layers of one geometry on the same quantized activations as ONE launch.  Returns
// SACQ_ERR_UNSUPPORTED (nothing launched) when they cannot share one: the caller falls back
// to one launch per layer.  An output's summation order depends on K alone, so the results are
// byte-identical to separate launches.
int launch_large_m_multi(const sacq_layer* const* layers, int n, const void* q, const float* scale, int64_t M,
                         void* const* ys, const int64_t* ldys, cudaStream_t s) {
  if (n < 2 || n > kSplitMaxLayers || M <= 0) return SACQ_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(q) % 16 != 0) return SACQ_ERR_UNSUPPORTED;
  for (int l = 0; l < n; ++l)
    if (!large_m_supported(layers[l])) return SACQ_ERR_UNSUPPORTED;
  SplitChoice c;
  if (!split_k_choose_multi(layers, n, M, kSplitHiLo, &c)) return SACQ_ERR_UNSUPPORTED;
  return launch_split_k(layers, n, q, scale, M, ys, ldys, kSplitHiLo, c, s);
}

}  // namespace sacq
