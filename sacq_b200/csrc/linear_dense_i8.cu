// The reference's 8-bit weight recipes as dense 8-bit work on the 5th-generation tensor cores.
// INT8 (the deployed one; FP8 below):
// The reference's deployed INT8 recipe as integer work on the 5th-generation tensor cores
// (sm_100a): per-token int8 activations x per-output-row int8 weights -> int32, then
//   y[m,n] = bf16( fma(sa[m], float(acc[m,n]) * sw[n], bias[n]) )        (bias given)
//   y[m,n] = bf16( sa[m] * (float(acc[m,n]) * sw[n]) )                   (no bias)
// -- weight scale first, then token scale, the bias inside one fused multiply-add
// (int8_small_m_gemm_20261028_r1.py:7-32, int8_ordered_epilogue_20261028_r1.py:11-22).
// Integer accumulation is exact, so the output bytes are a function of the operands alone:
// this path can be, and is tested to be, bit-identical to a CPU restatement of the recipe.
//
// Like the reference (perrow_a8_candidate_r3.py:52-63: "no persistent decoded weight cache")
// the int8 weight matrix is produced per call from the packed stream into the caller's
// workspace (decode_rows_kernel, dequant.cu) and consumed by a plain dense GEMM.  A CTA
// computes a tile of SUBS x 128 tokens x BN weight rows (256 x 256, 256 x 128, 128 x 128 or 128 x 64):
//   warp 0            : TMA producer: per 128-byte K block the token sub-tiles and one tile of BN weight
//                       rows, SWIZZLE_128B, no multicast, in as many stages as fit 200 KB;
//   warp 1            : tcgen05.mma kind::i8, M128 x N(BN) x K32, into one int32 accumulator per token
//                       sub-tile; the sub-tiles share every weight tile;
//   8 SUBS more warps : epilogue: TMEM lane quarter x token sub-tile x column half each, through shared memory
//                       so that four lanes store a token's 64 bytes (16-byte pieces of 32 rows at a time left half of
//                       every sector: 5.7 us of a 256 x 256 tile, now 2.5).
// Rows that begin or end anywhere go out an element per lane, 64 contiguous bytes a store (2048 -> 6137, INT8, 1,500 tokens:
// 112 us with a row per lane, 31 now).
// A last token tile of at most 128 tokens loads and multiplies one sub-tile only.
// What bounds it: the 256 x 256 tile the tensor cores (0.48 us per K block, 1024 of 1090 clocks), the small ones the
// operands through L2 (about 19 TB/s over the chip).  1,024 tokens, 6144 -> 2048, FP8, weight bytes included: 45 us
// with 256 x 256 tiles (32 CTAs), 22 with 128 x 128 (128 CTAs); 8,192 tokens, 2048 -> 6144: 132 -> 115.
// Every mbarrier wait is bounded (status word + CTA-wide abort flag), as in the other
// tensor-core kernels.
//
// The FP8 recipe (`projection_format: fp8_e4m3fn`; a8_joint_pair_r1.py:374,
// perrow_a8_candidate_r3.py:56-69: per-token e4m3 activations x per-output-row e4m3 weights,
// torch._scaled_mm / cutlass_scaled_mm with fp32 accumulation and the same epilogue order) is the
// same kernel with kind::f8f6f4 instructions and fp32 accumulators (FP8 = true).
#include <cuda.h>

#include "common.cuh"
#include "umma.cuh"

namespace sacq {

namespace {

using namespace umma;

constexpr int kDBK = 128;                 // bytes per K block

// A CTA's tile: SUBS sub-tiles of 128 tokens, one accumulator each, x BN weight rows.
template <int SUBS, int BN>
struct DenseTile {
  static constexpr int kTileA = kBM * kDBK;                          // 16 KB: one sub-tile of activations
  static constexpr int kTileB = BN * kDBK;
  static constexpr int kStageBytes = SUBS * kTileA + kTileB;
  static constexpr int kPerSm = SUBS * BN <= 128 ? 2 : 1;            // CTAs that may share an SM
  static constexpr int kStages = 200 * 1024 / kStageBytes;           // of a CTA that has the SM to itself
  static constexpr int kTmemCols = SUBS * BN;
  static constexpr int kEpiWarps = 8 * SUBS;
  static constexpr int kThreads = 64 + kEpiWarps * 32;
  static constexpr int kSwOff = 0, kBiasOff = BN * 4, kBarOff = 2 * BN * 4, kMiscOff = kBarOff + (2 * kStages + 1) * 8,
                       kStageOff = (kMiscOff + 16 + 1023) / 1024 * 1024;
  static constexpr size_t smem(int stages) { return 1024 + kStageOff + (size_t)stages * kStageBytes; }
};

struct DenseParams {
  const float* act_scale;       // [M]
  const float* w_scale;         // [N]
  const uint16_t* bias;         // bf16 [N] or null
  uint16_t* y;                  // bf16 [M, ldy]
  int64_t ldy;
  int* status;
  int M, N, K;
  int stages;
};

__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// FP8: e4m3 operands, fp32 accumulators (kind::f8f6f4); else int8 operands, int32 accumulators.
template <bool FP8, int SUBS, int BN>
__global__ void __launch_bounds__(DenseTile<SUBS, BN>::kThreads, DenseTile<SUBS, BN>::kPerSm)
dense_i8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                const __grid_constant__ DenseParams p) {
  using T = DenseTile<SUBS, BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const int stages = p.stages;
  constexpr int FULL = 0, EMPTY = T::kStages, ACC_FULL = 2 * T::kStages;
  const uint32_t bars = base + T::kBarOff;
  auto bar = [&](int i) { return bars + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + T::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + T::kMiscOff + 8);

  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * (SUBS * kBM);
  const int num_kb = (p.K + kDBK - 1) / kDBK;
  const int subs = SUBS == 2 && p.M - m0 > kBM ? 2 : 1;        // token sub-tiles of this CTA that hold tokens

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(bar(FULL + i), 1);
      mbar_init(bar(EMPTY + i), 1);
    }
    mbar_init(bar(ACC_FULL), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  // Two CTAs of different kernels may share an SM: neither holds TMEM while it waits for the kernel in front, nor lets
  // the kernel behind start before it has its own.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), T::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  if (warp == 0) {
    int st = 0;
    uint32_t free_parity = 1;
    for (int kb = 0; kb < num_kb; ++kb) {
      if (!mbar_wait_warp(bar(EMPTY + st), free_parity, abort_flag, p.status)) break;
      const uint32_t dst = base + T::kStageOff + st * T::kStageBytes;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar(FULL + st), (uint32_t)(subs * T::kTileA + T::kTileB));
        tma_load_2d(dst, &tmap_a, kb * kDBK, m0, bar(FULL + st));
        if (SUBS == 2 && subs == 2) tma_load_2d(dst + T::kTileA, &tmap_a, kb * kDBK, m0 + kBM, bar(FULL + st));
        tma_load_2d(dst + SUBS * T::kTileA, &tmap_b, kb * kDBK, n0, bar(FULL + st));
      }
      if (++st == stages) { st = 0; free_parity ^= 1; }
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t kIdesc = FP8 ? make_idesc(BN) : make_idesc_i8(BN);
    bool ok = true;
    int st = 0;
    uint32_t full_parity = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
      ok = mbar_wait_warp(bar(FULL + st), full_parity, abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      const uint64_t a0_desc = make_smem_desc(base + T::kStageOff + st * T::kStageBytes);
      const uint64_t a1_desc = make_smem_desc(base + T::kStageOff + st * T::kStageBytes + T::kTileA);
      const uint64_t b_desc = make_smem_desc(base + T::kStageOff + st * T::kStageBytes + SUBS * T::kTileA);
#pragma unroll
      for (int ks = 0; ks < kDBK / 32; ++ks) {
        const uint64_t adv = (uint64_t)((ks * 32) >> 4);
        const uint32_t acc = (kb | ks) != 0;
        if (elect_one()) {
          if constexpr (FP8) umma_f8(tmem_base, a0_desc + adv, b_desc + adv, kIdesc, acc);
          else umma_i8(tmem_base, a0_desc + adv, b_desc + adv, kIdesc, acc);
        }
        if (SUBS == 2 && subs == 2 && elect_one()) {
          if constexpr (FP8) umma_f8(tmem_base + BN, a1_desc + adv, b_desc + adv, kIdesc, acc);
          else umma_i8(tmem_base + BN, a1_desc + adv, b_desc + adv, kIdesc, acc);
        }
      }
      if (elect_one()) umma_commit(bar(EMPTY + st));
      if (++st == stages) { st = 0; full_parity ^= 1; }
    }
    if (ok && elect_one()) umma_commit(bar(ACC_FULL));
    __syncwarp();
  } else {
    const int et = threadIdx.x - 64;
    {
      if (et < BN) {
        const int n = min(n0 + et, p.N - 1);
        reinterpret_cast<float*>(sm + T::kSwOff)[et] = __ldg(p.w_scale + n);
        reinterpret_cast<float*>(sm + T::kBiasOff)[et] = p.bias ? bf16_bits_to_float(__ldg(p.bias + n)) : 0.f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(T::kEpiWarps * 32) : "memory");
    }
    const int ew = warp - 2;
    const int quarter = warp & 3;                     // the TMEM lane quarter a warp may read is warp % 4
    const int sub = SUBS == 2 ? (ew >> 2) & 1 : 0, chalf = ew / (4 * SUBS);   // every four consecutive warps cover the four quarters
    const int64_t mw = m0 + sub * kBM + quarter * 32, m = mw + lane;
    const float sa = m < p.M ? __ldg(p.act_scale + m) : 0.f;
    const bool ok = mbar_wait(bar(ACC_FULL), 0, abort_flag, p.status);   // tcgen05.ld below is per warp: no CTA-wide collective
    if (__all_sync(0xffffffffu, ok) && sub < subs) {
      tc_fence_after();
      const float* swp = reinterpret_cast<const float*>(sm + T::kSwOff);
      const float* bp = reinterpret_cast<const float*>(sm + T::kBiasOff);
      const bool has_bias = p.bias != nullptr;
      constexpr int kStagePitch = 80;                 // of a token's 64 bytes: the pitch spreads the banks
      uint8_t* stage = sm + T::kStageOff + ew * 32 * kStagePitch;      // every operand stage has been read by now
#pragma unroll 1
      for (int cc = 0; cc < BN / 64; ++cc) {
        const int c0 = chalf * (BN / 2) + cc * 32;
        if (n0 + c0 >= p.N) break;
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(sub * BN + c0), r);
        // weight scale first, then the token scale; the bias rides in the same fused multiply-add
        auto fin = [&](int c) -> uint32_t {
          const float scaled = __fmul_rn(FP8 ? __uint_as_float(r[c]) : __int2float_rn((int)r[c]), swp[c0 + c]);
          const float v = has_bias ? fmaf(sa, scaled, bp[c0 + c]) : __fmul_rn(sa, scaled);
          return (uint32_t)float_to_bf16_bits(v);
        };
        uint16_t* y = p.y + n0 + c0;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) o[j] = fin(v * 8 + 2 * j) | (fin(v * 8 + 2 * j + 1) << 16);
          *reinterpret_cast<uint4*>(stage + lane * kStagePitch + v * 16) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        __syncwarp();
        if (n0 + c0 + 32 <= p.N && (reinterpret_cast<uintptr_t>(y) & 15) == 0 && (p.ldy & 7) == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {               // four lanes per token: whole 32-byte sectors
            const int row = i * 8 + (lane >> 2);
            const uint4 o = *reinterpret_cast<const uint4*>(stage + row * kStagePitch + (lane & 3) * 16);
            if (mw + row < p.M) *reinterpret_cast<uint4*>(y + (mw + row) * p.ldy + (lane & 3) * 8) = o;
          }
        } else if (n0 + c0 + lane < p.N) {            // rows that begin or end anywhere: an element per lane
          const int rows = (int)(p.M - mw < 32 ? p.M - mw : 32);
#pragma unroll 8
          for (int row = 0; row < rows; ++row)
            y[(mw + row) * p.ldy + lane] = *reinterpret_cast<const uint16_t*>(stage + row * kStagePitch + lane * 2);
        }
        __syncwarp();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, T::kTmemCols);
}

template <bool FP8, int SUBS, int BN>
int launch_dense_tile(const CUtensorMap& ta, const CUtensorMap& tb, DenseParams p, int num_sms, cudaStream_t s) {
  using T = DenseTile<SUBS, BN>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    SACQ_CUDA_TRY(cudaFuncSetAttribute(dense_i8_kernel<FP8, SUBS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem(T::kStages)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.N + BN - 1) / BN), (unsigned)((p.M + SUBS * kBM - 1) / (SUBS * kBM)));
  if (cfg.gridDim.y > 65535) return set_error(SACQ_ERR_UNSUPPORTED, "M=%d exceeds the grid limit", p.M);
  cfg.blockDim = dim3(T::kThreads);
  // the operand stages of a whole SM for a CTA that has it to itself, half of them where two share one
  p.stages = T::kPerSm == 2 && (int)(cfg.gridDim.x * cfg.gridDim.y) > num_sms ? T::kStages / 2 : T::kStages;
  cfg.dynamicSmemBytes = T::smem(p.stages);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SACQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, dense_i8_kernel<FP8, SUBS, BN>, ta, tb, p));
  count_launch();
  return SACQ_OK;
}

template <bool FP8>
int launch_dense(int subs, int bn, const CUtensorMap& ta, const CUtensorMap& tb, const DenseParams& p, int sms, cudaStream_t s) {
  if (subs == 2) return bn == 256 ? launch_dense_tile<FP8, 2, 256>(ta, tb, p, sms, s) : launch_dense_tile<FP8, 2, 128>(ta, tb, p, sms, s);
  return bn == 128 ? launch_dense_tile<FP8, 1, 128>(ta, tb, p, sms, s) : launch_dense_tile<FP8, 1, 64>(ta, tb, p, sms, s);
}

// The tile of a call, by a model of its time that was fitted to 48 sizes (five widths, 64 to 8,192 tokens, FP8; the
// tile it names was within 2 % of the best at each): the largest number of tiles that an SM gets, at so much per K
// block and so much around them, or the time the operands take through L2 at 19 TB/s, whichever is longer.  The big
// tile, bound by the tensor cores (0.48 us per K block of 2 x 128 x 256 x 128), needs the fewest bytes; the small
// ones fill the chip at few tokens.
void dense_choose(const sacq_layer* L, int64_t M, int* subs, int* bn) {
  static const struct { int subs, bn; double block_us, tile_us; } tiles[] = {
      {2, 256, 0.48, 4.0}, {2, 128, 0.28, 4.0}, {1, 128, 0.17, 1.2}, {1, 64, 0.11, 1.5}};
  const int64_t kb = (L->d.in_features + kDBK - 1) / kDBK;
  double best = 1e30;
  for (const auto& t : tiles) {
    if ((M + t.subs * kBM - 1) / (t.subs * kBM) > 65535 && t.subs == 1) continue;   // token tiles are the grid's second dimension
    const int64_t ctas = ((M + t.subs * kBM - 1) / (t.subs * kBM)) * ((L->d.out_features + t.bn - 1) / t.bn);
    const double sm = (double)((ctas + L->num_sms - 1) / L->num_sms) * (kb * t.block_us + t.tile_us);
    const double l2 = (double)ctas * kb * (t.subs * kBM + t.bn) * kDBK / 19e6 + 1.2;
    const double us = sm > l2 ? sm : l2;
    if (us < best) {
      best = us;
      *subs = t.subs;
      *bn = t.bn;
    }
  }
}

}  // namespace

bool dense_i8_supported(const sacq_layer* L) { return L->d.in_features % 16 == 0 && L->d.in_features >= 16; }

// y = epilogue(q [M,K] int8 x wq [N,K] int8): the dense part of the INT8 recipe.
int launch_dense_i8(const sacq_layer* L, const void* q, const float* act_scale, const void* wq, const float* w_scale,
                    int64_t M, void* y, int64_t ldy, cudaStream_t s, bool fp8) {
  const sacq_layer_desc& d = L->d;
  if (M <= 0 || d.out_features == 0) return SACQ_OK;
  if (!dense_i8_supported(L))
    return set_error(SACQ_ERR_UNSUPPORTED, "the 8-bit GEMM needs in_features to be a multiple of 16, got %lld",
                     (long long)d.in_features);
  if (reinterpret_cast<uintptr_t>(q) % 16 != 0 || reinterpret_cast<uintptr_t>(wq) % 16 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "8-bit GEMM operands must be 16-byte aligned");
  if (!fp8 && (int64_t)d.in_features * 127 * 127 > 2147483647LL)
    return set_error(SACQ_ERR_UNSUPPORTED, "in_features=%lld could overflow the int32 accumulator", (long long)d.in_features);
  int subs = 2, bn = 256;
  dense_choose(L, M, &subs, &bn);
  CUtensorMap ta, tb;
  int rc = encode_bytes_2d(&ta, q, (uint64_t)d.in_features, (uint64_t)M, (uint64_t)d.in_features, kDBK, kBM,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != SACQ_OK) return rc;
  rc = encode_bytes_2d(&tb, wq, (uint64_t)d.in_features, (uint64_t)d.out_features, (uint64_t)d.in_features, kDBK, bn,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != SACQ_OK) return rc;
  DenseParams p{};
  p.act_scale = act_scale;
  p.w_scale = w_scale;
  p.bias = static_cast<const uint16_t*>(d.bias);
  p.y = static_cast<uint16_t*>(y);
  p.ldy = ldy;
  p.status = L->d_status;
  p.M = (int)M; p.N = (int)d.out_features; p.K = (int)d.in_features;
  return fp8 ? launch_dense<true>(subs, bn, ta, tb, p, L->num_sms, s) : launch_dense<false>(subs, bn, ta, tb, p, L->num_sms, s);
}

}  // namespace sacq
