// Large-M quantized linear for GROUPED scales with the expanded weights in tensor memory:
//   y[m,n] = bf16( s[m] * (sum_k q[m,k] * cb[idx[n,k/d], k%d] * scale[n, k/G]) + bias[n] )
//
// The layouts the reference deployed (dim-4 vectors, one scale per 64 weights, 5- to 11-bit
// indices; gr00t_libero/acceleration/presets/FROZEN_DECODE_SELECTION.json) change their scale
// inside the K loop, so the scale is folded into the weight operand: fp16(codeword x scale),
// tcgen05 kind::f16 (linear_large_m_grouped.cu explains the encoding).  Structured like
// linear_large_m_tmem.cu, persistent CTAs included:
//   * a tile is 128 weight rows (the 128 TMEM lanes) x up to 384 tokens;
//   * the packed index tile of a super-block (128 indices = 16*bits bytes per row) is staged as
//     16-byte column slices, [slice][row][16 B] (one TMA box of 16 bytes x 128 rows per slice): a
//     thread reads its row's slice with one 16-byte load and the 32 lanes of a warp read 512
//     contiguous bytes, free of bank conflicts (row-major rows of 16*bits bytes would put the
//     lanes of a warp 4 to 32 deep on the same banks);
//   * 16 expander warps: a thread owns one weight row and a quarter of each 64-k block (16
//     weights): it extracts its index fields (runtime width) from two slices held in registers,
//     gathers the fp16 codewords from the shared-memory codebook, multiplies by the row's group
//     scale (HMUL2) and writes 8 registers to the weight stage with tcgen05.st -- no
//     shared-memory store;
//   * the fp16 activation tiles (e4m3 or int8 widened exactly by a pre-pass into the caller's
//     workspace) are the MMA's B operand, TMA-loaded K-major / SWIZZLE_128B;
//   * warp 1 issues tcgen05.mma.kind::f16 with A from TMEM: four K = 16 steps per 64-k block
//     (384 tokens as two N = 192 instructions into two accumulators);
//   * epilogue: the shared transposing epilogue (tiled bulk stores).  The scales of the next tile's rows
//     are fetched while the last MMAs of a tile run.
// TMEM: the accumulator columns + up to four weight stages of 64 columns (two K blocks each).
// What bounds it: the expanders (gathers and scale products) up to 256 tokens, shared memory above.  Quantizer, widening and
// GEMM at d = 4, 10-bit, group 64, one tile per CTA / now: 2048 -> 6144 at 1,500 tokens 52 / 41 us, at 8,192 217 / 203;
// 1024 -> 4096 at 2,048 32.5 / 24.4; 6144 -> 2048 at 1,024 51 / 45, at 3,000 76 / 78.
//
// Replaces, for batched sizes, the reference's per-forward decode kernel plus 8-bit GEMM on
// these layouts (perrow_int8_fused_decode_r1.py:12-88, perrow_a8_candidate_r3.py:56-69).
#include <cuda.h>
#include <math.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "tmem_weights.cuh"
#include "umma.cuh"
#include "widen.cuh"

namespace sacq {

namespace {

using namespace umma;
using namespace tmemw;

constexpr int kBKh = 64;                      // fp16 elements per K block: one 128-byte swizzle row
constexpr int kSbIdx = 128;                   // indices per row per index super-block (16 * bits bytes)
constexpr int kAliasTok = 256;                // from here on an activation stage holds the epilogue's staging
static_assert(epi_staging(kAliasTok) <= kAliasTok * 128, "staging in an activation stage");
constexpr int kGMaxActStages = 6;
constexpr int kGMaxWStages = 4;               // TMEM weight stages of 64 columns (two K blocks)
constexpr float kPreScale = 4096.f;           // keeps fp16(codeword x scale) far from the subnormals

struct GTmemParams {
  const __half* cb_f16;         // [C][D] codebook * 2^cb_exp_shift
  const uint16_t* scales;       // bf16 [N, num_groups]
  const uint16_t* bias;         // bf16 [N] or null
  const float* act_scale;       // [M]
  TmemOut out;
  int* status;
  int K, C;
  int bits, num_groups, group_size;
  TilePlan plan;
  int act_stages;
  float scale_mul;              // 2^sc_exp_shift * kPreScale, applied to every scale
  float out_mul;                // 2^-(cb_exp_shift + sc_exp_shift) / kPreScale
};

struct GTmemLayout {
  uint32_t act_off, act_stage, stg_off, idx_off, idx_slot, cb_off, sc_off, sw_off, bias_off, sa_off, bar_off, misc_off, total;
};

__host__ __device__ inline GTmemLayout gtmem_layout(int tok, int act_stages, int bits, int cb_bytes, int num_groups) {
  GTmemLayout L;
  L.act_off = 0;
  L.act_stage = (uint32_t)(tok * 128);
  L.stg_off = (uint32_t)act_stages * L.act_stage;
  // wide tiles stage their output in the activation stage of their last block, which is the last to be refilled
  L.idx_off = L.stg_off + (tok >= kAliasTok ? 0u : epi_staging(tok));
  L.idx_slot = (uint32_t)(kRows * 16 * bits);
  L.cb_off = (L.idx_off + 2 * L.idx_slot + 127) & ~127u;
  L.sc_off = L.cb_off + (uint32_t)((cb_bytes + 127) & ~127);
  // bf16 scales of the tile's rows, row pitch num_groups + 1 (odd or even, never a multiple of the 32 banks'
  // period for the 32 consecutive rows of a warp: an unpadded pitch of 64 bytes made every read a 16-way conflict)
  L.sw_off = L.sc_off + (uint32_t)((kRows * (num_groups | 1) * 2 + 127) & ~127);
  L.bias_off = L.sw_off + kRows * 4;
  L.sa_off = L.bias_off + kRows * 4;
  L.bar_off = L.sa_off + kMaxTok * 4;
  L.misc_off = L.bar_off + 32 * 8;
  L.total = L.misc_off + 64;
  return L;
}

// D in {4, 8}.  grid = workers.
template <int D>
__global__ void __launch_bounds__(kCtaThreads, 1)
large_m_tmem_grouped_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_idx,
                            const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ BcastMaps tmap_bc,
                            const __grid_constant__ GTmemParams p) {
  constexpr int IDX_PER_KB = kBKh / D;                // indices per row per K block
  constexpr int KB_PER_SB = kSbIdx / IDX_PER_KB;      // K blocks per index super-block
  constexpr int IPT = IDX_PER_KB / 4;                 // indices per expander thread per K block (16 weights)
  // A weight stage holds TWO K blocks (128 k, 64 columns): the per-stage cost of the expanders and of the
  // issuer (barrier waits, tcgen05.wait::st, fences, commits) is paid half as often as with one block per stage.
  constexpr uint32_t kTmemCols = 512;
  using CwVec = typename std::conditional<D == 8, uint4, uint2>::type;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const GTmemLayout L = gtmem_layout(p.plan.tok, p.act_stages, p.bits, p.C * D * 2, p.num_groups);

  constexpr int ACT_FULL = 0, ACT_EMPTY = kGMaxActStages, W_FULL = 2 * kGMaxActStages,
                W_EMPTY = 2 * kGMaxActStages + kGMaxWStages, IDX_FULL = 2 * kGMaxActStages + 2 * kGMaxWStages,
                IDX_EMPTY = IDX_FULL + 2, ACC_FULL = IDX_FULL + 4, ACC_EMPTY = IDX_FULL + 5, CB_FULL = IDX_FULL + 6,
                EPI_DONE = IDX_FULL + 7;
  static_assert(EPI_DONE < 32, "barrier region");
  const uint32_t bars = base + L.bar_off;
  auto bar = [&](int i) { return bars + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L.misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L.misc_off + 8);

  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int worker = (int)blockIdx.x;
  const TileWalk walk(p.plan, worker);
  const int items = walk.items;
  auto tile = [&](int t, int& n0, int& m0, int& tok) { walk.tile(p.plan, worker, t, n0, m0, tok); };
  const int num_kb = p.K / kBKh;
  const int act_stages = p.act_stages;
  const int sb_bytes = 16 * p.bits;
  const int w_stages = min(kGMaxWStages, ((int)kTmemCols - p.plan.tok) / 64);
  const int sbs = (num_kb + KB_PER_SB - 1) / KB_PER_SB;         // index super-blocks of a tile

  if (threadIdx.x == 0) {
    for (int i = 0; i < kGMaxActStages; ++i) {
      mbar_init(bar(ACT_FULL + i), 1);
      mbar_init(bar(ACT_EMPTY + i), 1);
    }
    for (int i = 0; i < kGMaxWStages; ++i) {
      mbar_init(bar(W_FULL + i), kXWarps);
      mbar_init(bar(W_EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(IDX_FULL + i), 1);
      mbar_init(bar(IDX_EMPTY + i), kXWarps);
    }
    mbar_init(bar(ACC_FULL), 1);
    mbar_init(bar(ACC_EMPTY), kXWarps);
    mbar_init(bar(CB_FULL), 1);
    mbar_init(bar(EPI_DONE), kXWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == 0) {
    __syncwarp();
    if (elect_one()) {                                // constant operand: its copy starts before anything else
      mbar_arrive_expect_tx(bar(CB_FULL), (uint32_t)(p.C * D * 2));
      bulk_load(base + L.cb_off, p.cb_f16, (uint32_t)(p.C * D * 2), bar(CB_FULL));
      prefetch_tensormap(&tmap_a);
      prefetch_tensormap(&tmap_idx);
      if (p.out.y_tma) prefetch_tensormap(&tmap_y);
    }
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    int st = 0, sb = 0;                               // index super-blocks: counted over all tiles
    const bool alias = p.plan.tok >= kAliasTok;
    int until_staging = num_kb + act_stages - 1, epi = 0;   // blocks before the one that goes where tile `epi` staged its output
    uint32_t free_parity = 1;
    bool ok = true;
    for (int t = 0; t < items && ok; ++t) {
      int n0, m0, tok;
      tile(t, n0, m0, tok);
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        if (kb % KB_PER_SB == 0) {
          const int slot = sb & 1;
          ok = mbar_wait_warp(bar(IDX_EMPTY + slot), ((sb >> 1) & 1) ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (elect_one()) mbar_arrive_expect_tx(bar(IDX_FULL + slot), (uint32_t)(kRows * sb_bytes));
          for (int sl = 0; sl < p.bits; ++sl)          // one 16-byte column slice of the 128 rows per copy
            if (elect_one())
              tma_load_2d(base + L.idx_off + slot * L.idx_slot + sl * (kRows * 16), &tmap_idx,
                          kb / KB_PER_SB * sb_bytes + sl * 16, n0, bar(IDX_FULL + slot));
          ++sb;
          if (t == 0 && kb == 0) asm volatile("griddepcontrol.wait;" ::: "memory");   // activations: from the kernel in front
        }
        ok = mbar_wait_warp(bar(ACT_EMPTY + st), free_parity, abort_flag, p.status);
        if (!ok) break;
        if (alias && until_staging-- == 0) {
          ok = mbar_wait_warp(bar(EPI_DONE), (uint32_t)epi++ & 1u, abort_flag, p.status);
          if (!ok) break;
          until_staging = num_kb - 1;
        }
        const uint32_t dst = base + L.act_off + st * L.act_stage;
        if (elect_one()) mbar_arrive_expect_tx(bar(ACT_FULL + st), (uint32_t)(tok * 128));
        for (int b = 0; b < tok; b += p.plan.box)
          if (elect_one()) tma_load_2d(dst + (uint32_t)(b * 128), &tmap_a, kb * 128, m0 + b, bar(ACT_FULL + st));
        if (++st == act_stages) { st = 0; free_parity ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    bool ok = true;
    int st = 0, ws = 0;
    uint32_t act_parity = 0, w_parity = 0;
    for (int t = 0; t < items && ok; ++t) {
      int n0, m0, tok;
      tile(t, n0, m0, tok);
      const int mmas = tok > 256 ? 2 : 1;             // an instruction takes at most 256 tokens
      const uint32_t part = (uint32_t)(tok / mmas), idesc = make_idesc(tok / mmas);
      // the epilogue has read the last tile's accumulators
      if (t > 0 && !mbar_wait_warp(bar(ACC_EMPTY), (uint32_t)(t - 1) & 1u, abort_flag, p.status)) break;
      for (int wi = 0; wi < num_kb / 2 && ok; ++wi) {         // weight stage by weight stage: two K blocks each
        ok = mbar_wait_warp(bar(W_FULL + ws), w_parity, abort_flag, p.status);
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          ok = ok && mbar_wait_warp(bar(ACT_FULL + st), act_parity, abort_flag, p.status);
          if (!ok) break;
          tc_fence_after();
          const uint32_t act_addr = base + L.act_off + st * L.act_stage;
          const uint64_t b0 = make_smem_desc(act_addr), b1 = make_smem_desc(act_addr + part * 128u);
          const uint32_t w_col = tmem_base + (uint32_t)(kTmemCols - (ws + 1) * 64 + sub * 32);
#pragma unroll
          for (int ks = 0; ks < kBKh / 16; ++ks) {
            const uint64_t adv = (uint64_t)((ks * 32) >> 4);            // 16 fp16 = 32 bytes per K step
            const uint32_t a_tmem = w_col + (uint32_t)(ks * 8);
            const uint32_t acc = (wi | sub | ks) != 0;
            if (elect_one()) umma_f16_ts(tmem_base, a_tmem, b0 + adv, idesc, acc);
            if (mmas == 2 && elect_one()) umma_f16_ts(tmem_base + part, a_tmem, b1 + adv, idesc, acc);
          }
          if (elect_one()) umma_commit(bar(ACT_EMPTY + st));
          if (++st == act_stages) { st = 0; act_parity ^= 1; }
        }
        if (ok && elect_one()) umma_commit(bar(W_EMPTY + ws));
        if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
      }
      if (ok && elect_one()) umma_commit(bar(ACC_FULL));
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ expanders, then epilogue
    const int et = threadIdx.x - 64;                 // 0..511
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;             // weight row of the tile = TMEM lane
    const int kpart = (warp - 2) >> 2;               // which 16 weights of the 64-k block (0..3)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint16_t* sc_tile = reinterpret_cast<uint16_t*>(sm + L.sc_off);
    float* sw = reinterpret_cast<float*>(sm + L.sw_off);
    float* bias = reinterpret_cast<float*>(sm + L.bias_off);
    float* sa = reinterpret_cast<float*>(sm + L.sa_off);
    const int sc_pitch = p.num_groups | 1;
    const bool alias = p.plan.tok >= kAliasTok;
    // a tile's scales (bf16, all groups of its rows); between barriers of the expander warps
    auto fetch_scales = [&](int n0) {
      for (int i = et; i < kRows * p.num_groups; i += kXThreads) {
        const int r = i / p.num_groups, g = i - r * p.num_groups;
        const int n = min(n0 + r, p.out.N - 1);
        sc_tile[r * sc_pitch + g] = __ldg(p.scales + (int64_t)n * p.num_groups + g);
      }
    };
    int n0, m0, tok;
    tile(0, n0, m0, tok);
    fetch_scales(n0);
    if (et < kRows) sw[et] = p.out_mul;
    xbarrier();
    const CwVec* cbs = reinterpret_cast<const CwVec*>(sm + L.cb_off);
    const uint16_t* sc = sc_tile + row * sc_pitch;
    const uint32_t mask = (1u << p.bits) - 1u;
    const int kb_per_group = p.group_size / kBKh;
    bool ok = mbar_wait_warp(bar(CB_FULL), 0, abort_flag, p.status);
    int ws = 0, sb0 = 0;                              // the tile's first index super-block, counted over all tiles
    uint32_t w_parity = 1;
    for (int t = 0; t < items && ok; ++t) {
      int grp = 0, left_in_group = kb_per_group;
      for (int wi = 0; wi < num_kb / 2 && ok; ++wi) {
        ok = mbar_wait_warp(bar(W_EMPTY + ws), w_parity, abort_flag, p.status);
        if (!ok) break;
        tc_fence_after();                              // the MMAs that read this stage are complete
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          const int kb = 2 * wi + sub;
          const int sb = sb0 + kb / KB_PER_SB, slot = sb & 1;
          if (kb % KB_PER_SB == 0) ok = mbar_wait_warp(bar(IDX_FULL + slot), (sb >> 1) & 1, abort_flag, p.status);
          if (!ok) break;
          // scale * 2^sc_exp_shift * 4096 is a bf16 significand with a small exponent: exact in fp16
          const __half sh = __float2half_rn(bf16_bits_to_float(sc[grp]) * p.scale_mul);
          const __half2 s2 = __half2half2(sh);
          // this thread's IPT index fields: a window of at most 64 bits that starts at bit `bit0` of the row's
          // super-block, i.e. in slice bit0 / 128 and possibly the next one; bit0 is the same for the whole warp
          const int bit0 = ((kb % KB_PER_SB) * IDX_PER_KB + kpart * IPT) * p.bits;
          const int sl0 = bit0 >> 7;
          const uint8_t* slice = sm + L.idx_off + slot * L.idx_slot + row * 16;
          const uint4 a = *reinterpret_cast<const uint4*>(slice + sl0 * (kRows * 16));
          uint4 b = a;                                     // the next slice only when the window crosses into it
          if ((bit0 & 127) + IPT * p.bits > 128) b = *reinterpret_cast<const uint4*>(slice + (sl0 + 1) * (kRows * 16));
          uint32_t lo, mid, hi;
          switch ((bit0 >> 5) & 3) {                       // first word of the window inside slice sl0 (warp-uniform)
            case 0: lo = a.x; mid = a.y; hi = a.z; break;
            case 1: lo = a.y; mid = a.z; hi = a.w; break;
            case 2: lo = a.z; mid = a.w; hi = b.x; break;
            default: lo = a.w; mid = b.x; hi = b.y; break;
          }
          const uint32_t wsh = (uint32_t)(bit0 & 31);
          const uint64_t win = ((uint64_t)__funnelshift_r(mid, hi, wsh) << 32) | __funnelshift_r(lo, mid, wsh);
          uint32_t o[8];
#pragma unroll
          for (int j = 0; j < IPT; ++j) {
            const CwVec cw = cbs[(uint32_t)(win >> (j * p.bits)) & mask];
            if constexpr (D == 8) {
              const uint32_t w4[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&w4[e]), s2);
                o[4 * j + e] = *reinterpret_cast<const uint32_t*>(&h);
              }
            } else {
              const uint32_t w2[2] = {cw.x, cw.y};
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&w2[e]), s2);
                o[2 * j + e] = *reinterpret_cast<const uint32_t*>(&h);
              }
            }
          }
          tmem_st_32x8(lane_addr + (uint32_t)(kTmemCols - (ws + 1) * 64 + sub * 32 + kpart * 8), o);
          if (--left_in_group == 0) { ++grp; left_in_group = kb_per_group; }
        }
        if (!ok) break;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(W_FULL + ws));
          // the index slot is free once its last K block has been read (KB_PER_SB is even: that is an odd block)
          const int kb_last = 2 * wi + 1;
          if ((kb_last + 1) % KB_PER_SB == 0 || kb_last == num_kb - 1) mbar_arrive(bar(IDX_EMPTY + ((sb0 + kb_last / KB_PER_SB) & 1)));
        }
        if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
      }
      sb0 += sbs;

      // ---- epilogue.  While the last MMAs run: the token scales and biases, and the next tile's group scales
      ok = xall(ok);                                  // every warp is done with the tile's scales and the last tile's epilogue
      if (!ok) break;
      asm volatile("griddepcontrol.wait;" ::: "memory");   // the token scales; the kernel in front has long gone
      if (et < tok) sa[et] = m0 + et < p.out.M ? __ldg(p.act_scale + m0 + et) : 0.f;
      if (et < kRows) bias[et] = p.bias ? bf16_bits_to_float(__ldg(p.bias + min(n0 + et, p.out.N - 1))) : 0.f;
      const int n0_now = n0, m0_now = m0, tok_now = tok;
      if (t + 1 < items) {
        tile(t + 1, n0, m0, tok);
        fetch_scales(n0);
      }
      ok = mbar_wait_warp(bar(ACC_FULL), (uint32_t)t & 1u, abort_flag, p.status);
      ok = xall(ok);                                  // also: all of them are in place
      if (!ok) break;
      tc_fence_after();
      uint8_t* stage = alias ? sm + L.act_off + (uint32_t)(((t + 1) * num_kb - 1) % act_stages) * L.act_stage : sm + L.stg_off;
      tile_epilogue(p.out, &tmap_y, tmap_bc.m, lane_addr, quarter, kpart, tok_now, sa, sw, bias, stage, m0_now, n0_now,
                    bar(ACC_EMPTY));
      if (alias) {
        tma_store_wait_read<0>();                     // the stores have read the staged tiles
        // ... and so have the warp's own loads and stores (residual, unaligned y), which the activation copy that
        // overwrites the stage, an asynchronous one, has to come after
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(EPI_DONE));
      }
    }
    // shared memory stays valid until every store has read it; the writes themselves (local and peer)
    // are in the memory system then, like plain stores, and the grid's end orders them
    tma_store_wait_read<0>();
  }

  // ---- common exit: every thread arrives here, also after an aborted wait
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
}

constexpr int64_t kGSlabTokens = 3072;   // tokens widened per launch (8 tiles of 384): bounds the fp16 scratch

int g_act_stages(const sacq_layer* L, int tok) {
  const int cb_bytes = L->cb_entries * L->d.vector_dim * 2;
  for (int st = kGMaxActStages; st >= 2; --st)
    if (gtmem_layout(tok, st, L->d.index_bits, cb_bytes, (int)L->num_groups).total + 1024 <= 227 * 1024) return st;
  return 0;
}

template <int D>
cudaError_t glaunch(const CUtensorMap& ta, const CUtensorMap& ti, const CUtensorMap& ty, const BcastMaps& tb,
                    const GTmemParams& p, size_t smem, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(large_m_tmem_grouped_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.plan.workers);
  cfg.blockDim = dim3(kCtaThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, large_m_tmem_grouped_kernel<D>, ta, ti, ty, tb, p);
}

// Time of a tile (us), fitted to d = 4, 10-bit, group 64 at 1,024 - 8,192 tokens.
double g_tile_us(const sacq_layer* L, int tok) {
  if (g_act_stages(L, tok) < 2) return 1e9;
  // two activation stages (64 KB of codebook) leave the tensor cores waiting for tiles
  const double least = 0.75, rate = (tok <= 256 ? 0.0039 : g_act_stages(L, tok) > 2 ? 0.0035 : 0.0042) * tok;
  const double block = rate > least ? rate : least;
  return 3.0 + 0.0026 * tok + (double)L->d.in_features / 128 * block;
}

}  // namespace

int64_t large_m_tmem_grouped_slab(void) { return kGSlabTokens; }

bool large_m_tmem_grouped_supported(const sacq_layer* L) {
  const sacq_layer_desc& d = L->d;
  if (d.vector_dim != 8 && d.vector_dim != 4) return false;
  if (d.index_bits < 1 || d.index_bits > 16) return false;
  if (!L->rows_16b_aligned) return false;
  if (d.in_features % (2 * kBKh) != 0 || d.group_size % kBKh != 0) return false;   // whole weight stages of two K blocks
  if (((size_t)L->cb_entries * d.vector_dim * 2) % 16 != 0) return false;
  if (has_shift(L)) return false;
  return g_act_stages(L, 32) >= 2;
}

// From how many tokens this kernel beats the split-K kernel (linear_large_m_grouped.cu), whose clusters stop
// paying once whole token tiles fill the device, and which walks more than 1,024 tokens in slabs (quantizer + GEMM at
// d = 4, 10-bit, group 64, split-K / this: 2048x6144 32.4 / 23.8 us at 600 tokens; 1024x4096 13.1 / 12.8 at 600, 23.8 /
// 15.3 at 1,024; 2048x2048 19.7 / 20.9 at 1,024, 33.5 / 23.0 at 1,500; 6144x2048 45.0 / 45.3 and 69.5 / 56.2).
int64_t large_m_tmem_grouped_min_m(const sacq_layer* L) {
  return L->d.out_features >= 5120 ? 448 : L->d.out_features >= 4096 ? 600 : 1025;
}

double large_m_tmem_grouped_us(const sacq_layer* L, int64_t M) {
  TilePlan p;
  double us;
  return plan_tiles(L, M, g_tile_us, 0, &p, &us) ? us : 1e30;
}

// Workspace behind the counter region: the fp16 activations of one token slab.
int64_t large_m_tmem_grouped_workspace_bytes(const sacq_layer* L, int64_t M) {
  const int64_t rows = M < kGSlabTokens ? M : kGSlabTokens;
  return (rows * L->d.in_features * 2 + 255) & ~(int64_t)255;
}

int launch_large_m_tmem_grouped(const sacq_layer* L, const void* q, const float* scale, int64_t M, void* y, int64_t ldy,
                                void* ws, int64_t ws_bytes, cudaStream_t s, const void* residual, int64_t ldr,
                                ActForm form, const BcastDst* bc, int nt_force) {
  const sacq_layer_desc& d = L->d;
  if (!large_m_tmem_grouped_supported(L))
    return set_error(SACQ_ERR_UNSUPPORTED, "grouped TMEM-weight kernel cannot run this layer geometry");
  if (M <= 0 || d.out_features == 0) return SACQ_OK;
  if (reinterpret_cast<uintptr_t>(q) % 8 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "quantized activations must be 8-byte aligned");
  const int64_t need = large_m_tmem_grouped_workspace_bytes(L, M);
  if (form == kActHalf ? M > kGSlabTokens : ws == nullptr || ws_bytes < need)
    return set_error(SACQ_ERR_WORKSPACE, "workspace of %lld bytes needed behind the counter region, %lld given",
                     (long long)need, (long long)ws_bytes);
  if (form != kActHalf && reinterpret_cast<uintptr_t>(ws) % 256 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  const int64_t K = d.in_features, N = d.out_features;
  const int64_t slab = M < kGSlabTokens ? M : kGSlabTokens;
  const void* a16 = form == kActHalf ? q : ws;

  GTmemParams p{};
  p.cb_f16 = L->cb_f16;
  p.scales = static_cast<const uint16_t*>(d.scales);
  p.bias = static_cast<const uint16_t*>(d.bias);
  p.status = L->d_status;
  p.K = (int)K; p.C = L->cb_entries;
  p.bits = d.index_bits; p.num_groups = (int)L->num_groups; p.group_size = d.group_size;
  p.scale_mul = ldexpf(kPreScale, L->sc_exp_shift);
  p.out_mul = ldexpf(1.f / kPreScale, -(L->cb_exp_shift + L->sc_exp_shift));

  for (int64_t m0 = 0; m0 < M; m0 += slab) {
    const int64_t rows = (M - m0) < slab ? (M - m0) : slab;
    if (form != kActHalf)
      if (int rc = launch_widen(static_cast<const uint8_t*>(q) + m0 * K, rows, K, form == kActInt8, ws, s)) return rc;
    if (!plan_tiles(L, rows, g_tile_us, kBM * nt_force, &p.plan))
      return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld: too many tiles", (long long)M);
    p.act_stages = g_act_stages(L, p.plan.tok);
    if (p.act_stages < 2) return set_error(SACQ_ERR_UNSUPPORTED, "grouped TMEM-weight kernel: no tile fits shared memory");
    CUtensorMap ta, ti, ty;
    int rc = encode_bytes_2d(&ta, a16, (uint64_t)(K * 2), (uint64_t)rows, (uint64_t)(K * 2), 128, p.plan.box,
                             CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != SACQ_OK) return rc;
    const uint64_t row_bytes = (uint64_t)(L->row_bits / 8);
    rc = encode_bytes_2d(&ti, d.packed, row_bytes, (uint64_t)N, row_bytes, 16u, (uint32_t)kRows, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc != SACQ_OK) return rc;
    ty = ta;                                          // a valid map is passed either way
    BcastMaps tb = {};
    BcastDst bc_slab;
    if (bc != nullptr) {
      bc_slab = *bc;
      for (int i = 0; i < bc->n; ++i) bc_slab.ptr[i] = static_cast<uint16_t*>(bc->ptr[i]) + m0 * ldy;
    }
    rc = tile_output(L, rows, static_cast<uint16_t*>(y) + m0 * ldy, ldy,
                     residual ? static_cast<const uint16_t*>(residual) + m0 * ldr : nullptr, ldr, bc ? &bc_slab : nullptr, &p.out,
                     &ty, &tb);
    if (rc != SACQ_OK) return rc;
    p.act_scale = scale + m0;
    const GTmemLayout lay =
        gtmem_layout(p.plan.tok, p.act_stages, d.index_bits, L->cb_entries * d.vector_dim * 2, (int)L->num_groups);
    size_t smem = lay.total + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;      // two CTAs (each takes all 512 TMEM columns) never share an SM
    const cudaError_t e = d.vector_dim == 8 ? glaunch<8>(ta, ti, ty, tb, p, smem, s) : glaunch<4>(ta, ti, ty, tb, p, smem, s);
    count_launch();
    if (e != cudaSuccess) return cuda_fail(e, "grouped TMEM-weight launch");
  }
  return SACQ_OK;
}

}  // namespace sacq
