// Batched quantized linear with the expanded weights held in TENSOR MEMORY (sm_100a), persistent:
//   y[m,n] = bf16( s[m] * (sum_k q[m,k] * cb[idx[n,k/d], k%d]) * scale[n] + bias[n] )
//
//   * the WEIGHTS are the MMA's A operand (128 weight rows = the 128 TMEM lanes) and live in tensor
//     memory: an expander thread gathers its row's codewords (FP8 high and low halves) from the
//     shared-memory codebook into registers and writes them with tcgen05.st;
//   * the ACTIVATIONS are the B operand (N = tokens), TMA-loaded K-major / SWIZZLE_128B tiles, read by
//     the tensor core straight from shared memory;
//   * D[weight row, token] accumulates in TMEM: 128 lanes x `tok` fp32 columns.
// Per 32-wide K step one MMA with the high and one with the low codeword halves go into the same
// accumulator, so the summation order of an output element is the same for every tile shape (row shards
// of a layer reproduce it bit for bit).
//
// A tile is 128 weight rows x `tok` tokens, a multiple of 32 up to 256 (one MMA) or of 64 up to 384 (two of
// tok / 2).  TMEM: columns [0, tok) accumulate, the rest are weight stages of 64 (32 of high, 32 of low halves).
// One CTA per SM takes tile after tile: the start-up of a CTA (3 us to its first MMA) is paid once, activation
// tiles, indices and the first weight stages of the next tile are there when the epilogue ends, and a last, narrower
// tile per weight row takes the tokens that are left.
//
// Roles: warp 0 = TMA producer (activation tiles, packed index tiles; no multicast), warp 1 = MMA issuer
// and TMEM owner, warps 2..17 = expanders and, behind the first weight stages of the next tile, the epilogue.
// Every mbarrier wait is bounded (status word + CTA-wide abort flag).
//
// What bounds it: at 384 tokens the tensor cores and what feeds them (per K block 1536 clocks of MMAs; in shared memory
// 683 of gathers, 768 of operand reads, 384 of arriving tiles), at the clock the power limit leaves; at up to 256
// the expanders, 0.5 us per K block.  They gather AFTER the wait for their weight stage: gathering ahead of it, warps
// that had time took the shared-memory banks from those that were waited for (0.65 us per K block).  Pairs of CTAs
// (cta_group::2, half of the operand reads each) were no faster at 384 tokens and slower below.  GEMM alone, 8,192
// tokens: 2048 -> 6144 159 -> 144 us, 1024 -> 4096 69 -> 55; 1,024 tokens: 6144 -> 2048 36 -> 29, 2048 -> 2048 16 -> 13
// (before: one tile per CTA).
//
// Stands in for the reference's decode-to-8-bit + 8-bit GEMM pair at batched sizes
// (a8_joint_pair_r1.py:38-127,374; perrow_a8_candidate_r3.py:56-69) and for its
// decode-in-mainloop GEMM (codebook_cutlass_kernel.cu:234-583).
#include <cuda.h>
#include <math.h>

#include "common.cuh"
#include "umma.cuh"
#include "tmem_weights.cuh"

namespace sacq {

namespace {

using namespace umma;
using namespace tmemw;

constexpr int kBK = 128;             // e4m3 bytes per K block (one 128-byte swizzle row)
constexpr int kMaxActStages = 6;
constexpr int kMaxWStages = 4;
constexpr int kWCols = kBK / 2;      // TMEM columns of a weight stage: kBK / 4 high + kBK / 4 low
struct TmemParams {
  const uint8_t* cb_hilo;       // [C][2][D] e4m3
  const uint16_t* scales;       // bf16 [N]
  const uint16_t* bias;         // bf16 [N] or null
  const float* act_scale;       // [M]
  int* status;
  TmemOut out;
  int K, C;
  TilePlan plan;
  int act_stages;               // shared-memory activation stages, 2..kMaxActStages
  float out_mul;                // 2^-cb8_exp_shift
};

struct TmemLayout {
  uint32_t act_off, act_stage, stg_off, idx_off, idx_slot, cb_off, sw_off, bias_off, sa_off, bar_off, misc_off, total;
};

__host__ __device__ inline TmemLayout tmem_layout(int tok, int act_stages, int sb_bytes, int cb_bytes) {
  TmemLayout L;
  L.act_off = 0;
  L.act_stage = (uint32_t)(tok * kBK);
  L.stg_off = (uint32_t)act_stages * L.act_stage;
  L.idx_off = L.stg_off + epi_staging(tok);
  L.idx_slot = (uint32_t)(kRows * sb_bytes);
  L.cb_off = (L.idx_off + 2 * L.idx_slot + 127) & ~127u;
  L.sw_off = L.cb_off + (uint32_t)((cb_bytes + 127) & ~127);
  L.bias_off = L.sw_off + 2 * kRows * 4;             // two of each: a tile's are set up while the last one's are read
  L.sa_off = L.bias_off + 2 * kRows * 4;
  L.bar_off = L.sa_off + 2 * kMaxTok * 4;
  L.misc_off = L.bar_off + 32 * 8;
  L.total = L.misc_off + 64;
  return L;
}

// NIDX consecutive BITS-wide fields starting at field `first` (a multiple of NIDX) of a
// little-endian stream that begins at the 4-byte aligned address `base`.
template <int BITS, int NIDX>
__device__ __forceinline__ void load_fields_w(const uint8_t* base, int first, uint32_t (&out)[NIDX]) {
  constexpr int kBits = BITS * NIDX;
  constexpr uint32_t kMask = (1u << BITS) - 1u;
  if constexpr (kBits % 32 == 0) {
    constexpr int NW = kBits / 32;
    const uint32_t* w32 = reinterpret_cast<const uint32_t*>(base) + first * BITS / 32;
    uint32_t w[NW];
#pragma unroll
    for (int j = 0; j < NW; ++j) w[j] = w32[j];
#pragma unroll
    for (int j = 0; j < NIDX; ++j) {
      const int bit = j * BITS, word = bit >> 5, off = bit & 31;
      out[j] = (off + BITS <= 32) ? ((w[word] >> off) & kMask)
                                  : (__funnelshift_r(w[word], w[word + 1 < NW ? word + 1 : word], off) & kMask);
    }
  } else {
    // a window of at most 48 bits at a 16-bit aligned offset: two words (the second may belong to
    // the next row of the index tile; it is read, not used)
    static_assert(kBits <= 48, "unaligned windows must fit 64 bits after a 16-bit offset");
    const uint32_t* w32 = reinterpret_cast<const uint32_t*>(base);
    const int start = first * BITS;
    const uint64_t v = (((uint64_t)w32[(start >> 5) + 1] << 32) | w32[start >> 5]) >> (start & 31);
#pragma unroll
    for (int j = 0; j < NIDX; ++j) out[j] = (uint32_t)(v >> (j * BITS)) & kMask;
  }
}

// D in {4, 8}; BITS in {8, 12, 16}; CB_SMEM: the high/low codebook is staged in shared memory, else (a
// table too large for it: 65,536 entries) gathered from global memory, where it stays L2-resident.
// grid = workers.
template <int D, int BITS, bool CB_SMEM>
__global__ void __launch_bounds__(kCtaThreads, 1)
large_m_tmem_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_idx,
                    const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ BcastMaps tmap_bc,
                    const __grid_constant__ TmemParams p) {
  constexpr int IDX_PER_KB = kBK / D;                 // indices per row per K block
  constexpr int KB_BYTES = IDX_PER_KB * BITS / 8;     // index bytes per row per K block
  constexpr int SB_BYTES = 2 * KB_BYTES;              // ... per super block (two K blocks): multiple of 16
  constexpr int CW_BYTES = 2 * D;                     // hi + lo bytes per codeword
  constexpr int WQ = kBK / 16;                        // 32-bit words a thread writes per half
  constexpr int IPT = (kBK / D) / 4;                  // indices per expander thread per weight stage (a quarter row)
  constexpr uint32_t kTmemCols = 512;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const TmemLayout L = tmem_layout(p.plan.tok, p.act_stages, SB_BYTES, CB_SMEM ? p.C * CW_BYTES : 0);

  // barrier indices
  constexpr int ACT_FULL = 0, ACT_EMPTY = kMaxActStages, W_FULL = 2 * kMaxActStages, W_EMPTY = W_FULL + kMaxWStages,
                IDX_FULL = W_EMPTY + kMaxWStages, IDX_EMPTY = IDX_FULL + 2, ACC_FULL = IDX_FULL + 4, ACC_EMPTY = IDX_FULL + 5, CB_FULL = IDX_FULL + 6;
  static_assert(CB_FULL < 32, "barrier region");
  const uint32_t bars = base + L.bar_off;
  auto bar = [&](int i) { return bars + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L.misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L.misc_off + 8);

  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int worker = (int)blockIdx.x;
  const int num_kb = p.K / kBK;
  const int act_stages = p.act_stages;
  const int w_stages = min(kMaxWStages, ((int)kTmemCols - p.plan.tok) / kWCols);
  const TileWalk walk(p.plan, worker);
  const int items = walk.items;
  auto tile = [&](int t, int& n0, int& m0, int& tok) { walk.tile(p.plan, worker, t, n0, m0, tok); };
  const uint32_t cb_bytes = (uint32_t)(p.C * CW_BYTES);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxActStages; ++i) {
      mbar_init(bar(ACT_FULL + i), 1);
      mbar_init(bar(ACT_EMPTY + i), 1);
    }
    for (int i = 0; i < kMaxWStages; ++i) {
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
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == 0) {
    __syncwarp();
    if (elect_one()) {                                // constant operands: their copies start before anything else
      if constexpr (CB_SMEM) {
        mbar_arrive_expect_tx(bar(CB_FULL), cb_bytes);
        bulk_load(base + L.cb_off, p.cb_hilo, cb_bytes, bar(CB_FULL));
      }
      prefetch_tensormap(&tmap_a);
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
    int st = 0, sb = 0;                               // index super blocks: counted over all tiles
    uint32_t free_parity = 1;
    bool ok = true;
    for (int t = 0; t < items && ok; ++t) {
      int n0, m0, tok;
      tile(t, n0, m0, tok);
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        if ((kb & 1) == 0) {
          const int slot = sb & 1;
          ok = mbar_wait_warp(bar(IDX_EMPTY + slot), ((sb >> 1) & 1) ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (elect_one()) {
            mbar_arrive_expect_tx(bar(IDX_FULL + slot), kRows * SB_BYTES);
            tma_load_2d(base + L.idx_off + slot * L.idx_slot, &tmap_idx, (kb >> 1) * SB_BYTES, n0, bar(IDX_FULL + slot));
          }
          ++sb;
          if (t == 0 && kb == 0) asm volatile("griddepcontrol.wait;" ::: "memory");   // activations: from the kernel in front
        }
        ok = mbar_wait_warp(bar(ACT_EMPTY + st), free_parity, abort_flag, p.status);
        if (!ok) break;
        const uint32_t dst = base + L.act_off + st * L.act_stage;
        if (elect_one()) mbar_arrive_expect_tx(bar(ACT_FULL + st), (uint32_t)(tok * kBK));
        for (int b = 0; b < tok; b += p.plan.box)
          if (elect_one()) tma_load_2d(dst + (uint32_t)(b * kBK), &tmap_a, kb * kBK, m0 + b, bar(ACT_FULL + st));
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
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = mbar_wait_warp(bar(ACT_FULL + st), act_parity, abort_flag, p.status) &&
             mbar_wait_warp(bar(W_FULL + ws), w_parity, abort_flag, p.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t act_addr = base + L.act_off + st * L.act_stage;
        const uint64_t b0 = make_smem_desc(act_addr), b1 = make_smem_desc(act_addr + part * kBK);
        const uint32_t w_col = tmem_base + (uint32_t)(kTmemCols - (ws + 1) * kWCols);
#pragma unroll
        for (int ks = 0; ks < kBK / 32; ++ks) {
          const uint64_t adv = (uint64_t)((ks * 32) >> 4);
#pragma unroll
          for (int lo = 0; lo < 2; ++lo) {
            const uint32_t a_tmem = w_col + (uint32_t)(lo * (kWCols / 2) + ks * 8);
            const uint32_t acc = (kb | ks | lo) != 0;
            if (elect_one()) umma_f8_ts(tmem_base, a_tmem, b0 + adv, idesc, acc);
            if (mmas == 2 && elect_one()) umma_f8_ts(tmem_base + part, a_tmem, b1 + adv, idesc, acc);
          }
        }
        if (elect_one()) umma_commit(bar(ACT_EMPTY + st));
        if (elect_one()) umma_commit(bar(W_EMPTY + ws));
        if (++st == act_stages) { st = 0; act_parity ^= 1; }
        if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
      }
      if (ok && elect_one()) umma_commit(bar(ACC_FULL));
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ expanders, then epilogue
    const int et = threadIdx.x - 64;                 // 0..511
    const int quarter = warp & 3;                    // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;             // weight row of the tile = TMEM lane
    const int kpart = (warp - 2) >> 2;               // which 32 bytes of the 128-byte K block (0..3)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint8_t* cbs = CB_SMEM ? sm + L.cb_off : p.cb_hilo;
    bool ok = CB_SMEM ? mbar_wait_warp(bar(CB_FULL), 0, abort_flag, p.status) : true;
    // the codewords of the thread's quarter of the g-th K block, counted over all tiles: WQ words of high halves, WQ of low
    auto gather = [&](int g, uint32_t (&hi)[WQ], uint32_t (&lo)[WQ]) {
      const int sb = g >> 1, slot = sb & 1;           // K is a multiple of two blocks
      if (!mbar_wait_warp(bar(IDX_FULL + slot), (sb >> 1) & 1, abort_flag, p.status)) return false;
      uint32_t idx[IPT];
      load_fields_w<BITS, IPT>(sm + L.idx_off + slot * L.idx_slot + row * SB_BYTES + (g & 1) * KB_BYTES,
                               kpart * IPT, idx);
      if constexpr (D == 8) {
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
          const uint4 c = CB_SMEM ? *reinterpret_cast<const uint4*>(cbs + (size_t)idx[j] * 16)
                                  : __ldg(reinterpret_cast<const uint4*>(cbs + (size_t)idx[j] * 16));
          hi[2 * j] = c.x; hi[2 * j + 1] = c.y;
          lo[2 * j] = c.z; lo[2 * j + 1] = c.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
          const uint2 c = CB_SMEM ? *reinterpret_cast<const uint2*>(cbs + (size_t)idx[j] * 8)
                                  : __ldg(reinterpret_cast<const uint2*>(cbs + (size_t)idx[j] * 8));
          hi[j] = c.x;
          lo[j] = c.y;
        }
      }
      return true;
    };
    int ws = 0;
    uint32_t w_parity = 1;
    const int blocks = items * num_kb;
    // A tile's epilogue runs behind the first weight stages of the next tile, all but one of which are free before the
    // tile's last MMA ends: the tensor cores find them ready when the accumulators have been read.
    const int ahead = min(w_stages - 1, num_kb);
    int epi = 0, due = num_kb + ahead;                // the next epilogue, and behind how many blocks
    uint32_t hi[WQ], lo[WQ];
    for (int g = 0; g < blocks + ahead && ok; ++g) {
      if (g < blocks) {
        ok = mbar_wait_warp(bar(W_EMPTY + ws), w_parity, abort_flag, p.status);
        if (!ok) break;
        tc_fence_after();                              // the MMAs that read this stage are complete
        ok = gather(g, hi, lo);
        if (!ok) break;
        // the thread's quarter of the stage's k: WQ columns of the high half, WQ of the low half
        const uint32_t w_addr = lane_addr + (uint32_t)(kTmemCols - (ws + 1) * kWCols + kpart * WQ);
        tmem_st_32x8(w_addr, hi);
        tmem_st_32x8(w_addr + (uint32_t)(kWCols / 2), lo);
        if ((g & 1) == 1 && lane == 0) mbar_arrive(bar(IDX_EMPTY + ((g >> 1) & 1)));
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(W_FULL + ws));
        if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
      }
      if (g + 1 != due) continue;
      // ---- epilogue
      int n0, m0, tok;
      tile(epi, n0, m0, tok);
      float* sw = reinterpret_cast<float*>(sm + L.sw_off) + (epi & 1) * kRows;
      float* bias = reinterpret_cast<float*>(sm + L.bias_off) + (epi & 1) * kRows;
      float* sa = reinterpret_cast<float*>(sm + L.sa_off) + (epi & 1) * kMaxTok;
      if (et < kRows) {
        const int n = min(n0 + et, p.out.N - 1);
        sw[et] = bf16_bits_to_float(__ldg(p.scales + n)) * p.out_mul;
        bias[et] = p.bias ? bf16_bits_to_float(__ldg(p.bias + n)) : 0.f;
      }
      asm volatile("griddepcontrol.wait;" ::: "memory");   // the token scales; the kernel in front has long gone
      if (et < tok) sa[et] = m0 + et < p.out.M ? __ldg(p.act_scale + m0 + et) : 0.f;
      ok = mbar_wait_warp(bar(ACC_FULL), (uint32_t)epi & 1u, abort_flag, p.status);
      ok = xall(ok);                                  // also: the scales are in place
      if (!ok) break;
      tc_fence_after();
      tile_epilogue(p.out, &tmap_y, tmap_bc.m, lane_addr, quarter, kpart, tok, sa, sw, bias, sm + L.stg_off, m0, n0,
                        bar(ACC_EMPTY));
      ++epi;
      due += num_kb;
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

int sb_bytes_of(const sacq_layer* L) { return 2 * (kBK / L->d.vector_dim) * L->d.index_bits / 8; }

// Shared memory of a launch; the request is padded above half an SM's capacity so that two CTAs
// (each of which takes all 512 TMEM columns) never share an SM.
size_t smem_request(const TmemLayout& lay) {
  const size_t need = lay.total + 1024;
  return need < 120 * 1024 ? 120 * 1024 : need;
}

// Codebooks up to 64 KB (high + low halves) are staged in shared memory, larger ones gathered from global memory.
bool cb_in_smem(const sacq_layer* L) { return (size_t)L->cb_entries * L->d.vector_dim * 2 <= 64 * 1024; }

// Activation stages: as many as fit.  Gathers from global memory need the rest of the SM's memory as L1 (a line for every
// miss in flight): with 227 KB taken, 2048 -> 6144 with 65,536 codewords took 46 us at 1,024 tokens, with 164 KB 29.
int pick_act_stages(const sacq_layer* L, int tok) {
  const int cb_bytes = cb_in_smem(L) ? L->cb_entries * L->d.vector_dim * 2 : 0;
  const uint32_t most = (cb_in_smem(L) ? 227 : 164) * 1024;
  for (int st = kMaxActStages; st >= 2; --st)
    if (tmem_layout(tok, st, sb_bytes_of(L), cb_bytes).total + 1024 <= most) return st;
  return tmem_layout(tok, 2, sb_bytes_of(L), cb_bytes).total + 1024 <= 227 * 1024 ? 2 : 0;
}

template <int D, int BITS, bool CB_SMEM>
cudaError_t launch_cb(const CUtensorMap& ta, const CUtensorMap& ti, const CUtensorMap& ty, const BcastMaps& tb,
                      const TmemParams& p, dim3 grid, size_t smem, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(large_m_tmem_kernel<D, BITS, CB_SMEM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         227 * 1024);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kCtaThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, large_m_tmem_kernel<D, BITS, CB_SMEM>, ta, ti, ty, tb, p);
}

template <int D, int BITS>
cudaError_t launch_db(const CUtensorMap& ta, const CUtensorMap& ti, const CUtensorMap& ty, const BcastMaps& tb,
                      const TmemParams& p, bool cb_smem, dim3 grid, size_t smem, cudaStream_t s) {
  return cb_smem ? launch_cb<D, BITS, true>(ta, ti, ty, tb, p, grid, smem, s)
                 : launch_cb<D, BITS, false>(ta, ti, ty, tb, p, grid, smem, s);
}

// Time of a tile (us), fitted to 2048 -> 6144, 2048 -> 2048, 6144 -> 2048 and 1024 -> 4096 at 1,024 - 8,192 tokens.
double tile_us(const sacq_layer* L, int tok) {
  const double least = cb_in_smem(L) ? (L->d.vector_dim == 8 ? 0.52 : 0.65) : 11.5 / L->d.vector_dim;
  const double block = 0.0026 * tok > least ? 0.0026 * tok : least;
  return 2.3 + 0.0026 * tok + (double)L->d.in_features / kBK * block;
}

}  // namespace

bool large_m_tmem_supported(const sacq_layer* L) {
  const sacq_layer_desc& d = L->d;
  if (d.vector_dim != 8 && d.vector_dim != 4) return false;
  if (d.index_bits != 8 && d.index_bits != 12 && d.index_bits != 16) return false;
  if (!L->rows_16b_aligned) return false;
  if (d.in_features % (2 * kBK) != 0) return false;
  if (L->num_groups != 1 || has_shift(L)) return false;
  if (((size_t)L->cb_entries * d.vector_dim * 2) % 16 != 0) return false;
  return pick_act_stages(L, kMaxTok) >= 2;
}

double large_m_tmem_us(const sacq_layer* L, int64_t M) {
  TilePlan p;
  double us;
  return plan_tiles(L, M, tile_us, 0, &p, &us) ? us : 1e30;
}

int launch_large_m_tmem(const sacq_layer* L, const void* q, const float* scale, int64_t M, void* y, int64_t ldy,
                        cudaStream_t s, const void* residual, int64_t ldr, const BcastDst* bc, int nt_force) {
  const sacq_layer_desc& d = L->d;
  if (!large_m_tmem_supported(L)) return set_error(SACQ_ERR_UNSUPPORTED, "TMEM-weight kernel cannot run this layer geometry");
  if (M <= 0 || d.out_features == 0) return SACQ_OK;
  if (M > (1 << 30)) return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld too large", (long long)M);
  if (reinterpret_cast<uintptr_t>(q) % 16 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "quantized activations must be 16-byte aligned");
  TmemParams p{};
  if (!plan_tiles(L, M, tile_us, kBM * nt_force, &p.plan))
    return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld: too many tiles", (long long)M);
  const int tok = p.plan.tok;
  const bool cb_smem = cb_in_smem(L);
  const int act_stages = pick_act_stages(L, tok);
  CUtensorMap ta;
  {
    const int rc = encode_bytes_2d(&ta, q, (uint64_t)d.in_features, (uint64_t)M, (uint64_t)d.in_features, kBK, p.plan.box,
                                   CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != SACQ_OK) return rc;
  }
  const CUtensorMap* ti = nullptr;
  {
    const int rc = large_m_index_map(L, &ti);
    if (rc != SACQ_OK) return rc;
  }
  CUtensorMap ty = ta;                                // a valid map is passed either way
  BcastMaps tb = {};
  int rc = tile_output(L, M, y, ldy, residual, ldr, bc, &p.out, &ty, &tb);
  if (rc != SACQ_OK) return rc;
  p.cb_hilo = L->cb_hilo;
  p.scales = static_cast<const uint16_t*>(d.scales);
  p.bias = static_cast<const uint16_t*>(d.bias);
  p.act_scale = scale;
  p.status = L->d_status;
  p.K = (int)d.in_features; p.C = L->cb_entries;
  p.act_stages = act_stages;
  p.out_mul = ldexpf(1.f, -L->cb8_exp_shift);
  const TmemLayout lay = tmem_layout(tok, act_stages, sb_bytes_of(L), cb_smem ? L->cb_entries * d.vector_dim * 2 : 0);
  const size_t smem = smem_request(lay);
  const dim3 grid((unsigned)p.plan.workers);
  cudaError_t e;
  const int D = d.vector_dim, B = d.index_bits;
  if (D == 8 && B == 12) e = launch_db<8, 12>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  else if (D == 8 && B == 8) e = launch_db<8, 8>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  else if (D == 8 && B == 16) e = launch_db<8, 16>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  else if (D == 4 && B == 12) e = launch_db<4, 12>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  else if (D == 4 && B == 8) e = launch_db<4, 8>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  else e = launch_db<4, 16>(ta, *ti, ty, tb, p, cb_smem, grid, smem, s);
  count_launch();
  if (e != cudaSuccess) return cuda_fail(e, "TMEM-weight large-M launch");
  return SACQ_OK;
}

}  // namespace sacq
