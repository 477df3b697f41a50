// Shared pieces of the tensor-core kernels that keep the expanded weights in tensor memory
// (linear_large_m_tmem.cu, linear_large_m_tmem_grouped.cu): thread layout, PTX wrappers for
// tcgen05.mma with the A operand in TMEM, tcgen05.st, tiled bulk stores, and the epilogue that
// transposes the accumulator (lane = weight row, column = token) into y.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "encode.cuh"
#include "umma.cuh"

namespace sacq {
namespace tmemw {

using namespace umma;

constexpr int kRows = 128;           // weight rows per CTA = TMEM lanes
constexpr int kXWarps = 16;                  // expander warps: four per TMEM lane quarter
constexpr int kXThreads = kXWarps * 32;
constexpr int kCtaThreads = 64 + kXThreads;  // + TMA producer warp + MMA issuer warp

__device__ __forceinline__ void xbarrier() { asm volatile("bar.sync 1, %0;" ::"n"(kXThreads) : "memory"); }
// AND of a predicate over the expander threads (named barrier 1).
__device__ __forceinline__ bool xall(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "barrier.cta.red.and.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(kXThreads)
      : "memory");
  return r != 0;
}
// Tiled bulk store shared -> global (the tile is clipped at the tensor's edges).
__device__ __forceinline__ void tma_store_2d_issue(const CUtensorMap* map, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(x), "r"(y), "r"(src)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}


// D[tmem] (+)= A[tmem] * B[smem desc], e4m3 x e4m3 -> fp32; A = 128 lanes x 8 columns (32 bytes per lane).
__device__ __forceinline__ void umma_f8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 8 consecutive 32-bit columns of the warp's TMEM lane quarter, one lane per thread.
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }


// kind::f16 twin: fp16 x fp16 -> fp32; A = 128 lanes x 8 columns (16 halves per lane).
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// kind::i8 twin: int8 x int8 -> int32; A = 128 lanes x 8 columns (32 bytes per lane).
__device__ __forceinline__ void umma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Where a kernel's result goes.
struct TmemOut {
  uint16_t* y;                  // bf16 [M, ldy]
  int64_t ldy;
  const uint16_t* residual;     // bf16 [M, ldr] added to the rounded output, or null
  int64_t ldr;
  int n_bc;                     // further copies of the output (peer GPUs' buffers), same pitch as y
  uint16_t* ybc[kMaxBcast];
  int M, N;
  int y_tma;                    // y (and every peer copy) takes tiled bulk stores (aligned, no residual)
};

// Tensor maps over the peer GPUs' copies of the output (the column split's exchange): the same
// [M][N] view as y's map, one per peer.  Plain tiled stores into peer memory, no multicast.
struct BcastMaps {
  CUtensorMap m[kMaxBcast];
};

// ---- persistent tiles ------------------------------------------------------------------------------------

constexpr int kMaxTok = 384;         // tokens of a tile = accumulator columns

// The tiles of a call: `full` = `row_tiles` x the whole tiles of `tok` tokens, then `row_tiles` of `rem` tokens (0: none)
// at token `rem_m0`.  Worker w takes the full tiles w, w + workers, ...; a worker from `rem_first` on, every
// (workers - rem_first)-th of the others.
struct TilePlan {
  int tok, rem, rem_m0, rem_first, full, row_tiles, workers;
  int box;                      // tokens of one activation copy
};

// One worker's walk through them, whole tiles first.
struct TileWalk {
  int n_full, items, rem0, rem_step;
  __device__ __forceinline__ TileWalk(const TilePlan& p, int worker) {
    n_full = p.full > worker ? (p.full - worker + p.workers - 1) / p.workers : 0;
    rem_step = p.workers - p.rem_first;
    rem0 = worker - p.rem_first;
    items = n_full + (p.rem > 0 && rem0 >= 0 && rem0 < p.row_tiles ? (p.row_tiles - rem0 + rem_step - 1) / rem_step : 0);
  }
  __device__ __forceinline__ void tile(const TilePlan& p, int worker, int t, int& n0, int& m0, int& tok) const {
    int r;
    if (t < n_full) {
      const int i = worker + t * p.workers;
      r = i % p.row_tiles;
      m0 = i / p.row_tiles * p.tok;
      tok = p.tok;
    } else {
      r = rem0 + (t - n_full) * rem_step;
      m0 = p.rem_m0;
      tok = p.rem;
    }
    n0 = r * kRows;
  }
};

// 16 lanes x 32 consecutive fp32 columns, as four 16 x 8 fragments: registers 4 j + 0, 1 = lane (thread / 4), columns
// 8 j + 2 (thread % 4) + 0, 1; registers 4 j + 2, 3 = lane (thread / 4) + 8.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Four 8 x 8 tiles of 16-bit elements, each stored transposed; thread l gives the row address l % 8 of tile l / 8.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared::cta.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

constexpr int kWarpTile = 32 * 64;                    // a warp's staged output: 32 tokens x 32 weight rows, bf16
// One per expander warp that has tokens to store.
__host__ __device__ constexpr uint32_t epi_staging(int tok) { return (uint32_t)((tok >= 128 ? 4 : (tok + 31) / 32) * 4 * kWarpTile); }

// Epilogue of one tile, run by the expander warps after the accumulator is complete:
//   y[m0 + token, n0 + row] = bf16(fma(sa[token], acc[row][token] * sw[row], bias[row]))
// The accumulator holds y transposed (lane = weight row, column = token).  A warp takes its lane quarter of every
// fourth 32 tokens: fragments whose register pairs are two tokens of one row, packed to bf16 and stored transposed
// into a [32 tokens][32 rows] tile (stmatrix; 64-byte rows, 16-byte units swizzled as SWIZZLE_64B does), which
// leaves by one tiled bulk store, clipped at the edges of y.  No barrier between warps.  With a residual or an
// unaligned y the warp stores the tile itself, four lanes per token.  128 rows x 384 tokens take 2.4 us; with 2-byte
// stores into a tile of the whole CTA and two barriers per 128 tokens they took 3.3.
// `acc_empty` takes one arrival per warp as soon as it has read its accumulators.
__device__ __forceinline__ void tile_epilogue(const TmemOut& o, const CUtensorMap* tmap_y, const CUtensorMap* tmap_bc,
                                              uint32_t lane_addr, int quarter, int kpart, int tok, const float* sa,
                                              const float* sw, const float* bias, uint8_t* stage_base, int m0, int n0, uint32_t acc_empty) {
  const int lane = threadIdx.x & 31;
  const int nw = n0 + quarter * 32;                   // first weight row of the warp
  uint8_t* tile = stage_base + (quarter + 4 * kpart) * kWarpTile;
  const int last = nw < o.N ? min(tok, o.M - m0) - 1 : -1;             // the last token to store, counted from m0
  // the warp's accumulators have been read (or are not wanted): the next tile may overwrite them
  auto release = [&] {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(acc_empty);
  };
  if (kpart * 32 > last) {
    release();
    return;
  }
  uint64_t sw2[4], bs2[4];                            // of the thread's rows lane / 4 + 8 i
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = quarter * 32 + (lane >> 2) + 8 * i;
    sw2[i] = f32x2(sw[r], sw[r]);
    bs2[i] = f32x2(bias[r], bias[r]);
  }
#pragma unroll 1
  for (int c = kpart; c * 32 <= last; c += 4) {
    const int m = m0 + c * 32;
    uint32_t a[16], b[16];
    tmem_ld_16x32(lane_addr + (uint32_t)(c * 32), a);
    tmem_ld_16x32(lane_addr + (16u << 16) + (uint32_t)(c * 32), b);
    uint64_t s2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = *reinterpret_cast<const float2*>(sa + c * 32 + 8 * j + 2 * (lane & 3));
      s2[j] = f32x2(v.x, v.y);
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if ((c + 4) * 32 > last) release();
    tma_store_wait_read<0>();                         // the store before this one has read the tile
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t* r = i < 2 ? a : b;
        const int at = 4 * j + 2 * (i & 1);
        float lo, hi;
        halves_of(fma2(s2[j], mul2(f32x2(__uint_as_float(r[at]), __uint_as_float(r[at + 1])), sw2[i]), bs2[i]), lo, hi);
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        w[i] = *reinterpret_cast<const uint32_t*>(&v);
      }
      const int t = 8 * j + (lane & 7);               // token whose 16 bytes of rows 8 (lane / 8) .. + 7 the thread addresses
      stmatrix_x4_trans(smem_u32(tile) + (uint32_t)(t * 64 + (((lane >> 3) ^ ((t >> 1) & 3)) * 16)), w[0], w[1], w[2], w[3]);
    }
    if (o.y_tma) {
      fence_proxy_async();                            // generic-proxy writes -> visible to the bulk store
      __syncwarp();
      if (lane == 0) {
        // one bulk-store group: the local copy and, in a column split, every peer's copy
        tma_store_2d_issue(tmap_y, nw * 2, m, smem_u32(tile));
        for (int i = 0; i < o.n_bc; ++i) tma_store_2d_issue(tmap_bc + i, nw * 2, m, smem_u32(tile));
        tma_store_commit();
      }
    } else {
      __syncwarp();
      // rows that begin anywhere: an element per lane, so that a store still covers 64 contiguous bytes (16 bytes per lane
      // would take eight 2-byte stores to 32 scattered places: 6,000 tokens, 2048 -> 6137 263 us, now 142 at d = 4)
      const bool odd = o.residual == nullptr && o.n_bc == 0 && ((reinterpret_cast<uintptr_t>(o.y) & 15) != 0 || (o.ldy & 7) != 0);
      if (odd && nw + lane < o.N) {
        uint16_t* out = o.y + (int64_t)m * o.ldy + nw + lane;
        const int n_tok = min(32, o.M - m);
#pragma unroll 8
        for (int t = 0; t < n_tok; ++t)
          out[t * o.ldy] = *reinterpret_cast<const uint16_t*>(tile + t * 64 + (((lane >> 3) ^ ((t >> 1) & 3)) * 16) + (lane & 7) * 2);
      }
#pragma unroll 1
      for (int i = odd ? 4 : 0; i < 4; ++i) {
        const int t = i * 8 + (lane >> 2), ch = lane & 3;
        const int n = nw + ch * 8;
        if (m + t >= o.M || n >= o.N) continue;
        uint4 v = *reinterpret_cast<const uint4*>(tile + t * 64 + ((ch ^ ((t >> 1) & 3)) * 16));
        const int64_t off = (int64_t)(m + t) * o.ldy + n;
        const bool full = n + 8 <= o.N;
        if (o.residual != nullptr) {
          // bf16(bf16(v) + residual): the two roundings of `linear(x) + residual`
          const uint16_t* rp = o.residual + (int64_t)(m + t) * o.ldr + n;
          uint32_t w[4] = {v.x, v.y, v.z, v.w}, r[4] = {0u, 0u, 0u, 0u};
          if (full && (reinterpret_cast<uintptr_t>(rp) & 15) == 0) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(rp));
            r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (n + e < o.N) r[e >> 1] |= (uint32_t)__ldg(rp + e) << (16 * (e & 1));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 x = __floats2bfloat162_rn(
                __fadd_rn(__uint_as_float(w[e] << 16), __uint_as_float(r[e] << 16)),
                __fadd_rn(__uint_as_float(w[e] & 0xffff0000u), __uint_as_float(r[e] & 0xffff0000u)));
            w[e] = *reinterpret_cast<const uint32_t*>(&x);
          }
          v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        for (int i2 = -1; i2 < o.n_bc; ++i2) {
          uint16_t* out = (i2 < 0 ? o.y : o.ybc[i2]) + off;
          if (full && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
            *reinterpret_cast<uint4*>(out) = v;
          } else {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (n + e < o.N) out[e] = (uint16_t)(w[e >> 1] >> (16 * (e & 1)));
          }
        }
      }
    }
    __syncwarp();                                     // the tile may be written again
  }
}

}  // namespace tmemw

// Modelled time (us) of a tile of `tok` tokens; the plan with the shortest modelled time of the busiest worker (with
// `tok_force` > 0, of that width).  false: too many tiles.
typedef double (*TileTime)(const sacq_layer* L, int tok);
bool plan_tiles(const sacq_layer* L, int64_t M, TileTime tile_us, int tok_force, tmemw::TilePlan* p, double* us = nullptr);

// Where a kernel's result goes, and the tensor maps of tile_epilogue's bulk stores (boxes of 32 tokens x 32 rows) over y and
// over the peers' copies of it: they need a 16-byte aligned base and row pitch, and no residual.
int tile_output(const sacq_layer* L, int64_t M, void* y, int64_t ldy, const void* residual, int64_t ldr, const BcastDst* bc,
                tmemw::TmemOut* out, CUtensorMap* ty, tmemw::BcastMaps* tb);

}  // namespace sacq
