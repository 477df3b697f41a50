// Quantized linear for a few dozen to a few hundred tokens (sm_100a): tensor-memory weights, the K
// dimension split over a thread-block cluster.
//   y[m,n] = bf16( s[m] * (sum_k q[m,k] * W[n,k]) + bias[n] )
//
// What bounds these sizes is neither bandwidth nor the tensor pipe but how often a weight is expanded
// and how many SMs share the expansion: a codeword gather costs a fixed share of an SM's shared-memory
// rate (3 gathers per clock), so every token tile that expands the layer again costs the whole layer
// again, and a tile of 128 weight rows x all tokens leaves most SMs without work (2,048 rows are 16
// tiles).  Here a CTA takes 128 weight rows x ALL tokens (up to 384) x one slice of K, so each weight is
// expanded once on the whole device, and the S CTAs of a cluster that share an output tile add their
// fp32 partial sums through distributed shared memory:
//   * warp 0        TMA producer: the slice's packed indices (64 bytes of every row per box, swizzled, or 16 on the deepest
//                   layers: conflict-free reads whatever the index width), the codebook, then the activation tiles;
//   * warp 1        MMA issuer: tcgen05.mma with the weights as the A operand in tensor memory, N = tokens;
//   * warps 2..17   expanders: one weight row and a quarter of every 128-k stage each: index fields ->
//                   codeword gathers -> tcgen05.st.  kSplitHiLo: the e4m3 high and low halves of the
//                   codewords against e4m3 activations (kind::f8f6f4), one scale per row in the epilogue.
//                   kSplitHalf: fp16(codeword x group scale) against activations widened to fp16
//                   (kind::f16): grouped scales, and INT8 activations on any layer.  kSplitHalf2: that product
//                   as two fp16 operands, h = fp16(c s) and fma(c, s, -h), which together are exact; for the
//                   token counts and layers whose other kernel multiplies exact weights.  kSplitInt8 / kSplitFp8:
//                   the 8-bit weight bytes of the two recipes, made here instead of in a pass of their own
//                   over a 1-byte copy of the weights;
//   * reduction     each CTA of a cluster owns a token range of the tile.  Narrow tiles: the others send it their fp32
//                   partial sums, [token][row], and arrive at its mbarrier; wide ones: a CTA puts them into its own
//                   shared memory and its peers fetch theirs behind a cluster barrier.  The owner adds the slices
//                   pairwise and writes y.  (Shared memory crosses a cluster at 20 bytes a clock and SM either way; sent, it
//                   crosses once and without barriers, but holds up the storing warps: 64 tokens, 2048 -> 2048 with the
//                   quantizer 9.1 us fetched, 8.4 sent; 128 tokens, 2048 -> 6144 10.9 / 11.7.)
// A CTA may take several slices, each with accumulator columns of its own: the order in which an output is
// summed stays the same when many tokens leave no use for a cluster.
// A call of few tokens may be this launch alone (QUANT): the tokens' bf16 rows come to shared memory by bulk copies and the
// expander warps quantize them on the way, a warp per token.
// In a row of calls a CTA starts when one of the call before ends, its activations come 4 us later; what it can do until then
// is done ahead: copies, and the weights of up to seven stages.
// Every mbarrier wait is bounded (status word + CTA-wide abort flag); an aborted CTA still reaches every
// cluster barrier, so its peers do too, and stays until they have left.  No cluster multicast.
#include <cuda.h>
#include <math.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "encode.cuh"
#include "host/internal.h"
#include "split_k.cuh"
#include "tmem_weights.cuh"
#include "umma.cuh"

namespace sacq {

namespace {

using namespace umma;
using namespace tmemw;

constexpr int kStageK = 128;          // k per weight stage
constexpr int kMaxAct = 12;           // activation tiles in flight (128 bytes of every token each)
constexpr int kMaxW = 7;              // weight stages in tensor memory
constexpr int kSliceBytes = kRows * 16;
constexpr int kFirstSlices = 8;       // 16-byte index slices of every row that arrive ahead of the codebook
// fp16 forms: K may end in the middle of a stage; its second 64-k tile is then zeros on both sides.
__host__ __device__ constexpr int stages_of(int64_t K) { return (int)((K + kStageK - 1) / kStageK); }
__host__ __device__ constexpr int w_cols(int mode) { return mode == kSplitHalf2 ? 128 : mode >= kSplitInt8 ? 32 : 64; }
constexpr float kHalfPreScale = 4096.f;   // keeps fp16(codeword x scale) far from the subnormals

struct SplitLayer {
  const uint8_t* cb;            // kSplitHiLo: e4m3 [C][2][D]; kSplitHalf, kSplitHalf2: fp16 [C][D]; recipes: bf16 [C][D]
  const uint16_t* scales;       // bf16 [N, num_groups]
  const uint16_t* bias;         // bf16 [N] or null
  uint16_t* y;                  // bf16 [M, ldy]
  int64_t ldy;
  int* status;
  int N;
  float scale_mul;              // kSplitHalf: power of two that brings the scales into the middle of fp16's range
  const float* row_mul;         // kSplitHalf2: [N], the row's power of two (sacq_layer)
  float out_mul;                // power of two that undoes the operands' scaling
};

// mbarriers of a CTA
constexpr int ACT_FULL = 0, ACT_EMPTY = kMaxAct, W_FULL = 2 * kMaxAct, W_EMPTY = W_FULL + kMaxW, IDX_FULL = W_EMPTY + kMaxW,
              CB_FULL = IDX_FULL + 2, ACC_FULL = CB_FULL + 1, RECV = ACC_FULL + 1, X_FULL = RECV + 1, kBarriers = X_FULL + 1;

struct SplitLayout {
  uint32_t idx_off, cb_off, sc_off, recv_off, fixed_off, sa_off, sw_off, bias_off, bar_off, misc_off, total;
};

// What a CTA's start depends on comes first: kernel parameters are read through a cache that is cold in every launch, a miss
// per line.  The layout comes ready from the host, and what the kernel divides by is a power of two: with its divisions a CTA's
// way to its first copy took 0.2 us longer.
struct alignas(64) SplitParams {
  int split, split_shift;       // CTAs per cluster, its logarithm
  int slice_shift;              // ... of the slices of K, split * parts
  int own;                      // owned_tokens(tok, split)
  SplitLayout lay;
  int parts;                    // consecutive slices of K per CTA, each with accumulator columns of its own
  int tok;                      // tokens per CTA (multiple of 16; of 32 above 256)
  int M, K, C, bits, num_groups, group_size;
  int act_stages, max_slices;
  int own_recv;                 // the partial sums of the cluster have shared memory of their own
  uint16_t shift;               // recipes: bf16 bits
  const float* act_scale;       // [M]
  SplitLayer layer[kSplitMaxLayers];
  CUtensorMap idx[kSplitMaxLayers];     // [64 or 16 bytes][128 rows] boxes over the packed rows
  const float* row_scale;       // recipes: [N], the weight bytes' scale (the caller's buffer, not a layer constant)
  const uint16_t* residual;     // bf16 [M, ldr] added to the rounded output, or null
  int64_t ldr;
  int n_bc;                     // further copies of the output (peer GPUs' buffers), same pitch as y
  uint16_t* ybc[kMaxBcast];
  const uint16_t* x;            // QUANT: bf16 [M, x_pitch], instead of q and act_scale
  int64_t x_pitch;
};

// tokens of the tile a rank reduces and writes
__host__ __device__ constexpr int owned_tokens(int tok, int split) { return ((tok + split - 1) / split + 7) & ~7; }

__host__ __device__ constexpr int index_boxes(int slices, int box_shift) { return (slices + (1 << box_shift) - 1) >> box_shift; }

__host__ __device__ inline SplitLayout split_layout(int tok, int split, int act_stages, int slices, int box_shift, int groups,
                                                    int cb_bytes, bool own_recv, int x_bytes = 0) {
  SplitLayout L;
  L.idx_off = (uint32_t)((act_stages * tok * 128 + 1023) & ~1023);
  L.cb_off = L.idx_off + (uint32_t)(index_boxes(slices, box_shift) * (kSliceBytes << box_shift));
  L.sc_off = L.cb_off + (uint32_t)((cb_bytes + 127) & ~127);
  const uint32_t pipe = L.sc_off + (uint32_t)((groups > 0 ? kRows * (groups | 1) * 2 + 127 : 0) & ~127);
  // the partial sums: [source CTA][owned token][row] of a cluster, or of a CTA alone [token][row]
  const uint32_t recv = (uint32_t)((split > 1 ? split * owned_tokens(tok, split) : tok) * kRows * 4);
  L.recv_off = own_recv ? pipe : 0u;
  L.fixed_off = own_recv ? pipe + recv : pipe > recv ? pipe : recv;
  L.sa_off = L.fixed_off;
  L.sw_off = L.sa_off + (uint32_t)(tok * 4);
  L.bias_off = L.sw_off + kRows * 4;
  L.bar_off = L.bias_off + kRows * 4;
  L.misc_off = L.bar_off + kBarriers * 8;
  L.total = L.misc_off + 64;
  if (x_bytes > 0) L.total = ((L.total + 127) & ~127u) + (uint32_t)x_bytes;      // the rows of x come last
  return L;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_address(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_peer(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// Arrival at another CTA's mbarrier, behind this thread's stores into that CTA's shared memory (and those ordered before).
__device__ __forceinline__ void mbar_arrive_peer(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// Acquires, at cluster scope, what the arrivals of a completed phase released.
__device__ __forceinline__ void mbar_acquire_cluster(uint32_t bar, uint32_t parity) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%0], %1;\n\t}"
      ::"r"(bar), "r"(parity)
      : "memory");
}
__device__ __forceinline__ uint4 load_shared(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 load_peer(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Both barriers, by a whole converged warp: one vote where both phases are complete already.
__device__ __forceinline__ bool mbar_wait_two(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, volatile int* abort_flag, int* status) {
  const bool r0 = mbar_try_wait(b0, p0), r1 = mbar_try_wait(b1, p1);
  if (__all_sync(0xffffffffu, r0 && r1)) return true;
  return mbar_wait_warp(b0, p0, abort_flag, status) && mbar_wait_warp(b1, p1, abort_flag, status);
}
// Whether the phase is complete, without waiting; one answer for the warp.
__device__ __forceinline__ bool mbar_test_warp(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return __all_sync(0xffffffffu, done != 0);
}
// 16 accumulator columns of the warp's lane quarter.
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// a + b of two partial sums held as bits: fp32, or int32 (INT, exact).
template <bool INT>
__device__ __forceinline__ uint32_t add_bits(uint32_t a, uint32_t b) {
  return INT ? a + b : __float_as_uint(__uint_as_float(a) + __uint_as_float(b));
}
template <bool INT>
__device__ __forceinline__ uint4 add_bits4(const uint4& a, const uint4& b) {
  return make_uint4(add_bits<INT>(a.x, b.x), add_bits<INT>(a.y, b.y), add_bits<INT>(a.z, b.z), add_bits<INT>(a.w, b.w));
}
// r += 16 accumulator columns.
template <bool INT>
__device__ __forceinline__ void add_columns(uint32_t (&r)[16], uint32_t taddr) {
  uint32_t b[16];
  tmem_ld_16(taddr, b);
#pragma unroll
  for (int j = 0; j < 16; ++j) r[j] = add_bits<INT>(r[j], b[j]);
}

// The packed indices of a thread's row in the boxes, 1 << BOX_SHIFT slices of 16 bytes of every row each.  64 bytes: laid out
// by SWIZZLE_64B, so the slices of eight consecutive rows lie on different banks; 16 bytes: they do as they come.
template <int BOX_SHIFT>
struct IndexRow {
  const uint8_t* at;            // the row's first byte
  uint32_t swizzle;
  __device__ __forceinline__ IndexRow(const uint8_t* boxes, int row)
      : at(boxes + ((row * 16) << BOX_SHIFT)), swizzle(BOX_SHIFT == 2 ? (uint32_t)((row >> 1) & 3) << 4 : 0u) {}
  // The 16-byte slice `s` (warp-uniform).
  __device__ __forceinline__ uint4 slice(int s) const {
    constexpr int kInBox = (1 << BOX_SHIFT) - 1;
    return *reinterpret_cast<const uint4*>(at + (s >> BOX_SHIFT) * (kSliceBytes << BOX_SHIFT) + ((uint32_t)((s & kInBox) << 4) ^ swizzle));
  }
};
// A window of up to 64 bits at bit `bit` of a row; `bit` is warp-uniform, `need` bits of it are used (a slice is only
// read if one of them lies in it).
template <int BOX_SHIFT>
__device__ __forceinline__ uint64_t slice_window(const IndexRow<BOX_SHIFT>& row, int bit, int need) {
  const uint4 a = row.slice(bit >> 7);
  uint4 b = a;
  if ((bit & 127) + need > 128) b = row.slice((bit >> 7) + 1);
  uint32_t lo, mid, hi;
  switch ((bit >> 5) & 3) {
    case 0: lo = a.x; mid = a.y; hi = a.z; break;
    case 1: lo = a.y; mid = a.z; hi = a.w; break;
    case 2: lo = a.z; mid = a.w; hi = b.x; break;
    default: lo = a.w; mid = b.x; hi = b.y; break;
  }
  const uint32_t sh = (uint32_t)(bit & 31);
  return ((uint64_t)__funnelshift_r(mid, hi, sh) << 32) | __funnelshift_r(lo, mid, sh);
}

// Adds the slices of K pairwise, (0 + 1) + (2 + 3) and so on, whichever CTA does it, and writes y: tokens [0, count) of this
// CTA's share, a warp per token, four consecutive outputs per lane.  `part` = this lane's partial sums of token 0 in the CTA's
// own shared memory; those of the other CTAs are `stride` bytes apart, or (PEER) at the same place in theirs.  Everything that
// does not depend on the token is set up once: this loop is bound by instruction issue (with the addresses and alignment tests
// inside it took 0.4 us per token and warp).
template <int S, bool INT, bool PEER>
__device__ __forceinline__ void reduce_tokens(const SplitParams& p, const SplitLayer& lay, int warp, int lane, int count,
                                              int m_first, int n0, uint32_t part, uint32_t stride, const float* sa, float4 sw,
                                              float4 bs) {
  const int n = n0 + lane * 4;
  const int valid = min(4, lay.N - n);
  if (valid <= 0) return;
  uint32_t src[S];
#pragma unroll
  for (int s = 0; s < S; ++s) src[s] = PEER ? peer_address(part, (uint32_t)s) : part + (uint32_t)s * stride;
  uint16_t* y = lay.y + (int64_t)m_first * lay.ldy + n;
  const int64_t ldy = lay.ldy;
  const uint16_t* res = p.residual ? p.residual + (int64_t)m_first * p.ldr + n : nullptr;
  const int64_t ldr = p.ldr;
  const bool vec_y = valid == 4 && (reinterpret_cast<uintptr_t>(y) & 7) == 0 && (ldy & 3) == 0;
  const bool vec_r = valid == 4 && (reinterpret_cast<uintptr_t>(res) & 7) == 0 && (ldr & 3) == 0;
  const bool plain = vec_y && (res == nullptr || vec_r) && p.n_bc == 0;
  const uint2 none = make_uint2(0u, 0u);
  const bool has_bias = lay.bias != nullptr;
#pragma unroll 2
  for (int t = warp; t < count; t += kXWarps) {
    uint4 v[S];
#pragma unroll
    for (int s = 0; s < S; ++s) v[s] = PEER ? load_peer(src[s] + (uint32_t)(t * (kRows * 4))) : load_shared(src[s] + (uint32_t)(t * (kRows * 4)));
#pragma unroll
    for (int w = 1; w < S; w *= 2)
#pragma unroll
      for (int s = 0; s + w < S; s += 2 * w) v[s] = add_bits4<INT>(v[s], v[s + w]);
    const float sc = sa[t];
    auto fin = [&](uint32_t a, float w, float b) {
      const float x = __fmul_rn(INT ? __int2float_rn((int)a) : __uint_as_float(a), w);
      return has_bias ? fmaf(sc, x, b) : __fmul_rn(sc, x);
    };
    const float o0 = fin(v[0].x, sw.x, bs.x), o1 = fin(v[0].y, sw.y, bs.y), o2 = fin(v[0].z, sw.z, bs.z),
                o3 = fin(v[0].w, sw.w, bs.w);
    __nv_bfloat162 lo = __floats2bfloat162_rn(o0, o1), hi = __floats2bfloat162_rn(o2, o3);
    // bf16(bf16(v) + residual): the two roundings of `linear(x) + residual`
    auto add = [](__nv_bfloat162 o, uint32_t r) {
      const uint32_t b = *reinterpret_cast<const uint32_t*>(&o);
      return __floats2bfloat162_rn(__fadd_rn(__uint_as_float(b << 16), __uint_as_float(r << 16)),
                                   __fadd_rn(__uint_as_float(b & 0xffff0000u), __uint_as_float(r & 0xffff0000u)));
    };
    if (plain) {
      if (res != nullptr) {
        const uint2 r = __ldg(reinterpret_cast<const uint2*>(res + t * ldr));
        lo = add(lo, r.x);
        hi = add(hi, r.y);
      }
      *reinterpret_cast<uint2*>(y + t * ldy) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      continue;
    }
    if (res != nullptr) {
      uint2 r = none;
      const uint16_t* rp = res + t * ldr;
      r.x = __ldg(rp);
      if (valid > 1) r.x |= (uint32_t)__ldg(rp + 1) << 16;
      if (valid > 2) r.y = __ldg(rp + 2);
      if (valid > 3) r.y |= (uint32_t)__ldg(rp + 3) << 16;
      lo = add(lo, r.x);
      hi = add(hi, r.y);
    }
    const uint32_t w0 = *reinterpret_cast<const uint32_t*>(&lo), w1 = *reinterpret_cast<const uint32_t*>(&hi);
    for (int c = -1; c < p.n_bc; ++c) {
      uint16_t* out = c < 0 ? y + t * ldy : p.ybc[c] + (int64_t)(m_first + t) * ldy + n;
      if (valid == 4 && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
        *reinterpret_cast<uint2*>(out) = make_uint2(w0, w1);
      } else {
        out[0] = (uint16_t)w0;
        if (valid > 1) out[1] = (uint16_t)(w0 >> 16);
        if (valid > 2) out[2] = (uint16_t)w1;
        if (valid > 3) out[3] = (uint16_t)(w1 >> 16);
      }
    }
  }
}

// One token's row x (bf16, K values in shared memory), quantized as quant_act_kernel does it: the scale to *scale, the bytes of
// 128-byte stages [first, first + stages) to their rows of the SWIZZLE_128B tiles, `tile` bytes apart, as the TMA would put
// them.  A warp per token; row = null: zeros.
__device__ __forceinline__ void quantize_row(const uint4* row, int chunks, int first, int stages, uint8_t* act_row, int tile, int xor_row,
                                             int lane, float* scale) {
  uint32_t mx = 0u;
  if (row != nullptr)
    for (int c = lane; c < chunks; c += 32) {
      const uint4 v = row[c];
      mx = __vmaxu2(__vmaxu2(__vmaxu2(__vmaxu2(mx, v.x & 0x7fff7fffu), v.y & 0x7fff7fffu), v.z & 0x7fff7fffu), v.w & 0x7fff7fffu);
    }
  const RowDivisor d = scale_of<false>(__uint_as_float(warp_max_bits(max(mx << 16, mx & 0xffff0000u))));
  if (lane == 0) *scale = d.s;
  for (int c = lane; c < stages * 16; c += 32) {      // eight values, half of a 16-byte unit
    uint32_t o[2] = {0u, 0u};
    if (row != nullptr) {
      const uint4 v = row[first * 16 + c];
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      encode_pairs<false, 4>(w, d, o);
    }
    *reinterpret_cast<uint2*>(act_row + (c >> 4) * tile + ((((c >> 1) & 7) ^ xor_row) << 4) + (c & 1) * 8) = make_uint2(o[0], o[1]);
  }
}

// grid = (row tiles x split, token tiles, layers), clusters of `split` CTAs along x.
template <int D, int MODE, bool CB_SMEM, int BOX_SHIFT, bool QUANT>
__global__ void __launch_bounds__(kCtaThreads, 1)
split_k_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ SplitParams p) {
  static_assert(!QUANT || MODE == kSplitHiLo, "the kernel quantizes for itself where its activations are e4m3 bytes");
  constexpr uint32_t kTmemCols = 512;
  constexpr int CW_BYTES = 2 * D;
  constexpr bool PAIR = MODE == kSplitHalf2, F16 = MODE == kSplitHalf || PAIR, RECIPE = MODE >= kSplitInt8, INT = MODE == kSplitInt8;
  constexpr int TILES = F16 ? 2 : 1;                  // activation tiles (128 bytes of every token) per weight stage
  constexpr int W_COLS = w_cols(MODE);                // TMEM columns of a weight stage
  const int S = p.split;
  const int n0 = ((int)blockIdx.x >> p.split_shift) * kRows;
  const SplitLayer& lay = p.layer[blockIdx.z];
  if (n0 >= lay.N) return;                            // a narrower sibling: uniform over the cluster
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  const uint32_t cb_bytes = (uint32_t)(p.C * CW_BYTES);
  const SplitLayout& L = p.lay;

  const uint32_t bars = base + L.bar_off;
  auto bar = [&](int i) { return bars + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L.misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L.misc_off + 8);

  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)cluster_rank() : 0;
  const int m0 = blockIdx.y * p.tok;
  const int nkb = stages_of(p.K);
  const int parts = p.parts, slice_shift = p.slice_shift;
  // this CTA's weight stages, and the first one (counted from kb0) of its slice `v`
  const int kb0 = rank * parts * nkb >> slice_shift, kbs = ((rank + 1) * parts * nkb >> slice_shift) - kb0;
  auto part_begin = [&](int v) { return ((rank * parts + v) * nkb >> slice_shift) - kb0; };
  const int tok = p.tok, acc_cols = tok * parts;
  const bool halves = tok > 256;                      // an instruction (and a TMA box) takes at most 256 tokens
  const int w_stages = min(kMaxW, ((int)kTmemCols - acc_cols) / W_COLS);
  const int act_stages = p.act_stages;
  const int bit_begin = (kb0 * kStageK / D) * p.bits;
  const int slice0 = bit_begin >> 7;

  constexpr int kBoxBytes = kSliceBytes << BOX_SHIFT;
  const int boxes = index_boxes(p.max_slices, BOX_SHIFT), first_boxes = min(boxes, kFirstSlices >> BOX_SHIFT);
  auto load_indices = [&](int from, int to, uint32_t full) {
    mbar_arrive_expect_tx(full, (uint32_t)((to - from) * kBoxBytes));
    for (int i = from; i < to; ++i)
      tma_load_2d(base + L.idx_off + (uint32_t)(i * kBoxBytes), &p.idx[blockIdx.z], (slice0 + (i << BOX_SHIFT)) * 16, n0, full);
  };
  if (warp == 0) {
    // constant operands: their copies start before anything else, those that the first stage needs first
    if (elect_one()) {
      for (int i = 0; i < 3; ++i) mbar_init(bar(IDX_FULL + i), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      fence_proxy_async();
      load_indices(0, first_boxes, bar(IDX_FULL));
      if constexpr (CB_SMEM) {
        mbar_arrive_expect_tx(bar(CB_FULL), cb_bytes);
        bulk_load(base + L.cb_off, lay.cb, cb_bytes, bar(CB_FULL));
      }
    }
  } else if (warp == 2) {
    for (int i = lane; i < kBarriers; i += 32)
      if (i < IDX_FULL || i > CB_FULL) mbar_init(bar(i), (i >= W_FULL && i < W_EMPTY) || (QUANT && i == ACT_FULL) ? kXWarps : i == RECV ? kXWarps * S + 1 : 1);
    if (lane == 0) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  static_assert(CB_FULL == IDX_FULL + 2, "warp 0 makes these three");
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  // Where the partial sums have a place of their own, peers may write theirs there from now on.
  if (S > 1 && p.own_recv) cluster_arrive_relaxed();   // the mbarriers are released by their fence

  bool ok = true;
  if (warp == 0) {
    // ------------------------------------------------------------------ activation tiles, token scales
    if (elect_one()) {
      if (boxes > first_boxes) load_indices(first_boxes, boxes, bar(IDX_FULL + 1));
      prefetch_tensormap(&tmap_a);
    }
    __syncwarp();
    if (S > 1 && p.own_recv) cluster_wait();
    asm volatile("griddepcontrol.wait;" ::: "memory");   // q and the scales come from the kernel in front
    if constexpr (QUANT) {                            // ... or x
      const int rows = min(tok, p.M - m0), row_bytes = p.K * 2;
      if (elect_one()) mbar_arrive_expect_tx(bar(X_FULL), (uint32_t)(rows * row_bytes));
      __syncwarp();
      if (lane < rows) bulk_load(base + L.total - (uint32_t)((tok - lane) * row_bytes), p.x + (int64_t)(m0 + lane) * p.x_pitch, (uint32_t)row_bytes, bar(X_FULL));
      mbar_wait_warp(bar(X_FULL), 0, abort_flag, lay.status);
    }
    float sa[kMaxTok / 32];                           // the token scales: fetched now, put down behind the last copy
#pragma unroll
    for (int i = 0; i < kMaxTok / 32; ++i) {
      const int t = i * 32 + lane;
      sa[i] = !QUANT && t < tok && m0 + t < p.M ? __ldg(p.act_scale + m0 + t) : 0.f;
    }
    int st = 0;
    uint32_t free_parity = 1;
    for (int i = 0; i < (QUANT ? 0 : kbs * TILES); ++i) {
      if (i >= act_stages && !mbar_wait_warp(bar(ACT_EMPTY + st), free_parity, abort_flag, lay.status)) break;
      const uint32_t dst = base + (uint32_t)(st * tok * 128);
      const int x = (kb0 * TILES + i) * 128;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar(ACT_FULL + st), (uint32_t)(tok * 128));
        tma_load_2d(dst, &tmap_a, x, m0, bar(ACT_FULL + st));
        if (halves) tma_load_2d(dst + (uint32_t)(tok / 2 * 128), &tmap_a, x, m0 + tok / 2, bar(ACT_FULL + st));
      }
      if (++st == act_stages) { st = 0; free_parity ^= 1; }
    }
#pragma unroll
    for (int i = 0; i < kMaxTok / 32; ++i)
      if (!QUANT && i * 32 + lane < tok) reinterpret_cast<float*>(sm + L.sa_off)[i * 32 + lane] = sa[i];
    // every copy has landed before the CTA ends (the expanders see to it that none lands on partial sums)
    mbar_wait_warp(bar(IDX_FULL), 0, abort_flag, lay.status);
    if (boxes > first_boxes) mbar_wait_warp(bar(IDX_FULL + 1), 0, abort_flag, lay.status);
    if (CB_SMEM) mbar_wait_warp(bar(CB_FULL), 0, abort_flag, lay.status);
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(RECV));            // the token scales are in place (S > 1 and nothing sent: no one waits)
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc = INT ? make_idesc_i8(halves ? tok / 2 : tok) : make_idesc(halves ? tok / 2 : tok);
    int st = 0, ws = 0;
    uint32_t act_parity = 0, w_parity = 0;
    int part = -1, next_part = 0, begin = 0;          // slice of K, the stage at which the next one begins
    if (S > 1 && p.own_recv) cluster_wait();
    for (int wi = 0; wi < kbs && ok; ++wi) {
      if (wi == next_part) {
        begin = wi;
        next_part = ++part + 1 < parts ? part_begin(part + 1) : kbs;
      }
      const uint32_t w_col = tmem_base + (uint32_t)(acc_cols + ws * W_COLS);
      const uint32_t d_col = tmem_base + (uint32_t)(part * tok);
#pragma unroll
      for (int sub = 0; sub < TILES; ++sub) {
        // QUANT: one barrier for all activation tiles, none of which is filled again
        ok = sub == 0 ? mbar_wait_two(bar(W_FULL + ws), w_parity, bar(QUANT ? ACT_FULL : ACT_FULL + st), QUANT ? 0u : act_parity, abort_flag, lay.status)
                      : mbar_wait_warp(bar(ACT_FULL + st), act_parity, abort_flag, lay.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t act = base + (uint32_t)(st * tok * 128);
        const uint64_t b0 = make_smem_desc(act);
        const uint64_t b1 = make_smem_desc(act + (uint32_t)(tok / 2 * 128));
        const uint32_t fresh = (uint32_t)(((wi - begin) | sub) != 0);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {              // 32 bytes of every token per step
#pragma unroll
          for (int h = 0; h < (MODE == kSplitHiLo || PAIR ? 2 : 1); ++h) {       // high and low halves of the weights
            const uint32_t a = w_col + (F16 ? (uint32_t)(h * 64 + sub * 32 + ks * 8) : (uint32_t)(h * 32 + ks * 8));
            const uint32_t acc = ks == 0 && h == 0 ? fresh : 1u;
            const uint64_t adv = (uint64_t)(ks * 2);
            if (elect_one()) {
              if constexpr (F16) umma_f16_ts(d_col, a, b0 + adv, idesc, acc);
              else if constexpr (INT) umma_i8_ts(d_col, a, b0 + adv, idesc, acc);
              else umma_f8_ts(d_col, a, b0 + adv, idesc, acc);
            }
            if (halves && elect_one()) {
              if constexpr (F16) umma_f16_ts(d_col + (uint32_t)(tok / 2), a, b1 + adv, idesc, acc);
              else if constexpr (INT) umma_i8_ts(d_col + (uint32_t)(tok / 2), a, b1 + adv, idesc, acc);
              else umma_f8_ts(d_col + (uint32_t)(tok / 2), a, b1 + adv, idesc, acc);
            }
          }
        }
        // a stage that is not filled again needs no word that it is free
        if (wi * TILES + sub + act_stages < kbs * TILES && elect_one()) umma_commit(bar(ACT_EMPTY + st));
        if (sub == TILES - 1 && wi + w_stages < kbs && elect_one()) umma_commit(bar(W_EMPTY + ws));
        if (++st == act_stages) { st = 0; act_parity ^= 1; }
      }
      if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
    }
    if (ok && elect_one()) umma_commit(bar(ACC_FULL));
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ expanders
    const int et = threadIdx.x - 64;
    const int quarter = warp & 3;                     // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;
    const int kpart = (warp - 2) >> 2;                // which quarter of a stage's 128 bytes (or of each 64-k tile)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    if (et < kRows) {
      const int n = min(n0 + et, lay.N - 1);
      if constexpr (!RECIPE)
        reinterpret_cast<float*>(sm + L.sw_off)[et] = F16 ? lay.out_mul : bf16_bits_to_float(__ldg(lay.scales + n)) * lay.out_mul;
      reinterpret_cast<float*>(sm + L.bias_off)[et] = lay.bias ? bf16_bits_to_float(__ldg(lay.bias + n)) : 0.f;
    }
    constexpr bool GROUPS = F16 || RECIPE;             // scales enter the weight operand
    const int g_first = GROUPS ? kb0 * kStageK / p.group_size : 0;
    const int g_count = GROUPS ? (min((kb0 + kbs) * kStageK, p.K) - 1) / p.group_size - g_first + 1 : 0;
    const int sc_pitch = g_count | 1;                 // odd: the 32 rows of a warp fall on different banks
    uint16_t* sc = reinterpret_cast<uint16_t*>(sm + L.sc_off);
    if constexpr (GROUPS) {
      for (int i = et; i < kRows * g_count; i += kXThreads) {
        const int r = i / g_count, g = i - r * g_count;
        const int n = min(n0 + r, lay.N - 1);
        const uint16_t v = __ldg(lay.scales + (int64_t)n * p.num_groups + g_first + g);
        // fp16 forms: scale x 2^e, the row's or the layer's power of two, is a bf16 significand with a small exponent: exact in fp16
        const float mul = PAIR ? 1.f / __ldg(lay.row_mul + n) : lay.scale_mul;
        sc[r * sc_pitch + g] = F16 ? __half_as_ushort(__float2half_rn(bf16_bits_to_float(v) * mul)) : v;
      }
    }
    xbarrier();
    const uint8_t* cbs = CB_SMEM ? sm + L.cb_off : lay.cb;
    auto codeword16 = [&](uint32_t i) {
      return CB_SMEM ? *reinterpret_cast<const uint4*>(cbs + i * 16) : __ldg(reinterpret_cast<const uint4*>(cbs) + i);
    };
    auto codeword8 = [&](uint32_t i) {
      return CB_SMEM ? *reinterpret_cast<const uint2*>(cbs + i * 8) : __ldg(reinterpret_cast<const uint2*>(cbs) + i);
    };
    const IndexRow<BOX_SHIFT> rowidx(sm + L.idx_off, row);
    const uint32_t mask = (1u << p.bits) - 1u;
    const int bits = p.bits;
    // One answer per warp: what follows (tcgen05.st, its wait, __syncwarp) is the whole warp's.
    ok = mbar_wait_warp(bar(IDX_FULL), 0, abort_flag, lay.status) &&
         (!CB_SMEM || mbar_wait_warp(bar(CB_FULL), 0, abort_flag, lay.status));
    // The first stage whose indices reach beyond the first boxes.  It is not the very first one: the boxes hold 897 bits of the
    // slice at least, a stage has 512 at most.
    const int late = boxes == first_boxes ? kbs : ((slice0 + kFirstSlices) * 128 - bit_begin) / (kStageK / D * bits);
    int grp = 0, grp_end = GROUPS ? (g_first + 1) * p.group_size - kb0 * kStageK : 0;    // k (in the slice) at which the scale changes
    // One stage's 16 words of this thread.  The next stage's words are gathered before the wait for this
    // stage's tcgen05.st: the gathers, which bound the loop, then never wait for a store's latency.
    // A recipe's row scales are the caller's and may come from the kernel in front; what has been read so far is the layer's.
    if constexpr (RECIPE) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (et < kRows) reinterpret_cast<float*>(sm + L.sw_off)[et] = __ldg(p.row_scale + min(n0 + et, lay.N - 1));   // for the reduction
    }
    const RowWeights rw = row_weights<INT>(RECIPE ? __ldg(p.row_scale + min(n0 + row, lay.N - 1)) : 1.f);
    const __nv_bfloat162 shift2 = __halves2bfloat162(__ushort_as_bfloat16(p.shift), __ushort_as_bfloat16(p.shift));
    // kSplitHalf2: the codewords as they are, and the two 64-k tiles' scales; the products are made at the store.
    auto expand = [&](int wi, uint32_t (&w)[16], __half2 (&sc2)[2]) {
      if constexpr (RECIPE) {
        // 32 weights of this thread's row, 16 at a time: bf16(bf16(c * s) + shift) divided by the row scale and
        // encoded (the arithmetic of decode_rows_kernel in dequant.cu)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          constexpr int IPT = 16 / D;
          const int k = wi * kStageK + kpart * 32 + h * 16;       // in the slice
          const int g = p.num_groups == 1 ? 0 : (kb0 * kStageK + k) / p.group_size - g_first;
          const __nv_bfloat16 s = __ushort_as_bfloat16(sc[row * sc_pitch + g]);
          const uint64_t win = slice_window(rowidx, ((kb0 * kStageK + k) / D) * bits - slice0 * 128, IPT * bits);
          uint32_t pair[8];
#pragma unroll
          for (int j = 0; j < IPT; ++j) {
            const uint32_t i = (uint32_t)(win >> (j * bits)) & mask;
            if constexpr (D == 8) {
              const uint4 v = codeword16(i);
              pair[4 * j] = v.x; pair[4 * j + 1] = v.y; pair[4 * j + 2] = v.z; pair[4 * j + 3] = v.w;
            } else {
              const uint2 v = codeword8(i);
              pair[2 * j] = v.x; pair[2 * j + 1] = v.y;
            }
          }
          encode_weights16<INT>(pair, __halves2bfloat162(s, s), shift2, (p.shift & 0x7fffu) != 0, rw, reinterpret_cast<uint32_t (&)[4]>(w[4 * h]));
        }
      } else if constexpr (F16) {
        constexpr int IPT = 16 / D;                   // indices per thread and 64-k tile
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          if ((kb0 + wi) * kStageK + sub * 64 >= p.K) {
            sc2[sub] = __half2half2(__ushort_as_half(0));
#pragma unroll
            for (int j = 0; j < 8; ++j) w[sub * 8 + j] = 0u;
            continue;
          }
          if (wi * kStageK + sub * 64 >= grp_end) { ++grp; grp_end += p.group_size; }
          const __half2 s2 = __half2half2(__ushort_as_half(sc[row * sc_pitch + grp]));
          sc2[sub] = s2;
          const int bit = (((kb0 + wi) * kStageK + sub * 64 + kpart * 16) / D) * bits - slice0 * 128;
          const uint64_t win = slice_window(rowidx, bit, IPT * bits);
#pragma unroll
          for (int j = 0; j < IPT; ++j) {
            const uint32_t i = (uint32_t)(win >> (j * bits)) & mask;
            uint32_t c[D / 2];
            if constexpr (D == 8) {
              const uint4 v = codeword16(i);
              c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
            } else {
              const uint2 v = codeword8(i);
              c[0] = v.x; c[1] = v.y;
            }
#pragma unroll
            for (int e = 0; e < D / 2; ++e) {
              const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&c[e]), s2);
              w[sub * 8 + j * (D / 2) + e] = PAIR ? c[e] : *reinterpret_cast<const uint32_t*>(&h);
            }
          }
        }
      } else {
        const int bit = (((kb0 + wi) * kStageK + kpart * 32) / D) * bits - slice0 * 128;
#pragma unroll
        for (int v = 0; v < 8 / D; ++v) {             // four indices per window
          const uint64_t win = slice_window(rowidx, bit + v * 4 * bits, 4 * bits);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t i = (uint32_t)(win >> (j * bits)) & mask;
            if constexpr (D == 8) {
              const uint4 c = codeword16(i);
              w[2 * j] = c.x; w[2 * j + 1] = c.y;
              w[8 + 2 * j] = c.z; w[8 + 2 * j + 1] = c.w;
            } else {
              const uint2 c = codeword8(i);
              w[4 * v + j] = c.x;
              w[8 + 4 * v + j] = c.y;
            }
          }
        }
      }
    };
    int ws = 0;
    uint32_t w_parity = 1;
    uint32_t cur[16], nxt[16];
    __half2 cur_s[2], nxt_s[2];
    if (ok) expand(0, cur, cur_s);
    __syncwarp();
    if (S > 1 && p.own_recv) cluster_wait();
    bool quantized = !QUANT;
    for (int wi = 0; wi < kbs + (QUANT ? 1 : 0) && ok; ++wi) {
      if constexpr (QUANT) {
        // The warp's tokens: as soon as their rows have landed, at the latest when nothing is left to expand ahead of the MMAs.
        const bool now = wi >= w_stages || wi == kbs;
        if (!quantized && (now || mbar_test_warp(bar(X_FULL), 0))) {
          if (now) ok = mbar_wait_warp(bar(X_FULL), 0, abort_flag, lay.status);
          if (!ok) break;
          for (int t = warp - 2; t < tok; t += kXWarps)
            quantize_row(m0 + t < p.M ? reinterpret_cast<const uint4*>(sm + L.total - (tok - t) * p.K * 2) : nullptr, p.K >> 3, kb0, kbs,
                         sm + t * 128, tok * 128, t & 7, lane, reinterpret_cast<float*>(sm + L.sa_off) + t);
          fence_proxy_async();                        // the tensor cores read them
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(ACT_FULL));
          quantized = true;
        }
        if (wi == kbs) break;
      }
      if (wi >= w_stages) {
        ok = mbar_wait_warp(bar(W_EMPTY + ws), w_parity, abort_flag, lay.status);
        if (!ok) break;
        tc_fence_after();                             // the MMAs that read this stage are complete
      }
      // two quarters of the stage: high and low halves, or the two 64-k tiles
      const uint32_t w_addr = lane_addr + (uint32_t)(acc_cols + ws * W_COLS + kpart * 8);
      if constexpr (PAIR) {
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const __half2 c = *reinterpret_cast<const __half2*>(&cur[sub * 8 + j]);
            const __half2 h = __hmul2_rn(c, cur_s[sub]), l = __hfma2(c, cur_s[sub], __hneg2(h));
            hi[j] = *reinterpret_cast<const uint32_t*>(&h);
            lo[j] = *reinterpret_cast<const uint32_t*>(&l);
          }
          tmem_st_32x8(w_addr + (uint32_t)(sub * 32), hi);
          tmem_st_32x8(w_addr + (uint32_t)(64 + sub * 32), lo);
        }
      } else {
        tmem_st_32x8(w_addr, reinterpret_cast<const uint32_t (&)[8]>(cur[0]));
        if constexpr (!RECIPE) tmem_st_32x8(w_addr + 32u, reinterpret_cast<const uint32_t (&)[8]>(cur[8]));
      }
      if (wi + 1 == late && late < kbs) ok = mbar_wait_warp(bar(IDX_FULL + 1), 0, abort_flag, lay.status);
      if (wi + 1 < kbs && ok) expand(wi + 1, nxt, nxt_s);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(W_FULL + ws));
      if (++ws == w_stages) { ws = 0; w_parity ^= 1; }
#pragma unroll
      for (int j = 0; j < (RECIPE ? 8 : 16); ++j) cur[j] = nxt[j];
      if constexpr (PAIR) {
        cur_s[0] = nxt_s[0];
        cur_s[1] = nxt_s[1];
      }
    }
    // Every CTA loads as many boxes as the longest slice of K has.  One whose own slice ends in the first of them has not
    // waited for the others yet, and partial sums that are fetched go where those land.
    if (ok && late >= kbs && boxes > first_boxes) ok = mbar_wait_warp(bar(IDX_FULL + 1), 0, abort_flag, lay.status);
    if (ok) ok = mbar_wait_warp(bar(ACC_FULL), 0, abort_flag, lay.status);
  }

  // ---- reduction: the accumulators of the cluster's CTAs -> y.  Every thread takes part in the cluster barrier.
  const int own = p.own;
  const bool send = S > 1 && p.own_recv, fetch = S > 1 && !send;   // fetch: a CTA keeps its partial sums, its peers read them
  if (warp >= 2 && ok) {
    // [token][row] fp32 into the shared memory of the CTA that owns the token, or the own; a warp writes 128 consecutive
    // bytes per token.  (The main loop's last MMA has completed, so every stage has been written and read.)
    const int quarter = warp & 3, row = quarter * 32 + lane, kpart = (warp - 2) >> 2;
    const float row_mul = PAIR ? __ldg(lay.row_mul + min(n0 + row, lay.N - 1)) : 1.f;
    const int tokens = min(tok, p.M - m0);
    tc_fence_after();
    for (int c0 = kpart * 16; c0 < tokens; c0 += 64) {
      const uint32_t at = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
      uint32_t r[16];
      tmem_ld_16(at, r);
      if (parts >= 2) add_columns<INT>(r, at + (uint32_t)tok);
      if (parts == 4) {                               // (0 + 1) + (2 + 3), as the reduction over CTAs adds them
        uint32_t r2[16];
        tmem_ld_16(at + (uint32_t)(2 * tok), r2);
        add_columns<INT>(r2, at + (uint32_t)(3 * tok));
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = add_bits<INT>(r[j], r2[j]);
      }
      if constexpr (PAIR) {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * row_mul);
      }
      if (!send) {
        uint32_t* dst = reinterpret_cast<uint32_t*>(sm) + c0 * kRows + row;
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[j * kRows] = r[j];
        continue;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {                   // eight tokens have one owner
        const int t = c0 + h * 8, owner = t / own;
        const uint32_t dst = base + L.recv_off + (uint32_t)(((rank * own + t - owner * own) * kRows + row) * 4);
        if (owner == rank) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (uint32_t)(j * kRows * 4)), "r"(r[h * 8 + j]) : "memory");
        } else {
          const uint32_t at_owner = peer_address(dst, (uint32_t)owner);
#pragma unroll
          for (int j = 0; j < 8; ++j) store_peer(at_owner + (uint32_t)(j * kRows * 4), r[h * 8 + j]);
        }
      }
    }
    tc_fence_before();
    __syncwarp();
    if (!fetch && lane < S) mbar_arrive_peer(peer_address(bar(RECV), (uint32_t)lane));
  }
  __syncwarp();
  if (fetch) {
    cluster_arrive();
    cluster_wait();
  }
  if (warp >= 2 && ok) {
    if (!fetch) ok = mbar_wait_warp(bar(RECV), 0, abort_flag, lay.status);
    if (ok) {
      if (!fetch) mbar_acquire_cluster(bar(RECV), 0);
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const int first = rank * own;                   // the tokens this CTA writes
      const int count = min(own, min(tok, p.M - m0) - first);
      const float* sa = reinterpret_cast<const float*>(sm + L.sa_off) + first;
      const float4 sw = reinterpret_cast<const float4*>(sm + L.sw_off)[lane];
      const float4 bs = reinterpret_cast<const float4*>(sm + L.bias_off)[lane];
      const uint32_t stride = (uint32_t)(own * kRows * 4);
      const uint32_t part = base + L.recv_off + (uint32_t)(lane * 16) + (send ? 0u : (uint32_t)rank * stride);
      auto reduce = [&](auto slices) {
        constexpr int kS = decltype(slices)::value;
        if (kS > 1 && fetch) reduce_tokens<kS, INT, true>(p, lay, warp - 2, lane, count, m0 + first, n0, part, 0u, sa, sw, bs);
        else reduce_tokens<kS, INT, false>(p, lay, warp - 2, lane, count, m0 + first, n0, part, stride, sa, sw, bs);
      };
      if (S == 1) reduce(std::integral_constant<int, 1>{});
      else if (S == 2) reduce(std::integral_constant<int, 2>{});
      else if (S == 8) reduce(std::integral_constant<int, 8>{});
      else reduce(std::integral_constant<int, 4>{});
    }
  }

  // ---- common exit.  What peers send here has arrived (RECV), but a CTA that gave up may still be written to, and a CTA
  // whose partial sums are fetched may still be read: it stays until its peers have arrived here too (or have left).
  tc_fence_before();
  __syncwarp();
  if (!fetch) __syncthreads();
  if (fetch || (S > 1 && *abort_flag)) {
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace

struct SplitPlan {
  CUtensorMap idx[2];           // boxes of [16 bytes][128 rows] and of [64 bytes][128 rows] over the packed rows
  bool have[2];
};

namespace {

std::atomic<int64_t> g_searches{0};
std::mutex g_split_mutex;       // layers build their index maps on first use, possibly from several host threads

// Boxes of 64 bytes of 128 rows over the packed rows.  (Boxes of 16 bytes, in the order the expanders read them, cost the
// copy engine a clock per 16 bytes: 24 slices of a row took 1.3 us longer to arrive.  They are for layers so deep that what a
// last box of 64 bytes holds beyond the slice of K, up to 6 KB, is the room of a wider token tile.)
int index_map(sacq_layer* L, int box_shift, CUtensorMap* out) {
  std::lock_guard<std::mutex> lock(g_split_mutex);
  if (L->split_plan == nullptr) L->split_plan = new SplitPlan();
  SplitPlan* plan = L->split_plan;
  const int wide = box_shift != 0;
  if (!plan->have[wide]) {
    const uint64_t row_bytes = (uint64_t)(L->row_bits / 8);
    const int rc = encode_bytes_2d(&plan->idx[wide], L->d.packed, row_bytes, (uint64_t)L->d.out_features, row_bytes, 16u << box_shift,
                                   (uint32_t)kRows, wide ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc != SACQ_OK) return rc;
    plan->have[wide] = true;
  }
  *out = plan->idx[wide];
  return SACQ_OK;
}

bool is_f16(SplitMode mode) { return mode == kSplitHalf || mode == kSplitHalf2; }

size_t split_smem(const SplitLayout& l) {
  const size_t need = l.total + 1024 - 128;           // the kernel rounds its start, a multiple of 128, up to one of 1,024
  return need < 116 * 1024 ? 116 * 1024 : need;       // two CTAs (each takes all 512 TMEM columns) never share an SM
}

// Clusters of `split` such CTAs that run at once (a cluster stays within one GPC).
int active_clusters(int split, int num_sms) {
  return split == 8 ? num_sms * 15 / 148 : split == 4 ? num_sms * 33 / 148 : num_sms / split;
}

template <int D, int MODE, bool CB_SMEM, int BOX_SHIFT, bool QUANT = false>
cudaError_t launch_kernel(const CUtensorMap& ta, const SplitParams& p, dim3 grid, size_t smem, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(split_k_kernel<D, MODE, CB_SMEM, BOX_SHIFT, QUANT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kCtaThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.split;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, split_k_kernel<D, MODE, CB_SMEM, BOX_SHIFT, QUANT>, ta, p);
}

template <int D, bool CB_SMEM, int BOX_SHIFT>
cudaError_t launch_mode(SplitMode mode, const CUtensorMap& ta, const SplitParams& p, dim3 grid, size_t smem, cudaStream_t s) {
  switch (mode) {
    case kSplitHiLo:
      if constexpr (BOX_SHIFT == 2)
        if (p.x != nullptr) return launch_kernel<D, kSplitHiLo, CB_SMEM, BOX_SHIFT, true>(ta, p, grid, smem, s);
      return launch_kernel<D, kSplitHiLo, CB_SMEM, BOX_SHIFT>(ta, p, grid, smem, s);
    case kSplitHalf: return launch_kernel<D, kSplitHalf, CB_SMEM, BOX_SHIFT>(ta, p, grid, smem, s);
    case kSplitHalf2: return launch_kernel<D, kSplitHalf2, CB_SMEM, BOX_SHIFT>(ta, p, grid, smem, s);
    case kSplitInt8: return launch_kernel<D, kSplitInt8, CB_SMEM, BOX_SHIFT>(ta, p, grid, smem, s);
    default: return launch_kernel<D, kSplitFp8, CB_SMEM, BOX_SHIFT>(ta, p, grid, smem, s);
  }
}

// Shared memory of the codebook: tables above 64 KB (65,536 entries) are gathered from global memory, where they stay
// in L2.
int codebook_smem(const sacq_layer* L) {
  const int64_t bytes = (int64_t)L->cb_entries * L->d.vector_dim * 2;
  return bytes <= 64 * 1024 ? (int)bytes : 0;
}

// Index slices and scale groups of the largest K slice.
void slice_extent(const sacq_layer* L, int split, int* slices, int* groups) {
  const int nkb = stages_of(L->d.in_features), d = L->d.vector_dim, bits = L->d.index_bits;
  *slices = *groups = 0;
  for (int r = 0; r < split; ++r) {
    const int k0 = r * nkb / split * kStageK;
    const int k1 = r + 1 < split ? (r + 1) * nkb / split * kStageK : (int)L->d.in_features;
    const int n = ((k1 / d * bits + 127) >> 7) - ((k0 / d * bits) >> 7);
    const int g = (k1 - 1) / L->d.group_size - k0 / L->d.group_size + 1;
    if (n > *slices) *slices = n;
    if (g > *groups) *groups = g;
  }
}

// How many slices K is cut into: a function of K alone, so the order in which an output is summed depends
// neither on the number of tokens nor on the layer's width -- a batch gives each of its rows the bytes of a
// smaller call, sibling layers share a launch, and the row shards of a split layer reproduce it.  About 1,024
// of K per CTA: measured at 64 and 300 tokens, two slices are the best or within 10 % of it for K = 1,024 and
// 2,048 on 1,024- to 6,144-row layers, four for K = 4,096 and 6,144 (larger clusters leave SMs idle: 33 clusters
// of 4, 22 of 6, 15 of 8 run at once); eight above, where a slice's indices would no longer fit shared memory.
int slices_for(int64_t K) { return K < 1024 ? 1 : K < 4096 ? 2 : K < 8192 ? 4 : 8; }

// Completes a choice of tokens and slices; false if it does not fit shared memory.  Gathers from global memory need the
// rest of the SM's memory as L1, a line for every miss in flight: beyond 164 KB only what is needed at all (65,536
// codewords: 2048 -> 6144 at 300 tokens 26.4 us with 227 KB taken, 20.6 now; 6144 -> 2048 at 400 38.8 / 27.4).
bool split_fits(const sacq_layer* L, SplitMode mode, SplitChoice* c) {
  const int cb_bytes = codebook_smem(L), groups = mode == kSplitHiLo ? 0 : 1;
  const int cut = c->split == 1 ? 0 : c->split == 2 ? 1 : c->split == 4 ? 2 : 3;
  c->max_slices = L->slice_idx[cut];
  c->max_groups = L->slice_groups[cut];
  const int tiles = (stages_of(L->d.in_features) + c->split - 1) / c->split * (is_f16(mode) ? 2 : 1);
  const size_t most = (cb_bytes > 0 ? 224 : 164) * 1024;
  auto bytes = [&](int stages) {
    return split_smem(split_layout(c->tok, c->split, stages, c->max_slices, c->box_shift, groups * c->max_groups, cb_bytes, c->own_recv));
  };
  const int all = tiles < 2 ? 2 : tiles < kMaxAct ? tiles : kMaxAct;
  c->box_shift = 2;
  if (c->split > 1 && c->tok <= (c->split == 2 ? 96 : 64)) {
    c->own_recv = true;
    for (c->act_stages = all; c->act_stages >= (all < 4 ? all : 4); --c->act_stages)
      if (bytes(c->act_stages) <= most) return true;
  }
  c->own_recv = false;
  for (; c->box_shift >= 0; c->box_shift -= 2) {
    for (c->act_stages = all; c->act_stages > 2; --c->act_stages)
      if (bytes(c->act_stages) <= most) return true;
    if (bytes(2) <= 227 * 1024) return true;
  }
  return false;
}

// Time of one CTA with `tok` tokens and `kbs` weight stages (us): prologue, the slower of expansion, MMAs and
// activation tiles per stage, reduction.
double split_cta_us(int vector_dim, SplitMode mode, bool cb_smem, int tok, int kbs, int split) {
  double stage = mode >= kSplitInt8 ? 0.75 : vector_dim == 8 ? 0.48 : 0.6;
  if (!cb_smem) stage = 8.0 / vector_dim;             // gathers from L2
  const double mma = (mode == kSplitHalf2 ? 0.0042 : 0.002) * tok;
  if (mma > stage) stage = mma;
  return 2.5 + kbs * stage + 0.015 * tok + (split > 1 ? 0.8 : 0.0);
}

// What the kernel's index arithmetic needs of a layer.
bool takes_layer(const sacq_layer* L, SplitMode mode) {
  const sacq_layer_desc& d = L->d;
  if (d.vector_dim != 8 && d.vector_dim != 4) return false;
  if (d.index_bits > 16 || !L->rows_16b_aligned || d.in_features % (is_f16(mode) ? 64 : kStageK) != 0) return false;
  if (mode < kSplitInt8 && has_shift(L)) return false;
  if (mode == kSplitHiLo ? L->num_groups != 1 : d.group_size % (is_f16(mode) ? 64 : 16) != 0) return false;
  // the recipes read the codebook as it came, which is not padded to whole 16-byte units
  if (mode >= kSplitInt8 && d.codebook_size * d.vector_dim % 8 != 0) return false;
  return (int64_t)L->cb_entries * d.vector_dim * 2 % 16 == 0;
}

// Accumulator columns beside two weight stages.
int most_columns(SplitMode mode) { return mode == kSplitHalf2 ? 512 - 2 * w_cols(mode) : kMaxTok; }

// Tokens of one of `tiles` equal tiles, in whole instructions: a multiple of 16, two of them above 256.
int tile_width(int64_t M, int64_t tiles) {
  const int64_t tok = ((M + tiles - 1) / tiles + 15) & ~(int64_t)15;
  return (int)(tok > 256 ? (tok + 31) & ~(int64_t)31 : tok);
}
int least_tiles(int64_t M) { return (int)((M + kMaxTok - 1) / kMaxTok); }
int most_tiles(int64_t M) { return 3 * least_tiles(M) + 1; }       // that the model is asked about

SplitChoice cut_of(int64_t M, int tok, int split, int parts) {
  SplitChoice c;
  c.tok = tok;
  c.tiles = (int)((M + tok - 1) / tok);
  c.split = split;
  c.parts = parts;
  return c;
}

// Fills in what follows from a cut, its modelled time included; false if it does not fit.
bool complete(const sacq_layer* L, SplitMode mode, SplitChoice* c) {
  if (!split_fits(L, mode, c)) return false;
  const int64_t row_tiles = (L->d.out_features + kRows - 1) / kRows;
  const int kbs = (stages_of(L->d.in_features) + c->split - 1) / c->split;
  const int at_once = active_clusters(c->split, L->num_sms);
  const int64_t waves = (row_tiles * c->tiles + at_once - 1) / at_once;
  // every CTA fetches the codebook through L2
  const int64_t ctas = row_tiles * c->tiles * c->split, resident = waves * L->num_sms;
  c->us = waves * split_cta_us(L->d.vector_dim, mode, codebook_smem(L) > 0, c->tok, kbs, c->split) +
          0.01 * (double)(ctas < resident ? ctas : resident);
  return true;
}

}  // namespace

void split_k_init(sacq_layer* L) {
  for (int i = 0; i < 4; ++i) slice_extent(L, 1 << i, &L->slice_idx[i], &L->slice_groups[i]);
  for (int mode = kSplitHiLo; mode <= kSplitFp8; ++mode) {
    const SplitMode m = (SplitMode)mode;
    int tok = takes_layer(L, m) ? most_columns(m) : 0;
    for (; tok > 0; tok -= tok > 256 ? 32 : 16) {
      SplitChoice c = cut_of(tok, tok, slices_for(L->d.in_features), 1);
      if (split_fits(L, m, &c)) break;
    }
    L->split_tok[mode] = tok > 0 ? tok : 0;
  }
}

bool split_k_tiles_fit(const sacq_layer* L, int64_t M, SplitMode mode) {
  return L->split_tok[mode] == most_columns(mode) || M <= L->split_tok[mode];
}

bool split_k_choose(const sacq_layer* L, int64_t M, SplitMode mode, SplitChoice* out) {
  *out = SplitChoice();
  g_searches.fetch_add(1, std::memory_order_relaxed);
  if (L->split_tok[mode] == 0 || M <= 0 || M > kSplitMaxM) return false;
  const int slices = slices_for(L->d.in_features);
  for (int split = 1; split <= slices; split *= 2) {
    const int parts = slices / split;
    for (int tiles = least_tiles(M); parts <= 4 && tiles <= most_tiles(M); ++tiles) {
      SplitChoice c = cut_of(M, tile_width(M, tiles), split, parts);
      if (c.tok * parts <= most_columns(mode) && complete(L, mode, &c) && c.us < out->us) *out = c;
    }
  }
  if (out->tok != 0) return true;
  *out = cut_of(M, L->split_tok[mode], slices, 1);    // narrower tiles than that: as wide as they fit
  return complete(L, mode, out);
}

int64_t split_k_ctas(const sacq_layer* L, const SplitChoice& c) {
  return (L->d.out_features + kRows - 1) / kRows * c.tiles * c.split;
}

Beside split_k_beside(const sacq_layer* L, int64_t M, const SplitChoice& c) {
  const bool wide = L->d.out_features >= 4096;
  const int64_t ctas = split_k_ctas(L, c), room = L->num_sms + (L->d.in_features <= 2048 ? 12 : 0);
  if (codebook_smem(L) == 0 || M > (wide ? 512 : 1024) || 2 * ctas + M <= room) return kBesideNone;
  return wide || 6 * ctas > 5 * L->num_sms ? kBesideMost : kBesideSome;
}

bool split_k_codebook_in_smem(const sacq_layer* L) { return codebook_smem(L) > 0; }

bool split_k_quantizes(const sacq_layer* L, const SplitChoice& c) {
  const int64_t K = L->d.in_features;
  if (c.tok > 32 || c.parts > 1 || c.box_shift != 2 || (c.split > 1 && !c.own_recv)) return false;
  const int stages = (stages_of(K) + c.split - 1) / c.split;
  if (stages > c.act_stages) return false;            // every activation tile has a place of its own
  const SplitLayout l = split_layout(c.tok, c.split, c.act_stages, c.max_slices, c.box_shift, 0, codebook_smem(L), c.own_recv, (int)(c.tok * K * 2));
  return split_smem(l) <= (codebook_smem(L) > 0 ? 224 : 164) * 1024;
}

bool split_k_choose_multi(const sacq_layer* const* layers, int n, int64_t M, SplitMode mode, SplitChoice* out) {
  const sacq_layer_desc& d0 = layers[0]->d;
  int64_t rows = 0;
  for (int l = 0; l < n; ++l) {
    const sacq_layer_desc& d = layers[l]->d;
    if (d.in_features != d0.in_features || d.vector_dim != d0.vector_dim || d.index_bits != d0.index_bits ||
        d.codebook_size != d0.codebook_size || d.group_size != d0.group_size || d.device != d0.device || d.out_features <= 0)
      return false;
    rows += (d.out_features + kRows - 1) / kRows * kRows;
  }
  sacq_layer all = *layers[0];                        // token tiles for the rows of all layers together
  all.d.out_features = rows;
  return split_k_choose(&all, M, mode, out);
}

void split_k_release(sacq_layer* L) {
  delete L->split_plan;
  L->split_plan = nullptr;
}

int launch_split_k(const sacq_layer* const* layers, int n, const void* act, const float* scale, int64_t M, void* const* ys,
                   const int64_t* ldys, SplitMode mode, const SplitChoice& c, cudaStream_t s, const void* residual,
                   int64_t ldr, const BcastDst* bc, const float* row_scale, const void* x, int64_t x_pitch) {
  const sacq_layer_desc& d0 = layers[0]->d;
  if (reinterpret_cast<uintptr_t>(act) % 16 != 0)
    return set_error(SACQ_ERR_ALIGNMENT, "quantized activations must be 16-byte aligned");
  SplitParams p;
  memset(&p, 0, sizeof(p));
  int rc = SACQ_OK;
  CUtensorMap ta;
  const uint64_t act_row = (uint64_t)d0.in_features * (is_f16(mode) ? 2 : 1);
  if (x == nullptr)
    rc = encode_bytes_2d(&ta, act, act_row, (uint64_t)M, act_row, 128u, (uint32_t)(c.tok <= 256 ? c.tok : c.tok / 2),
                         CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != SACQ_OK) return rc;
  p.x = static_cast<const uint16_t*>(x);
  p.x_pitch = x_pitch;
  int64_t widest = 0;
  for (int l = 0; l < n; ++l) {
    const sacq_layer* L = layers[l];
    rc = index_map(const_cast<sacq_layer*>(L), c.box_shift, &p.idx[l]);
    if (rc != SACQ_OK) return rc;
    SplitLayer& q = p.layer[l];
    q.cb = mode == kSplitHiLo ? L->cb_hilo
           : is_f16(mode) ? reinterpret_cast<const uint8_t*>(L->cb_f16) : static_cast<const uint8_t*>(L->d.codebook);
    q.scales = static_cast<const uint16_t*>(L->d.scales);
    q.bias = static_cast<const uint16_t*>(L->d.bias);
    q.y = static_cast<uint16_t*>(ys[l]);
    q.ldy = ldys[l];
    q.status = L->d_status;
    q.N = (int)L->d.out_features;
    q.scale_mul = ldexpf(kHalfPreScale, L->sc_exp_shift);
    q.row_mul = L->row_mul;
    q.out_mul = mode == kSplitHalf    ? ldexpf(1.f / kHalfPreScale, -(L->cb_exp_shift + L->sc_exp_shift))
                : mode == kSplitHalf2 ? ldexpf(1.f, -L->cb_exp_shift)
                                      : ldexpf(1.f, -L->cb8_exp_shift);
    if (L->d.out_features > widest) widest = L->d.out_features;
  }
  if (x != nullptr) ta = p.idx[0];                    // a valid map is passed either way
  p.act_scale = scale;
  p.row_scale = row_scale;
  p.shift = d0.shift_bf16;
  p.residual = static_cast<const uint16_t*>(residual);
  p.ldr = ldr;
  if (bc != nullptr) {
    p.n_bc = bc->n;
    for (int i = 0; i < bc->n; ++i) p.ybc[i] = static_cast<uint16_t*>(bc->ptr[i]);
  }
  p.M = (int)M; p.K = (int)d0.in_features; p.C = mode >= kSplitInt8 ? d0.codebook_size : layers[0]->cb_entries;
  p.bits = d0.index_bits; p.num_groups = (int)layers[0]->num_groups; p.group_size = d0.group_size;
  p.split = c.split; p.parts = c.parts; p.tok = c.tok; p.act_stages = c.act_stages; p.max_slices = c.max_slices;
  p.own_recv = c.own_recv ? 1 : 0;
  auto log2_of = [](int v) { int n = 0; while (1 << n < v) ++n; return n; };     // split and parts are powers of two
  p.split_shift = log2_of(c.split);
  p.slice_shift = log2_of(c.split * c.parts);
  p.own = owned_tokens(c.tok, c.split);
  p.lay = split_layout(c.tok, c.split, c.act_stages, c.max_slices, c.box_shift, mode == kSplitHiLo ? 0 : c.max_groups, codebook_smem(layers[0]), c.own_recv,
                       x != nullptr ? c.tok * p.K * 2 : 0);
  const dim3 grid((unsigned)((widest + kRows - 1) / kRows * c.split), (unsigned)c.tiles, (unsigned)n);
  const size_t smem = split_smem(p.lay);
  const bool cb = codebook_smem(layers[0]) > 0;
  auto launch = [&](auto box_shift) {
    constexpr int kB = decltype(box_shift)::value;
    if (d0.vector_dim == 8) return cb ? launch_mode<8, true, kB>(mode, ta, p, grid, smem, s) : launch_mode<8, false, kB>(mode, ta, p, grid, smem, s);
    return cb ? launch_mode<4, true, kB>(mode, ta, p, grid, smem, s) : launch_mode<4, false, kB>(mode, ta, p, grid, smem, s);
  };
  const cudaError_t e = c.box_shift == 2 ? launch(std::integral_constant<int, 2>{}) : launch(std::integral_constant<int, 0>{});
  count_launch();
  if (e != cudaSuccess) return cuda_fail(e, "split-K launch");
  return SACQ_OK;
}

}  // namespace sacq

extern "C" SACQ_API int64_t sacq_split_search_count(void) { return sacq::g_searches.load(std::memory_order_relaxed); }
