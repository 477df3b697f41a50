// Fused per-token FP8 activation quantizer.
//
// Restates quantize_rows(x, 'fp8_e4m3fn') of the reference
// (inference_acceleration_2026_10_11/a8_accuracy_recovery_2026_10_20_r1/
// perrow_a8_candidate_r3.py:17-25; zero-scale rule a8_rtn_r2.py:29-30):
//   z = float(x); s = max|z| / 448 per row, 1 for an all-zero row;
//   q = e4m3( clamp(z / s, -448, 448) )   with IEEE division and RNE conversion.
// The reference spends five elementwise torch kernels on this; here one launch reads
// the bf16 row once from HBM (second pass from registers), so the algorithmic traffic
// is 2 bytes read + 1 byte written per element.
#include "common.cuh"
#include "encode.cuh"
#include "widen.cuh"

namespace sacq {

namespace {

constexpr int kThreads = 256;

// Eight bf16 values (16 bytes) of one row -> eight bytes.
template <bool I8>
__device__ __forceinline__ uint2 encode8(const uint4& v, const RowDivisor& d) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[2];
  encode_pairs<I8, 4>(w, d, o);
  return make_uint2(o[0], o[1]);
}

// Where a quantizer puts eight encoded values: bytes, or (WIDE) the same values as fp16, exactly.
template <bool I8, bool WIDE>
__device__ __forceinline__ void store8(void* row, int64_t ch, const uint2& o) {
  if constexpr (WIDE) reinterpret_cast<uint4*>(row)[ch] = widen8<I8>(o);
  else reinterpret_cast<uint2*>(row)[ch] = o;
}

// Threads of a CTA that handles one row of K elements in 16-byte chunks: a chunk per thread while the rows
// are few (their latency is all there is: 6,144 elements on 768 threads instead of three rounds of 256), at most 256
// threads when the rows outnumber what the device holds at once; as many chunks for each thread as for the others
// (1,025 chunks on 1,024 threads took 8.2 us, 296 rows, GELU; on 544, as on 256, 6.9).
inline unsigned row_threads(int64_t M, int64_t K, int64_t few) {
  const int64_t chunks = (K + 7) / 8, most = M <= few ? 1024 : kThreads;
  const int64_t rounds = (chunks + most - 1) / most;
  const int64_t threads = rounds > 4 ? most : ((chunks + rounds - 1) / rounds + 31) / 32 * 32;
  return (unsigned)(threads < 64 ? 64 : threads);
}
constexpr int64_t kFewRows = 296;   // two per SM

// max over the CTA of a bit pattern; `red` has one word per warp (at most 32).
__device__ __forceinline__ uint32_t block_max_bits(uint32_t v, uint32_t* red) {
  v = warp_max_bits(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const unsigned lane = threadIdx.x & 31;
  return warp_max_bits(lane < (blockDim.x >> 5) ? red[lane] : 0u);
}

// Running |x| maximum of bf16 values as bit patterns, one per half of a word: among non-negative bf16 values integer
// order is value order, infinity is above every finite value and every NaN above infinity, so both survive the
// reduction the way they do in torch's amax.
__device__ __forceinline__ uint32_t pair_max(uint32_t mx, uint32_t w) { return __vmaxu2(mx, w & 0x7fff7fffu); }
__device__ __forceinline__ uint32_t chunk_max(uint32_t mx, const uint4& v) {
  return pair_max(pair_max(pair_max(pair_max(mx, v.x), v.y), v.z), v.w);
}
// ... of both halves, as the bits of an fp32 value.
__device__ __forceinline__ uint32_t pair_max_bits(uint32_t mx) { return max(mx << 16, mx & 0xffff0000u); }

// One CTA per row.  CH > 0: rows are 16-byte aligned and K % 8 == 0; a thread keeps CH 16-byte chunks of the row in
// registers between the two passes (a longer row's tail is read again).  CH = 0: any row.
template <int CH, bool I8, bool WIDE>
__global__ void __launch_bounds__(1024)
quant_act_kernel(const uint16_t* __restrict__ x, int64_t pitch, int64_t K, uint8_t* __restrict__ q,
                 float* __restrict__ scale_out) {
  __shared__ uint32_t red[32];
  SACQ_TL_BEGIN(1);
  // A GEMM launched with programmatic stream serialization may start its prologue now; it
  // waits for this grid to finish before it reads q or the scales.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // This grid is itself launched that way behind whatever precedes it on the stream (so its
  // launch latency overlaps that kernel's tail): wait for it before touching x, q or the scales
  // (the kernel in front may have produced x, or may still be reading q).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  SACQ_TL(t_dep);
  const int64_t m = blockIdx.x;
  const uint16_t* row = x + m * pitch;
  uint8_t* qrow = q + m * K * (WIDE ? 2 : 1);
  const int tid = threadIdx.x, T = blockDim.x;

  uint32_t mx = 0u;                                  // bit pattern of the running |x| maximum (absmax_bits)
  uint4 keep[CH > 0 ? CH : 1];
  const int64_t chunks = K >> 3;
  if constexpr (CH > 0) {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int64_t ch = tid + (int64_t)c * T;
      keep[c] = make_uint4(0, 0, 0, 0);
      if (ch < chunks) keep[c] = __ldg(reinterpret_cast<const uint4*>(row) + ch);
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) mx = chunk_max(mx, keep[c]);
    for (int64_t ch = tid + (int64_t)CH * T; ch < chunks; ch += T)
      mx = chunk_max(mx, __ldg(reinterpret_cast<const uint4*>(row) + ch));
    mx = pair_max_bits(mx);
  } else {
    for (int64_t k = tid; k < K; k += T) mx = absmax_bits(mx, bf16_bits_to_float(__ldg(row + k)));
  }
  const RowDivisor d = scale_of<I8>(__uint_as_float(block_max_bits(mx, red)));
  if (tid == 0) scale_out[m] = d.s;

  if constexpr (CH > 0) {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int64_t ch = tid + (int64_t)c * T;
      if (ch < chunks) store8<I8, WIDE>(qrow, ch, encode8<I8>(keep[c], d));
    }
    for (int64_t ch = tid + (int64_t)CH * T; ch < chunks; ch += T)
      store8<I8, WIDE>(qrow, ch, encode8<I8>(__ldg(reinterpret_cast<const uint4*>(row) + ch), d));
  } else {
    for (int64_t k = tid; k < K; k += T) {
      const float z = bf16_bits_to_float(__ldg(row + k));
      qrow[k] = (uint8_t)(encode2<I8>(z, 0.f, d.s) & 0xff);
    }
  }
  SACQ_TL(t_exit);
}

// The same quantizer for many rows: one WARP per row, eight rows per CTA, no block-wide barrier.  A lane keeps its
// 16-byte chunks of the row in registers across the warp reduction: 8 chunks of 8 elements, i.e. rows of up to 2,048
// elements (8,192 rows of 2,048: 9.4 us, 7.7 of HBM time).  Longer rows stay on the kernel above: 24 chunks per lane
// cost 240 registers, and reading the tail again was slower than a CTA per row too.  Same arithmetic, same bytes.  Rows
// are 16-byte aligned, K % 8 == 0.
constexpr int kRowsPerCta = 8;
constexpr int kKeepChunks = 8;
constexpr int64_t kRowsKernelMaxK = 256 * kKeepChunks;   // rows the lanes hold entirely in registers
constexpr int64_t kRowsKernelMinM = 256;   // from here on the per-row CTAs outnumber what the device holds at once

template <bool I8, bool WIDE>
__global__ void __launch_bounds__(kRowsPerCta * 32)
quant_act_rows_kernel(const uint16_t* __restrict__ x, int64_t pitch, int64_t M, int64_t K, uint8_t* __restrict__ q,
                      float* __restrict__ scale_out) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int64_t m = (int64_t)blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
  if (m >= M) return;
  const uint4* row = reinterpret_cast<const uint4*>(x + m * pitch);
  uint8_t* qrow = q + m * K * (WIDE ? 2 : 1);
  const int64_t chunks = K >> 3;
  uint32_t mx = 0u;
  uint4 keep[kKeepChunks];
#pragma unroll
  for (int c = 0; c < kKeepChunks; ++c) {
    const int64_t ch = lane + (int64_t)c * 32;
    keep[c] = make_uint4(0, 0, 0, 0);
    if (ch < chunks) keep[c] = __ldg(row + ch);
    mx = chunk_max(mx, keep[c]);
  }
  for (int64_t ch = lane + (int64_t)kKeepChunks * 32; ch < chunks; ch += 32) mx = chunk_max(mx, __ldg(row + ch));
  const RowDivisor d = scale_of<I8>(__uint_as_float(warp_max_bits(pair_max_bits(mx))));
  if (lane == 0) scale_out[m] = d.s;
#pragma unroll
  for (int c = 0; c < kKeepChunks; ++c) {
    const int64_t ch = lane + (int64_t)c * 32;
    if (ch < chunks) store8<I8, WIDE>(qrow, ch, encode8<I8>(keep[c], d));
  }
  for (int64_t ch = lane + (int64_t)kKeepChunks * 32; ch < chunks; ch += 32)
    store8<I8, WIDE>(qrow, ch, encode8<I8>(__ldg(row + ch), d));
}

// The same quantizer in front of a split-K GEMM (linear_split_k.cu), made to share an SM with that kernel's CTAs.  In a row of
// calls this grid waits for the GEMM before it while the GEMM behind it already fetches and expands weights, so whatever
// keeps the three apart is paid on every call.  Two things did.  An SM whose memory is divided for a kernel of little
// shared memory takes no CTA of the GEMM before it is idle again, hence the carve-out.  And a GEMM CTA (18 warps of
// 88 registers) leaves 2,304 registers of an SM quarter: a warp of up to 72, where the row kernels have two or six.  GEMM CTAs
// entered only when the one before had left, 1 to 2 us late.  Quantizer + GEMM in a graph, without / with this kernel:
// 2048 -> 2048 at 64 tokens 7.5 / 6.5 us, 128 9.2 / 7.6, 6144 -> 2048 at 64 11.0 / 9.6, 128 13.2 / 11.5, 2048 -> 6144 at 64
// 9.2 / 8.2, 300 16.0 / 14.4, 2048 -> 2048, d = 4, at 100 10.9 / 8.0.
// T threads per row, 128 / T rows per CTA; a row lies in registers between the passes, CH 16-byte chunks per thread.
// Same arithmetic, same bytes.
constexpr int kBesideThreads = 128;

template <int T, int CH, bool I8, bool WIDE>
__global__ void __launch_bounds__(kBesideThreads, 7)
quant_act_beside_kernel(const uint16_t* __restrict__ x, int64_t pitch, int64_t M, int64_t K, uint8_t* __restrict__ q,
                        float* __restrict__ scale_out) {
  constexpr int W = T / 32;                          // warps per row
  __shared__ uint32_t red[kBesideThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x % T;
  const int64_t m = (int64_t)blockIdx.x * (kBesideThreads / T) + threadIdx.x / T;
  const bool live = m < M;
  const uint4* row = reinterpret_cast<const uint4*>(x + m * pitch);
  uint8_t* qrow = q + m * K * (WIDE ? 2 : 1);
  const int64_t chunks = live ? K >> 3 : 0;
  uint4 keep[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int64_t ch = tid + c * T;
    keep[c] = make_uint4(0, 0, 0, 0);
    if (ch < chunks) keep[c] = __ldg(row + ch);
  }
  uint32_t mx = 0u;
#pragma unroll
  for (int c = 0; c < CH; ++c) mx = chunk_max(mx, keep[c]);
  mx = warp_max_bits(pair_max_bits(mx));
  if constexpr (W > 1) {
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[warp] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < W; ++w) mx = max(mx, red[warp / W * W + w]);
  }
  const RowDivisor d = scale_of<I8>(__uint_as_float(mx));
  if (live && tid == 0) scale_out[m] = d.s;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int64_t ch = tid + c * T;
    if (ch < chunks) store8<I8, WIDE>(qrow, ch, encode8<I8>(keep[c], d));
  }
}

// Threads per row of the kernel above; 0: one of the others.  Quantizer + GEMM in a graph, without / row CTAs / warps:
// up to 255 tokens a row per CTA (2048 -> 2048 at 100 9.0 / 7.5 / 7.7 us); from there a warp per row, which is four times fewer
// CTAs to start (2048 -> 1024 at 300 8.8 / 9.4 / 8.4, grouped scales 10.2 / 11.3 / 9.4; 2048 -> 2048 at 700 13.6 / 12.2), but up to
// 340 row CTAs where GEMM CTAs on most SMs leave few warps a place (2048 -> 6144 at 300 16.0 / 14.3 / 14.9, 370 16.8 / 15.9 / 15.7).
// Rows that a warp's registers do not hold keep to row CTAs while about two per SM hold them, 370 (4096 -> 1024 at 300
// 12.1 / 10.2, 6144 -> 1536 INT8 at 340 a twentieth), and 3.5 MB of them next to GEMM CTAs on most SMs (6144 -> 2048 at 290
// 15.8 / 15.2, 300 15.7 / 16.2, 370 16.8 / 17.6).
inline int beside_threads(Beside beside, int64_t M, int64_t K) {
  if (K > kRowsKernelMaxK)
    return K <= kBesideThreads * 8 * kKeepChunks && M <= 370 && (beside == kBesideSome || M * K <= (7 << 18)) ? kBesideThreads : 0;
  return M < kRowsKernelMinM || (beside == kBesideMost && M <= 340) ? kBesideThreads : 32;
}

// The carve-out as an attribute of the function: as one of each launch it costs the host 0.25 us a call (1536 x 1536 at 80 tokens,
// eager 8.3 against 8.0).
template <auto Kern, typename... Args>
cudaError_t launch_carved(const cudaLaunchConfig_t& cfg, Args... args) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(Kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  return cudaLaunchKernelEx(&cfg, Kern, args...);
}

template <int T, bool I8, bool WIDE>
cudaError_t launch_beside(cudaLaunchConfig_t& cfg, const uint16_t* x, int64_t pitch, int64_t M, int64_t K, uint8_t* q, float* scale) {
  constexpr int R = kBesideThreads / T;
  cfg.gridDim = dim3((unsigned)((M + R - 1) / R));
  cfg.blockDim = dim3(kBesideThreads);
  const int64_t per_thread = (K / 8 + T - 1) / T;
  if (per_thread <= 2) return launch_carved<quant_act_beside_kernel<T, 2, I8, WIDE>>(cfg, x, pitch, M, K, q, scale);
  if (per_thread <= 4) return launch_carved<quant_act_beside_kernel<T, 4, I8, WIDE>>(cfg, x, pitch, M, K, q, scale);
  return launch_carved<quant_act_beside_kernel<T, kKeepChunks, I8, WIDE>>(cfg, x, pitch, M, K, q, scale);
}

template <bool I8, bool WIDE>
cudaError_t launch_quant(cudaLaunchConfig_t& cfg, bool vec, Beside beside, const uint16_t* x, int64_t pitch, int64_t M, int64_t K,
                         uint8_t* q, float* scale) {
  const int t = vec && beside != kBesideNone ? beside_threads(beside, M, K) : 0;
  if (t > 0)
    return t == 32 ? launch_beside<32, I8, WIDE>(cfg, x, pitch, M, K, q, scale)
                   : launch_beside<kBesideThreads, I8, WIDE>(cfg, x, pitch, M, K, q, scale);
  if (vec && M >= kRowsKernelMinM && K <= kRowsKernelMaxK) {
    cfg.gridDim = dim3((unsigned)((M + kRowsPerCta - 1) / kRowsPerCta));
    cfg.blockDim = dim3(kRowsPerCta * 32);
    return cudaLaunchKernelEx(&cfg, quant_act_rows_kernel<I8, WIDE>, x, pitch, M, K, q, scale);
  }
  if (vec) {
    // few: while CTAs of a thread per chunk are all resident (512 rows of 4,096: 3.7 us on 256 threads, 2.6 on 512)
    const int64_t fit = 148 * (2048 / ((K / 8 + 31) / 32 * 32));
    const unsigned threads = row_threads(M, K, fit > kFewRows ? fit : kFewRows);
    cfg.blockDim = dim3(threads);
    switch ((K / 8 + threads - 1) / threads) {
      case 1: return cudaLaunchKernelEx(&cfg, quant_act_kernel<1, I8, WIDE>, x, pitch, K, q, scale);
      case 2: return cudaLaunchKernelEx(&cfg, quant_act_kernel<2, I8, WIDE>, x, pitch, K, q, scale);
      case 3: return cudaLaunchKernelEx(&cfg, quant_act_kernel<3, I8, WIDE>, x, pitch, K, q, scale);
      default: return cudaLaunchKernelEx(&cfg, quant_act_kernel<4, I8, WIDE>, x, pitch, K, q, scale);
    }
  }
  if constexpr (WIDE) return cudaErrorInvalidValue;
  else return cudaLaunchKernelEx(&cfg, quant_act_kernel<0, I8, false>, x, pitch, K, q, scale);
}

}  // namespace

#ifdef SACQ_TRACE
SACQ_TL_DEFINE_DUMP(sacq_debug_timeline_quant)
#endif

int launch_quant_act(const void* x, int64_t pitch, int64_t M, int64_t K, bool int8, bool wide, void* q, float* scale,
                     cudaStream_t s, Beside beside) {
  if (M == 0 || K == 0) return SACQ_OK;
  const bool vec = (K % 8 == 0) && (pitch % 8 == 0) && (reinterpret_cast<uintptr_t>(x) % 16 == 0) &&
                   (reinterpret_cast<uintptr_t>(q) % (wide ? 16 : 8) == 0);
  if (M > 2147483647LL) return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld exceeds the grid limit", (long long)M);
  if (wide && !vec) return set_error(SACQ_ERR_ALIGNMENT, "the fp16 form needs 16-byte aligned rows");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)M);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const uint16_t* xp = static_cast<const uint16_t*>(x);
  uint8_t* qp = static_cast<uint8_t*>(q);
  if (int8) SACQ_CUDA_TRY(wide ? (launch_quant<true, true>(cfg, vec, beside, xp, pitch, M, K, qp, scale))
                               : (launch_quant<true, false>(cfg, vec, beside, xp, pitch, M, K, qp, scale)));
  else SACQ_CUDA_TRY(wide ? (launch_quant<false, true>(cfg, vec, beside, xp, pitch, M, K, qp, scale))
                          : (launch_quant<false, false>(cfg, vec, beside, xp, pitch, M, K, qp, scale)));
  count_launch();
  return SACQ_OK;
}

}  // namespace sacq

// ----------------------------------------------------------------------------
// Activation function fused into the quantizer.
//
// The MLP of a transformer block feeds its down projection with act(gate) * up (gated) or
// act(x); run as separate tensor operations that is two or three elementwise kernels and a
// round trip of the [M, K] intermediate before the quantizer reads it again.  Here one launch
// produces the e4m3 row and its scale directly; the intermediate is never written.  The
// arithmetic follows the tensor operations it replaces, rounding to bf16 where they do, so the
// bytes equal quantize_rows(silu(gate) * up) and quantize_rows(gelu(x)) (the reference fuses
// the same stage for its INT8 path, int8_swiglu_lookup_fusion_20261028_r1.py:9-21).
// ----------------------------------------------------------------------------
namespace sacq {

namespace {

__device__ __forceinline__ float round_bf16(float v) { return bf16_bits_to_float(float_to_bf16_bits(v)); }

// fp32 silu of a bf16 value.  The quotient of the approximate exponential and division rounds to the bf16 value of
// a / (1 + expf(-a)) for every bf16 a (all 65,536 compared), but where the divisor is out of __fdividef's range.  The
// plain form, an IEEE division per element, bounded the kernel
// (8,192 rows of 6,144: 73.8 us, now 50.3; 300 rows: 6.4, now 5.0).
__device__ __forceinline__ float silu(float a) {
  return a < -87.0f ? a / (1.0f + expf(-a)) : __fdividef(a, 1.0f + __expf(-a));
}

// KIND 0: bf16(bf16(silu(a)) * b); KIND 1: bf16(gelu(a)), erf form;
// KIND 2: bf16(bf16(a * bf16(1 + b)) + c), the AdaLN modulation a * (1 + scale) + shift.
template <int KIND>
__device__ __forceinline__ float act_value(float a, float b, float c) {
  if constexpr (KIND == 0) {
    return round_bf16(round_bf16(silu(a)) * b);
  } else if constexpr (KIND == 1) {
    return round_bf16(a * 0.5f * (1.0f + erff(a * 0.70710678118654752440f)));
  } else {
    return round_bf16(round_bf16(a * round_bf16(1.0f + b)) + c);
  }
}

// act_value of the two bf16 values in each word.
template <int KIND>
__device__ __forceinline__ uint32_t act_pair(uint32_t a, uint32_t b, uint32_t c) {
  const float a0 = __uint_as_float(a << 16), a1 = __uint_as_float(a & 0xffff0000u);
  if constexpr (KIND == 0) {
    // the product of two bf16 values is exact in fp32, so one rounding to bf16 is the same from either form
    const __nv_bfloat162 y = __hmul2(__floats2bfloat162_rn(silu(a0), silu(a1)), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&y);
  } else {
    const float y0 = act_value<KIND>(a0, __uint_as_float(b << 16), __uint_as_float(c << 16));
    const float y1 = act_value<KIND>(a1, __uint_as_float(b & 0xffff0000u), __uint_as_float(c & 0xffff0000u));
    return (__float_as_uint(y0) >> 16) | (__float_as_uint(y1) & 0xffff0000u);   // both are bf16 values
  }
}

// CH > 0: every row of a, b, c and q is 16-byte (q: 8-byte) aligned, K % 8 == 0 and a thread holds CH chunks of 8
// results in registers between the passes; of a row longer than that (TAIL) it keeps the rest in shared memory.
// CH = 0: any row, kept in shared memory, an element at a time (512 rows of 14,336, SiLU: 26.8 us that way, 11.5 here).
template <int KIND, int CH, bool TAIL>
__global__ void __launch_bounds__(1024)
act_quant_fp8_kernel(const uint16_t* __restrict__ a, int64_t a_pitch, const uint16_t* __restrict__ b, int64_t b_pitch,
                     const uint16_t* __restrict__ c, int64_t K, uint8_t* __restrict__ q,
                     float* __restrict__ scale_out) {
  extern __shared__ __align__(16) uint16_t yrow[];    // CH = 0, TAIL: the row's (the tail's) bf16 values between the passes
  __shared__ uint32_t red[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // launched behind the producer of a / b with programmatic serialization
  const int64_t m = blockIdx.x;
  const int tid = threadIdx.x, T = blockDim.x;
  const uint16_t* arow = a + m * a_pitch;
  const uint16_t* brow = KIND == 1 ? nullptr : b + m * b_pitch;      // pitch 0: one vector for every row
  uint8_t* qrow = q + m * K;
  uint32_t mx = 0u;                                  // bit pattern of the running maximum (absmax_bits)
  if constexpr (CH > 0) {
    const int64_t chunks = K >> 3, kept = (int64_t)CH * T;
    auto load = [&](int64_t ch, uint4& v, uint4& w, uint4& u) {
      v = __ldg(reinterpret_cast<const uint4*>(arow) + ch);
      if constexpr (KIND != 1) w = __ldg(reinterpret_cast<const uint4*>(brow) + ch);
      if constexpr (KIND == 2) u = __ldg(reinterpret_cast<const uint4*>(c) + ch);
    };
    auto act = [&](const uint4& v, const uint4& w, const uint4& u) {
      return make_uint4(act_pair<KIND>(v.x, w.x, u.x), act_pair<KIND>(v.y, w.y, u.y), act_pair<KIND>(v.z, w.z, u.z),
                        act_pair<KIND>(v.w, w.w, u.w));
    };
    uint4 y[CH], bb[CH], cc[CH];
#pragma unroll
    for (int h = 0; h < CH; ++h) {                   // all loads first
      const int64_t ch = tid + (int64_t)h * T;
      y[h] = bb[h] = cc[h] = make_uint4(0, 0, 0, 0);
      if (ch < chunks) load(ch, y[h], bb[h], cc[h]);
    }
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      y[h] = act(y[h], bb[h], cc[h]);
      if (tid + (int64_t)h * T < chunks) mx = chunk_max(mx, y[h]);
    }
    if constexpr (TAIL) {
      uint4* tail = reinterpret_cast<uint4*>(yrow);
#pragma unroll 4
      for (int64_t ch = kept + tid; ch < chunks; ch += T) {
        uint4 v, w = make_uint4(0, 0, 0, 0), u = w;
        load(ch, v, w, u);
        v = act(v, w, u);
        tail[ch - kept] = v;                         // read again by this thread only
        mx = chunk_max(mx, v);
      }
    }
    mx = pair_max_bits(mx);
    const RowDivisor d = scale_of<false>(__uint_as_float(block_max_bits(mx, red)));
    if (tid == 0) scale_out[m] = d.s;
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      const int64_t ch = tid + (int64_t)h * T;
      if (ch < chunks) reinterpret_cast<uint2*>(qrow)[ch] = encode8<false>(y[h], d);
    }
    if constexpr (TAIL) {
#pragma unroll 2
      for (int64_t ch = kept + tid; ch < chunks; ch += T)
        reinterpret_cast<uint2*>(qrow)[ch] = encode8<false>(reinterpret_cast<const uint4*>(yrow)[ch - kept], d);
    }
  } else {
#pragma unroll 4
    for (int64_t k = tid; k < K; k += T) {
      const float av = bf16_bits_to_float(__ldg(arow + k));
      const float bv = KIND == 1 ? 0.f : bf16_bits_to_float(__ldg(brow + k));
      const float cv = KIND == 2 ? bf16_bits_to_float(__ldg(c + k)) : 0.f;
      const float y = act_value<KIND>(av, bv, cv);
      yrow[k] = float_to_bf16_bits(y);
      mx = absmax_bits(mx, y);
    }
    const float s = scale_of<false>(__uint_as_float(block_max_bits(mx, red))).s;
    if (tid == 0) scale_out[m] = s;
    for (int64_t k2 = 2 * (int64_t)tid; k2 < K; k2 += 2 * T) {
      const float y0 = bf16_bits_to_float(yrow[k2]);
      const float y1 = k2 + 1 < K ? bf16_bits_to_float(yrow[k2 + 1]) : 0.f;
      const uint32_t pair = float2_to_e4m3x2(sat448(__fdiv_rn(y0, s)), sat448(__fdiv_rn(y1, s)));
      if (k2 + 1 < K && (reinterpret_cast<uintptr_t>(qrow + k2) & 1) == 0)
        *reinterpret_cast<uint16_t*>(qrow + k2) = (uint16_t)pair;
      else {
        qrow[k2] = (uint8_t)(pair & 0xff);
        if (k2 + 1 < K) qrow[k2 + 1] = (uint8_t)(pair >> 8);
      }
    }
  }
}

// The instance for rows of that many chunks a thread: 1..4 in registers, -1: four and a tail, else (0) any row.
template <int KIND>
const void* act_quant_instance(int64_t per_thread) {
  switch (per_thread) {
    case 1: return (const void*)act_quant_fp8_kernel<KIND, 1, false>;
    case 2: return (const void*)act_quant_fp8_kernel<KIND, 2, false>;
    case 3: return (const void*)act_quant_fp8_kernel<KIND, 3, false>;
    case 4: return (const void*)act_quant_fp8_kernel<KIND, 4, false>;
    case -1: return (const void*)act_quant_fp8_kernel<KIND, 4, true>;
    default: return (const void*)act_quant_fp8_kernel<KIND, 0, false>;
  }
}

}  // namespace

int launch_act_quant_fp8(int kind, const void* a, int64_t a_pitch, const void* b, int64_t b_pitch, const void* c,
                         int64_t M, int64_t K, void* q, float* scale, cudaStream_t s) {
  if (M == 0 || K == 0) return SACQ_OK;
  if (M > 2147483647LL) return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld exceeds the grid limit", (long long)M);
  const bool vec = (K % 8 == 0) && (a_pitch % 8 == 0) && (reinterpret_cast<uintptr_t>(a) % 16 == 0) &&
                   (reinterpret_cast<uintptr_t>(q) % 8 == 0) &&
                   (kind == 1 || ((kind == 2 || b_pitch % 8 == 0) && reinterpret_cast<uintptr_t>(b) % 16 == 0)) &&
                   (kind != 2 || reinterpret_cast<uintptr_t>(c) % 16 == 0);
  const unsigned threads = row_threads(M, K, kFewRows);
  int64_t per_thread = vec ? (K / 8 + threads - 1) / threads : 0;
  if (per_thread > 4) per_thread = -1;
  const size_t smem = per_thread > 0 ? 0 : (size_t)(K - (per_thread < 0 ? 32 * (int64_t)threads : 0)) * sizeof(uint16_t);
  if ((size_t)K * sizeof(uint16_t) > 200 * 1024 && per_thread <= 0)
    return set_error(SACQ_ERR_UNSUPPORTED, "K=%lld: a row does not fit shared memory", (long long)K);
  const void* fn = kind == 0 ? act_quant_instance<0>(per_thread) : kind == 1 ? act_quant_instance<1>(per_thread)
                                                                             : act_quant_instance<2>(per_thread);
  static bool configured[3][2][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const int tail = per_thread < 0;
  if (smem > 48 * 1024 && (dev < 0 || dev >= 64 || !configured[kind][tail][dev])) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute");
    if (dev >= 0 && dev < 64) configured[kind][tail][dev] = true;
  }
  const uint16_t* ap = static_cast<const uint16_t*>(a);
  const uint16_t* bp = kind == 1 ? nullptr : static_cast<const uint16_t*>(b);
  const uint16_t* cp = kind == 2 ? static_cast<const uint16_t*>(c) : nullptr;
  int64_t bpitch = kind == 0 ? b_pitch : 0;
  uint8_t* qp = static_cast<uint8_t*>(q);
  void* args[] = {&ap, &a_pitch, &bp, &bpitch, &cp, &K, &qp, &scale};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)M);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SACQ_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, args));
  count_launch();
  SACQ_CUDA_TRY(cudaGetLastError());
  return SACQ_OK;
}

}  // namespace sacq

// ----------------------------------------------------------------------------
// LayerNorm (+ AdaLN modulation) fused into the quantizer.
//
// A pre-norm transformer block normalises its input only to feed quantized projections, so
// the normalised tensor need not exist in memory: one launch reads x once, keeps the row in
// shared memory, and emits the e4m3 row and its scale (the reference fuses this stage in
// codex_norm3_regpack_20261029_r1/kernel.cu and codex_adaln_sharedmax_20261029_r2/kernel.cu
// for its INT8 path).  Arithmetic: fp32 mean, fp32 centred variance (two passes over the
// on-chip row), rstd = 1 / sqrt(var + eps), y = bf16((x - mean) * rstd * gamma + beta),
// optionally the AdaLN modulation bf16(bf16(y * bf16(1 + s)) + t), then the quantizer.  The
// reduction order differs from a framework LayerNorm's, so y agrees with it to one bf16 ulp,
// not to the bit; the quantizer's bytes are exactly those of quantizing this kernel's own y.
// ----------------------------------------------------------------------------
namespace sacq {

namespace {

// Sum over the CTA, the same order in every thread; `red` has one word per warp.
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;
}

// The row's element after normalisation and modulation, a bf16 value.
template <bool MOD>
__device__ __forceinline__ float norm_value(float x, float mean, float rstd, bool affine_w, float gamma, bool affine_b,
                                            float beta, float ms, float mt) {
  float y = (x - mean) * rstd;
  if (affine_w) y = y * gamma;
  if (affine_b) y = y + beta;
  y = round_bf16(y);
  if constexpr (MOD) y = round_bf16(round_bf16(y * round_bf16(1.0f + ms)) + mt);
  return y;
}

// CH > 0: x, the vectors, y_out and q are 16-byte (q: 8-byte) aligned, K % 8 == 0 and a thread holds CH chunks of 8
// elements in registers through all passes (in shared memory and one element at a time this kernel took 4.2 us for
// 300 rows of 2,048); of a row longer than that (TAIL) it keeps the rest in shared memory, as bf16.  CH = 0: any row,
// kept in shared memory.
template <bool MOD, int CH, bool TAIL>
__global__ void __launch_bounds__(1024)
layernorm_quant_fp8_kernel(const uint16_t* __restrict__ x, int64_t pitch, const uint16_t* __restrict__ gamma,
                           const uint16_t* __restrict__ beta, float eps, const uint16_t* __restrict__ mod_scale,
                           const uint16_t* __restrict__ mod_shift, int64_t K, uint16_t* __restrict__ y_out,
                           int64_t y_pitch, uint8_t* __restrict__ q, float* __restrict__ scale_out) {
  extern __shared__ __align__(16) float xrow[];       // CH = 0: the row in fp32, later its bf16 result in place; TAIL: chunks
  __shared__ float red_sum[32], red_sq[32];
  __shared__ uint32_t red_max[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x, T = blockDim.x;
  const int64_t m = blockIdx.x, chunks = K >> 3;
  const uint16_t* row = x + m * pitch;
  uint8_t* qrow = q + m * K;
  uint32_t mx = 0u;                                  // bit pattern of the running maximum (absmax_bits)
  if constexpr (CH > 0) {
    asm volatile("griddepcontrol.wait;" ::: "memory");   // launched behind the producer of x with programmatic serialization
    uint4 v[CH];
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      const int64_t ch = tid + (int64_t)h * T;
      v[h] = ch < chunks ? __ldg(reinterpret_cast<const uint4*>(row) + ch) : make_uint4(0, 0, 0, 0);
    }
    const int64_t kept = (int64_t)CH * T;
    uint4* tail = reinterpret_cast<uint4*>(xrow);     // chunk ch at ch - kept, read by the thread that wrote it only
    auto word = [](const uint4& u, int j) { return j == 0 ? u.x : j == 1 ? u.y : j == 2 ? u.z : u.w; };
    auto lo = [](uint32_t w) { return __uint_as_float(w << 16); };
    auto hi = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
    float sum = 0.f;
    auto add = [&](const uint4& u) {
#pragma unroll
      for (int j = 0; j < 4; ++j) sum += lo(word(u, j)) + hi(word(u, j));
    };
#pragma unroll
    for (int h = 0; h < CH; ++h) add(v[h]);
    if constexpr (TAIL) {
#pragma unroll 4
      for (int64_t ch = kept + tid; ch < chunks; ch += T) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(row) + ch);
        tail[ch - kept] = u;
        add(u);
      }
    }
    const float mean = block_sum(sum, red_sum) / (float)K;
    float sq = 0.f;
    auto add_sq = [&](const uint4& u) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d0 = lo(word(u, j)) - mean, d1 = hi(word(u, j)) - mean;
        sq += d0 * d0;
        sq += d1 * d1;
      }
    };
#pragma unroll
    for (int h = 0; h < CH; ++h)
      if (tid + (int64_t)h * T < chunks) add_sq(v[h]);
    if constexpr (TAIL) {
#pragma unroll 4
      for (int64_t ch = kept + tid; ch < chunks; ch += T) add_sq(tail[ch - kept]);
    }
    const float var = block_sum(sq, red_sq) / (float)K;
    const float rstd = 1.0f / sqrtf(var + eps);
    const bool aw = gamma != nullptr, ab = beta != nullptr;
    auto normalize = [&](const uint4& u, int64_t ch) {
      uint4 g = make_uint4(0, 0, 0, 0), b = g, ms = g, mt = g;
      if (aw) g = __ldg(reinterpret_cast<const uint4*>(gamma) + ch);
      if (ab) b = __ldg(reinterpret_cast<const uint4*>(beta) + ch);
      if constexpr (MOD) {
        ms = __ldg(reinterpret_cast<const uint4*>(mod_scale) + ch);
        mt = __ldg(reinterpret_cast<const uint4*>(mod_shift) + ch);
      }
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y0 = norm_value<MOD>(lo(word(u, j)), mean, rstd, aw, lo(word(g, j)), ab, lo(word(b, j)), lo(word(ms, j)),
                                         lo(word(mt, j)));
        const float y1 = norm_value<MOD>(hi(word(u, j)), mean, rstd, aw, hi(word(g, j)), ab, hi(word(b, j)), hi(word(ms, j)),
                                         hi(word(mt, j)));
        o[j] = (__float_as_uint(y0) >> 16) | (__float_as_uint(y1) & 0xffff0000u);    // both are bf16 values
      }
      const uint4 y = make_uint4(o[0], o[1], o[2], o[3]);
      mx = chunk_max(mx, y);
      if (y_out != nullptr) reinterpret_cast<uint4*>(y_out + m * y_pitch)[ch] = y;
      return y;
    };
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      const int64_t ch = tid + (int64_t)h * T;
      if (ch < chunks) v[h] = normalize(v[h], ch);
    }
    if constexpr (TAIL) {
#pragma unroll 2
      for (int64_t ch = kept + tid; ch < chunks; ch += T) tail[ch - kept] = normalize(tail[ch - kept], ch);
    }
    mx = pair_max_bits(mx);
    const RowDivisor d = scale_of<false>(__uint_as_float(block_max_bits(mx, red_max)));
    if (tid == 0) scale_out[m] = d.s;
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      const int64_t ch = tid + (int64_t)h * T;
      if (ch < chunks) reinterpret_cast<uint2*>(qrow)[ch] = encode8<false>(v[h], d);
    }
    if constexpr (TAIL) {
#pragma unroll 2
      for (int64_t ch = kept + tid; ch < chunks; ch += T) reinterpret_cast<uint2*>(qrow)[ch] = encode8<false>(tail[ch - kept], d);
    }
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float sum = 0.f;
#pragma unroll 4
    for (int64_t k = tid; k < K; k += T) {
      const float v = bf16_bits_to_float(__ldg(row + k));
      xrow[k] = v;
      sum += v;
    }
    const float mean = block_sum(sum, red_sum) / (float)K;
    float sq = 0.f;
#pragma unroll 4
    for (int64_t k = tid; k < K; k += T) {
      const float dlt = xrow[k] - mean;
      sq += dlt * dlt;
    }
    const float var = block_sum(sq, red_sq) / (float)K;
    const float rstd = 1.0f / sqrtf(var + eps);
#pragma unroll 4
    for (int64_t k = tid; k < K; k += T) {
      const float y = norm_value<MOD>(xrow[k], mean, rstd, gamma != nullptr, gamma ? bf16_bits_to_float(__ldg(gamma + k)) : 0.f,
                                      beta != nullptr, beta ? bf16_bits_to_float(__ldg(beta + k)) : 0.f,
                                      MOD ? bf16_bits_to_float(__ldg(mod_scale + k)) : 0.f,
                                      MOD ? bf16_bits_to_float(__ldg(mod_shift + k)) : 0.f);
      xrow[k] = y;
      if (y_out != nullptr) y_out[m * y_pitch + k] = float_to_bf16_bits(y);
      mx = absmax_bits(mx, y);
    }
    const float s = scale_of<false>(__uint_as_float(block_max_bits(mx, red_max))).s;
    if (tid == 0) scale_out[m] = s;
#pragma unroll 4
    for (int64_t k = tid; k < K; k += T)
      qrow[k] = (uint8_t)(float2_to_e4m3x2(sat448(__fdiv_rn(xrow[k], s)), 0.f) & 0xff);
  }
}

}  // namespace

namespace {
template <bool MOD>
const void* layernorm_instance(int64_t per_thread) {  // as act_quant_instance
  switch (per_thread) {
    case 1: return (const void*)layernorm_quant_fp8_kernel<MOD, 1, false>;
    case 2: return (const void*)layernorm_quant_fp8_kernel<MOD, 2, false>;
    case 3: return (const void*)layernorm_quant_fp8_kernel<MOD, 3, false>;
    case 4: return (const void*)layernorm_quant_fp8_kernel<MOD, 4, false>;
    case -1: return (const void*)layernorm_quant_fp8_kernel<MOD, 4, true>;
    default: return (const void*)layernorm_quant_fp8_kernel<MOD, 0, false>;
  }
}
}  // namespace

int launch_layernorm_quant_fp8(const void* x, int64_t pitch, const void* gamma, const void* beta, float eps,
                               const void* mod_scale, const void* mod_shift, int64_t M, int64_t K, void* y_out,
                               int64_t y_pitch, void* q, float* scale, cudaStream_t s) {
  if (M == 0 || K == 0) return SACQ_OK;
  if (M > 2147483647LL) return set_error(SACQ_ERR_UNSUPPORTED, "M=%lld exceeds the grid limit", (long long)M);
  const bool mod = mod_scale != nullptr;
  auto al = [](const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };   // null: aligned
  const bool vec = K % 8 == 0 && pitch % 8 == 0 && al(x, 16) && al(gamma, 16) && al(beta, 16) && al(mod_scale, 16) &&
                   al(mod_shift, 16) && al(q, 8) && (y_out == nullptr || (al(y_out, 16) && y_pitch % 8 == 0));
  const unsigned threads = row_threads(M, K, kFewRows);
  int64_t per_thread = vec ? (K / 8 + threads - 1) / threads : 0;
  if (per_thread > 4) per_thread = -1;
  const size_t smem = per_thread > 0 ? 0 : per_thread < 0 ? (size_t)(K - 32 * (int64_t)threads) * sizeof(uint16_t) : (size_t)K * sizeof(float);
  if ((size_t)K * sizeof(float) > 200 * 1024 && per_thread <= 0)
    return set_error(SACQ_ERR_UNSUPPORTED, "K=%lld: a row does not fit shared memory", (long long)K);
  const void* fn = mod ? layernorm_instance<true>(per_thread) : layernorm_instance<false>(per_thread);
  static bool configured[2][2][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const int tail = per_thread < 0;
  if (smem > 48 * 1024 && (dev < 0 || dev >= 64 || !configured[mod][tail][dev])) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute");
    if (dev >= 0 && dev < 64) configured[mod][tail][dev] = true;
  }
  const uint16_t* xp = static_cast<const uint16_t*>(x);
  const uint16_t* gp = static_cast<const uint16_t*>(gamma);
  const uint16_t* bp = static_cast<const uint16_t*>(beta);
  const uint16_t* sp = static_cast<const uint16_t*>(mod_scale);
  const uint16_t* tp = static_cast<const uint16_t*>(mod_shift);
  uint16_t* yp = static_cast<uint16_t*>(y_out);
  uint8_t* qp = static_cast<uint8_t*>(q);
  void* args[] = {&xp, &pitch, &gp, &bp, &eps, &sp, &tp, &K, &yp, &y_pitch, &qp, &scale};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)M);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SACQ_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, args));
  count_launch();
  return SACQ_OK;
}

}  // namespace sacq
