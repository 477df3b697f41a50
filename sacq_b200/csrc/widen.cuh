// Activation bytes -> fp16 (exact), the pre-pass of the fp16 tensor-core kernels (widen.cu).
#pragma once

#include "common.cuh"

namespace sacq {

// Eight encoded values -> fp16.
template <bool I8>
__device__ __forceinline__ uint4 widen8(const uint2& v) {
  const uint32_t in[2] = {v.x, v.y};
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if constexpr (I8) {
      // 1024 + (b + 128) is fp16 0x6400 | (b ^ 0x80); minus 1152 leaves b
      const uint32_t u = in[j] ^ 0x80808080u;
      const uint32_t lo = __byte_perm(u, 0x64646464u, 0x4140), hi = __byte_perm(u, 0x64646464u, 0x4342);
      const __half2 bias = __half2half2(__ushort_as_half(0x6480));
      const __half2 a = __hsub2(*reinterpret_cast<const __half2*>(&lo), bias), b = __hsub2(*reinterpret_cast<const __half2*>(&hi), bias);
      w[2 * j] = *reinterpret_cast<const uint32_t*>(&a);
      w[2 * j + 1] = *reinterpret_cast<const uint32_t*>(&b);
    } else {
      const __half2_raw a = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(in[j] & 0xffff), __NV_E4M3);
      const __half2_raw b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(in[j] >> 16), __NV_E4M3);
      w[2 * j] = (uint32_t)a.x | ((uint32_t)a.y << 16);
      w[2 * j + 1] = (uint32_t)b.x | ((uint32_t)b.y << 16);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// e4m3 (or int8) [M, K] -> fp16 [M, K]; K a multiple of 8, q 8-byte and a16 16-byte aligned.
int launch_widen(const void* q, int64_t M, int64_t K, bool int8, void* a16, cudaStream_t s);

}  // namespace sacq
