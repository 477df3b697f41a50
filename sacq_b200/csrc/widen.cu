// Activation bytes -> fp16, the pre-pass of the fp16 tensor-core kernels (grouped scales, INT8 activations).
// A streaming kernel (1 byte read, 2 written per element) that is bound by its launch up to a few hundred
// rows; it starts early behind the quantizer and lets the GEMM behind it start early in turn.
#include "widen.cuh"

namespace sacq {

namespace {

// One thread widens 8 consecutive elements.
template <bool I8>
__global__ void __launch_bounds__(256) widen_kernel(const uint8_t* __restrict__ q, int64_t chunks, __half* __restrict__ a16) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= chunks) return;
  reinterpret_cast<uint4*>(a16)[i] = widen8<I8>(__ldg(reinterpret_cast<const uint2*>(q) + i));
}

}  // namespace

int launch_widen(const void* q, int64_t M, int64_t K, bool int8, void* a16, cudaStream_t s) {
  const int64_t chunks = M * (K >> 3);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((chunks + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const uint8_t* qp = static_cast<const uint8_t*>(q);
  __half* ap = static_cast<__half*>(a16);
  if (int8) SACQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, widen_kernel<true>, qp, chunks, ap));
  else SACQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, widen_kernel<false>, qp, chunks, ap));
  count_launch();
  return SACQ_OK;
}

}  // namespace sacq
