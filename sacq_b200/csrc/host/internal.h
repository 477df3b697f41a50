/* Entry points between the library and its Python extension (native_calls.cpp); not part of the public C ABI. */
#ifndef SACQ_B200_INTERNAL_H_
#define SACQ_B200_INTERNAL_H_

#include "../../../include/sacq_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Quantizer + GEMM with the bytes of the separate calls, optionally with a residual (bf16 [M, ldr], e4m3 activations
 * only) or with INT8 activations.  Scratch and workspace as for those; what they hold afterwards is undefined (few
 * tokens are quantized inside the GEMM, fp16 GEMMs take their activations as fp16). */
SACQ_API int sacq_forward_call(const sacq_layer_t* layer, const void* x_bf16, int64_t x_pitch, int64_t M, int int8,
                               const void* residual, int64_t ldr, void* q_scratch, float* scale_scratch, void* y_out,
                               int64_t ldy, void* workspace, int64_t workspace_bytes, void* stream);

/* How often the cut of a split-K call has been searched so far (host time that a call should pay once). */
SACQ_API int64_t sacq_split_search_count(void);

#ifdef __cplusplus
}
#endif
#endif
