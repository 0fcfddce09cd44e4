// FP8 E4M3 linears in the tensor-core layout, few activation rows (qgemm.cu takes the others); implemented in
// fp8_mma.cu.
#pragma once

#include "goph_internal.cuh"

namespace goph {

// Up to 4 rows of f32 or 16 of bf16 activations: e4m3 operands read by the MMA from shared memory, nothing converted.
int tc_gemm_fp8(const goph_fp8_linear* w, float* out, const void* x, bool x_bf16, int batch, cudaStream_t stream);

// True when an FP8 linear of this shape can take the tiled layout (in_dim a multiple of 256).
bool tc_fp8_supported(int in_dim);
// Builds w->tiled from w->weight (row-major bytes on the device); the caller then frees w->weight.
// Sets *has_nan when a byte is one of the two NaN codes (such a matrix stays row-major).
int tc_fp8_make_tiled(goph_fp8_linear* w, int* has_nan);
// fp8.Linear.DequantRowTo from the tiled layout.
int tc_fp8_dequant_tiled(const goph_fp8_linear* w, float* out, cudaStream_t stream);
// Device status word of the kernel (0 = every wait completed).
int fp8_mma_status(int device);
void fp8_mma_status_clear(int device);

}  // namespace goph
