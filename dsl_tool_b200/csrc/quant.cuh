// Host launchers of the quantise / scale-pack kernels (definitions in quant.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dslgemm.h"

namespace dsl {
cudaError_t launch_quant_fp8(const void* x, int dtype, long long rows, long long cols, int mode, float* scale_io,
                             int scale_given, uint8_t* q, uint32_t* ws, cudaStream_t st);
cudaError_t launch_quant_fp4(const void* x, int dtype, long long rows, long long cols, int format, float* gs_io,
                             int gs_given, uint8_t* q, uint8_t* sf, size_t sf_bytes, int sf_needs_clear,
                             const int* group_offsets, int num_groups, uint32_t* ws, cudaStream_t st);
cudaError_t launch_quant_nvfp4_per_token(const void* x, int dtype, long long rows, long long cols, float* gs_out, uint8_t* q,
                                         uint8_t* sf, size_t sf_bytes, int sf_needs_clear, const int* group_offsets,
                                         int num_groups, cudaStream_t st);
// dsl_quant_fp4 / dsl_quant_fp4_per_token (abi.cu).  rows_unpadded: only scale bytes past the last K block of a row are
// zeroed - those meet zero-filled elements in the GEMM, where a NaN pattern would spread; the bytes of rows that do not
// exist are left as they are (a row's scales touch that row of the product alone).
int quant_fp4_impl(const void* x, int dtype, long long rows, long long cols, int format, float* gs_io, int gs_given, uint8_t* q_out,
                   uint8_t* sf_out, const int* group_offsets, int groups, void* ws, bool rows_unpadded, void* stream);
int quant_fp4_per_token_impl(const void* x, int dtype, long long rows, long long cols, float* gs_out, uint8_t* q_out, uint8_t* sf_out,
                             const int* group_offsets, int groups, bool rows_unpadded, void* stream);
cudaError_t launch_pack_kn(const void* w, int dtype, int groups, int K, int N, int format, int half, float* scale_io, int scale_given,
                           uint8_t* q, uint8_t* scales, size_t scale_bytes, uint32_t* ws, cudaStream_t st);
cudaError_t launch_transpose_u8(const uint8_t* in, uint8_t* out, int R, int C, cudaStream_t st);
}  // namespace dsl
