// The 32-bit product on the tensor cores (gemm_split_tcgen05.cu), for gemm_simt.cu.
#pragma once

#include <cuda_runtime.h>

// Whether products with these weights (fp32, [N, K]) are made there.  For all M alike: the two forms round differently.
bool gemm_split_takes(const void* W, int N, int K);
// err: device int set to 1 when a bounded wait ran out (may be null); the result is right even then.
int gemm_split(const float* A, const float* W, const void* bias, int bias_dtype, float* C, int M, int N, int K, int lda, int ldc, int* err,
               cudaStream_t s);
