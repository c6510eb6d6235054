// GEMM for few rows (gemm_skinny.cu), called by the dispatch of gemm_ops.cu.
#pragma once
#include <cuda_runtime.h>

#include "iris/host_api.h"

// C = A @ B (+ bias) for M <= 256; operands and bias as in IrisGemmDesc. 0 or a negative error code.
int iris_gemm_skinny(const IrisGemmDesc* d, cudaStream_t stream);
// 1 when the local GEMM of this descriptor goes to that kernel, else 0.
extern "C" int iris_gemm_skinny_takes(const IrisGemmDesc* d);
// CTAs that share one column tile's K for this shape (the cluster size).
int iris_gemm_skinny_split(int M, int N, int K);
