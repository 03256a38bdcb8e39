// Interface of the tensor-core GEMM that keeps every operand's full precision (qgemm_exact.cu).
#pragma once

#include "qgemm.cuh"

namespace mlxq {

// Serves a batch of 17 or more tokens when the layer has 16-bit scales in groups of 32, 64 or 128, K is a multiple of
// 128 and the packed rows and the activations are 16-byte aligned: every bit width, every activation type.
bool qgemm_exact_takes(const GemmLayer& L, int x_dtype, long long x_stride, const void* x, long long T);

// Enqueues it.  cudaErrorMemoryAllocation: the scratch memory could not be had, nothing was enqueued.
cudaError_t launch_qgemm_exact(const GemmLayer& L, const GemmCall& c, cudaStream_t st, const char** why);

}  // namespace mlxq
