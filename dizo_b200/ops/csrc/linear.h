// out[M,N] = act((A W^T + bias) * out_scale) + residual: one rule for which GEMM kernel takes a shape.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

extern "C" int dz_linear(const void* A, long long lda, const void* W, long long ldw, void* out, long long ldo,
                         const void* bias, const void* residual, long long ldr, int M, int N, int K, int act,
                         int out_fp32, float out_scale, uint32_t* err, cudaStream_t stream);
