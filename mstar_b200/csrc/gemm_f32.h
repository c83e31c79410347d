// The 32-bit product on tensor cores (gemm_f32_tc.cu), for the dispatch in gemm_f32.cu, and that dispatch, for
// kernels whose launch begins with such a product.
#pragma once

#include <cuda_runtime.h>

// By the matrices alone, never by the number of rows of A: a row's sums are the same in every batch.
bool sgemm_parts_takes(const float* A, const float* W, int N, int K, int lda, int ldw);
// bn: rows of A a tile (16, 32, 48, 64 or 80; 0: chosen by the sizes), cluster: CTAs that share K.
int sgemm_parts(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int bn,
                int cluster, int* error, cudaStream_t s);

// C[M,N] = A[M,K] W[N,K]^T in 32 bits (gemm_f32.cu); error: null, or the device word of bounded waits.
extern "C" __attribute__((visibility("default"))) int mstar_sgemm_nt(const float* A, const float* W, float* C, int M,
                                                                     int N, int K, int lda, int ldw, int ldc,
                                                                     int* error, void* stream);
