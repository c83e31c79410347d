// C[M,N] = A[M,K] * W[N,K]^T in true 32-bit: float inputs, float FMA accumulation on
// CUDA cores, no tensor-core mode of reduced precision (gemm_f32_tc.cu: the same by parts on the tensor cores
// for wide matrices, chosen at the end of this file).  This is the matrix product
// of the float32 path of the whole model (the reference has no such path: it lets
// float matmuls run as TF32, mstar/engine/__init__.py:6).
//
// Every output element is two sequential sums over K, one of the even and one of the odd
// positions, added at the end: the pair is one packed FMA (fma.rn.f32x2: two IEEE FMAs an
// instruction, which is what the FMA pipe needs for its full rate), and both its factors lie
// side by side in the row-major operands.  All tile shapes below sum in this order, so a row's
// result does not depend on what else is in the batch.
//
// What bounds it: the shared loads that feed the FMA pipe where there are tiles for every SM (a
// thread's 8 x 4 outputs take 12 loads of 16 bytes for 64 packed FMAs; 46 of the pipe's 74
// TFLOP/s), the stream of W and the depth of the copies where there are few rows.  Both operands come by cp.async, STAGES k-blocks deep, in their own
// row-major order; rows are BK + 4 floats apart in shared memory, so that eight threads reading
// 16 bytes of eight neighbouring rows meet no bank twice, and nothing has to be transposed.
#include "common.cuh"
#include "gemm_f32.h"
#include "mma_util.cuh"

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// 4 bytes global -> shared (rows that do not lie on 16 bytes); bytes 0: zeros
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

// A block of (BM / TM) x (BN / TN) threads makes a BM x BN tile; thread (ty, tx) has rows
// ty + i (BM / TM) and columns tx + j (BN / TN).  VEC: rows of both operands start on 16 bytes
// and K is a multiple of 4.
template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
sgemm_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int TY = BM / TM, TX = BN / TN, THREADS = TY * TX, LD = BK + 4;
    constexpr int STAGE = (BM + BN) * LD;          // floats: the A rows, then the W rows
    extern __shared__ __align__(16) float sg_smem[];
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

    auto load_stage = [&](int stage, int k0) {
        float* dst = sg_smem + stage * STAGE;
        if (VEC) {
            constexpr int PER_ROW = BK / 4;
#pragma unroll
            for (int c = tid; c < (BM + BN) * PER_ROW; c += THREADS) {
                const int r = c / PER_ROW, k = k0 + (c % PER_ROW) * 4;
                const bool is_a = r < BM;
                const int row = is_a ? m0 + r : n0 + r - BM;
                const bool ok = row < (is_a ? M : N) && k < K;
                const float* src = is_a ? A : W;
                if (ok) src += (size_t)row * (is_a ? lda : ldw) + k;
                cp_async_16(smem_u32(dst + r * LD + (c % PER_ROW) * 4), src, ok ? 16 : 0);
            }
        } else if (THREADS % BK == 0) {
            // a thread keeps its place in k and walks down the rows, of A, then of W
            constexpr int STEP = THREADS / BK > 0 ? THREADS / BK : 1;
            const int k = k0 + tid % BK, r0 = tid / BK;
            const bool in = k < K;
            const float* src = A + (size_t)(m0 + r0) * lda + k;
            uint32_t to = smem_u32(dst + r0 * LD + tid % BK);
#pragma unroll 8
            for (int r = r0; r < BM; r += STEP, src += (size_t)STEP * lda, to += STEP * LD * 4) {
                const bool ok = in && m0 + r < M;
                cp_async_4(to, ok ? src : A, ok ? 4 : 0);
            }
            src = W + (size_t)(n0 + r0) * ldw + k;
            to = smem_u32(dst + (BM + r0) * LD + tid % BK);
#pragma unroll 8
            for (int r = r0; r < BN; r += STEP, src += (size_t)STEP * ldw, to += STEP * LD * 4) {
                const bool ok = in && n0 + r < N;
                cp_async_4(to, ok ? src : W, ok ? 4 : 0);
            }
        } else {
            for (int c = tid; c < (BM + BN) * BK; c += THREADS) {
                const int r = c / BK, k = k0 + c % BK;
                const bool is_a = r < BM;
                const int row = is_a ? m0 + r : n0 + r - BM;
                const bool ok = row < (is_a ? M : N) && k < K;
                const float* src = is_a ? A : W;
                if (ok) src += (size_t)row * (is_a ? lda : ldw) + k;
                cp_async_4(smem_u32(dst + r * LD + c % BK), src, ok ? 4 : 0);
            }
        }
    };

    unsigned long long acc[TM][TN];                // (sum over even k, sum over odd k)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    const int blocks = (K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < blocks) load_stage(s, s * BK);
        cp_async_commit();
    }
    for (int kb = 0; kb < blocks; ++kb) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        const int next = kb + STAGES - 1;
        if (next < blocks) load_stage(next % STAGES, next * BK);
        cp_async_commit();
        const float* as = sg_smem + (kb % STAGES) * STAGE + ty * LD;
        const float* ws = sg_smem + (kb % STAGES) * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            ulonglong2 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + i * TY * LD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(ws + j * TX * LD + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    fma2(acc[i][j], a[i].x, w.x);
                    fma2(acc[i][j], a[i].y, w.y);
                }
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * TY;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * TX;
            if (n < N)
                C[(size_t)m * ldc + n] = __uint_as_float((uint32_t)acc[i][j]) +
                                         __uint_as_float((uint32_t)(acc[i][j] >> 32));
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
static int launch_sgemm(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                        int ldw, int ldc, bool vec, cudaStream_t s) {
    constexpr int smem = STAGES * (BM + BN) * (BK + 4) * (int)sizeof(float);
    constexpr int threads = (BM / TM) * (BN / TN);
    auto kernel = vec ? sgemm_nt_kernel<BM, BN, TM, TN, BK, STAGES, true>
                      : sgemm_nt_kernel<BM, BN, TM, TN, BK, STAGES, false>;
    static bool configured[2] = {false, false};
    if (smem > 48 * 1024 && !configured[vec]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        configured[vec] = true;
    }
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    kernel<<<grid, threads, smem, s>>>(A, W, C, M, N, K, lda, ldw, ldc);
    return launch_status();
}

MSTAR_API int mstar_sgemm_nt(const float* A, const float* W, float* C, int M, int N, int K,
                             int lda, int ldw, int ldc, int* error, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    // Wide matrices of aligned rows go to the tensor cores, three bfloat16 parts a float (gemm_f32_tc.cu, with both
    // sides measured; no error word: never).  From K = 1,024 on: the start and end of a tile there take some
    // 8 us, and a row alone takes 8.7 with K = 512 where the FMAs take 6.7 to 8.0 (N = 128 to 3,072; at 1,024: 8.7 to 11 against
    // 11 to 12), while matrices alone decide, so that a row's sums are the same in every batch.  From 75 tiles of W on, where no
    // CTAs share K, from K = 512: one row of 10,240 columns 12.6 against 14.6 us (of 8,192, 64 tiles: 10.6 against 9.3).
    if (error != nullptr && sgemm_parts_takes(A, W, N, K, lda, ldw))
        return sgemm_parts(A, W, C, M, N, K, lda, ldw, ldc, 0, 0, error, s);
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
    const int sms = device_sm_count();
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    // What comes here has a short K, few columns or rows off 16 bytes.
    // Few rows: the stream of W counts, so narrow tiles with deep stages.  [1, 512] x [3072, 512] 7.6 us, 8.6 with 16
    // rows a tile, 13 with 32; [8, 2048] x [64, 2048] 19, 23 and 43.
    if (M <= 8) return launch_sgemm<8, 16, 2, 1, 128, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, s);
    // up to 32 rows: 10.6 us against 13.7 for tiles of 32 rows at [30, 512] x [3072, 512], 31 against 58 at [30, 2047] x
    // [2048, 2047] off 16 bytes; twice as wide where that still makes two blocks an SM ([30, 512] x [16384, 512]: 35 against 41)
    if (M <= 32) {
        if (tiles(16, 32) >= 2 * sms)
            return launch_sgemm<16, 32, 2, 2, 64, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, s);
        return launch_sgemm<16, 16, 2, 2, 64, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, s);
    }
    // 64 x 64 tiles with 8 x 4 outputs a thread where they give every SM more than one block (several share an SM): 46
    // us against 53 for 32 x 32 at [1536, 128] x [4096, 128], 389 against 445 at [2048, 512] x [8192, 512] (44 TFLOP/s).  Below
    // that 32 x 32 tiles: 14 against 21 us at [64, 512] x [1024, 512].
    if (tiles(64, 64) * 2 >= 3 * sms)
        return launch_sgemm<64, 64, 8, 4, 32, 3>(A, W, C, M, N, K, lda, ldw, ldc, vec, s);
    return launch_sgemm<32, 32, 4, 4, 32, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, s);
}
