// C[M,N] = A[M,K] * W[N,K]^T in 32 bits on the fifth-generation tensor cores.
//
// A float is the sum of three bfloat16 numbers, its 24 bits eight at a time.  Of the nine products of such
// parts the six that are 2^-16 or more of the whole are made (tcgen05.mma kind::f16): the leading
// one into one accumulator, the others into two more, since a tensor-core accumulator is cut off rather
// than rounded and every sum into it costs half a bit of its last place.  After a slice of K (128
// positions, more from K = 2,048 on) the three are read out of tensor memory and added, rounded to nearest,
// to the sums in registers.  Error against 64 bits (2-norm over 2-norm, normal operands; the FMA kernel of
// gemm_f32.cu in brackets): 1.4e-7 (5.8e-7) at K = 2,048, 4.8e-7 (1.2e-6) at K = 8,192.  Operands of one sign
// are where the cutting off shows most: 1.7e-7 (3.3e-7) and 8.5e-7 (6.6e-7).
//
// A CTA has 128 rows of W (the M side of the product, lanes of tensor memory) and BN rows of A (the
// N side, columns).  Two groups of eight warps, one for the even and one for the odd k-blocks of 64,
// read both operands straight into registers, a block of their own ahead, cut them into their
// parts, put these into the group's stage in shared memory in the layout the products read (K-major,
// 128-byte swizzle) and add up the slices; one more warp issues the products.
//
// Every element is the sum, in this order, of its slices.  Where there are few tiles, the CTAs of a
// cluster share K slice by slice, keep each slice's sum in tensor memory and add them in the same
// order through distributed shared memory, so a row's result depends neither on what else is in
// the batch nor on how the work was cut.
//
// Operands that are not finite: a NaN anywhere in a row of either operand makes its outputs NaN, as
// it has to; where there is an infinity and no NaN the parts say nothing (infinity times a part that is
// zero), so those outputs are made again with plain FMAs.
//
// What bounds it: the way of a block through the splitters, its fence, the products and back, 1.1 us with 16
// rows of A and 1.5 with 80 where the products alone take 0.3 and 0.5; shared memory, which the splitters
// fill and the products read, and instruction slots (half of them) are what the two groups compete for.
// Measured, against the FMA kernel: [448, 2048] x [3072, 2048] 55 (183) us, [50, 2048] x [16384, 2048] 49 (129),
// [7, 2048] x [16384, 2048] 41 (57), [1, 2048] x [3072, 2048] 19 (23).  Slower: a warpgroup of its own for the sums,
// blocks of 32 in five stages (70 us where this takes 55), three stages of 64.
#include "common.cuh"
#include "tcgen05_util.cuh"
#include "tma_util.cuh"
#include "gemm_f32.h"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace {

constexpr int BW = 128;              // rows of W a CTA
constexpr int BK = 64;               // k-block: a row of a part is 128 bytes
constexpr int GROUP = 256;           // threads that fill a stage
constexpr int WORKERS = 2 * GROUP;   // then the issuer's warp
constexpr int THREADS = WORKERS + 32;
constexpr int ISSUER = WORKERS / 32;
// k-blocks a tensor-core sum runs over: 128 positions up to K = 2,048, so that at most 16 sums make an element
__host__ __device__ constexpr int slice_blocks(int k) { return 2 * ((k + 2047) / 2048); }
constexpr int W_PLANE = BW * 128;     // bytes of a part of the W tile

__host__ __device__ constexpr int stage_bytes(int bn) { return 3 * (W_PLANE + bn * 128); }
constexpr int smem_bytes(int bn) { return 2 * stage_bytes(bn) + 1024; }

// Two floats into their three parts, packed, each part rounded to nearest; t collects the last
// remainders: they are tiny unless a float was not finite, or so large that its first part is not,
// which leaves NaN or an infinity.
typedef unsigned long long pair_t;                               // two floats, the first in the lower half
__device__ __forceinline__ pair_t without(pair_t x, uint32_t part) {     // x - part, exactly
    pair_t d;
    asm("{\n\t.reg .b32 lo, hi;\n\t.reg .b64 p;\n\t"
        "shl.b32 lo, %2, 16;\n\tand.b32 hi, %2, 0xffff0000;\n\tmov.b64 p, {lo, hi};\n\t"
        "fma.rn.f32x2 %0, p, %3, %1;\n\t}"
        : "=l"(d) : "l"(x), "r"(part), "l"(0xbf800000bf800000ull));
    return d;
}
__device__ __forceinline__ uint32_t pack2(pair_t v) {
    uint32_t d;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tcvt.rn.bf16x2.f32 %0, hi, lo;\n\t}" : "=r"(d) : "l"(v));
    return d;
}
__device__ __forceinline__ void split2(pair_t x, uint32_t& h, uint32_t& m, uint32_t& l, pair_t& t) {
    h = pack2(x);
    const pair_t r = without(x, h);
    m = pack2(r);
    const pair_t s = without(r, m);
    l = pack2(s);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(t) : "l"(s));
}

// Marks rows (every 16th, `rows` of them) by what there is among their four floats at p: 2 a NaN, 1 one
// whose first part is not finite.
__device__ __forceinline__ void mark(const float* p, size_t step, int rows, uint32_t* kind) {
#pragma unroll 1
    for (int i = 0; i < rows; ++i, p += step)
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            const uint32_t is = isnan(p[j]) ? 2u : fabsf(p[j]) > 3.38e38f ? 1u : 0u;
            if (is != 0) atomicOr(kind + i * 16, is);
        }
}

// A sum that is not finite, of rows with these marks.  (Without a mark: finite numbers whose products pass the
// largest float; those of the middle parts may then be infinities of the other sign.)
__device__ __forceinline__ float not_finite(uint32_t kind, const float* a, const float* w, int K) {
    if (kind & 2) return __uint_as_float(0x7fffffffu);
    float even = 0.f, odd = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; k += 2) {          // K is a multiple of 4
        even = fmaf(a[k], w[k], even);
        odd = fmaf(a[k + 1], w[k + 1], odd);
    }
    return even + odd;
}

__device__ __forceinline__ void tc_ld(uint32_t taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_ld(uint32_t taddr, float (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3])
                 : "r"(taddr)
                 : "memory");
}

// Whether a phase is over, without waiting.
__device__ __forceinline__ bool is_over(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

template <int BN, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
sgemm_parts_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N,
                   int K, int lda, int ldw, int ldc, int cluster, uint32_t tmem_cols, int* error) {
    constexpr int STAGE = stage_bytes(BN), A_PLANE = BN * 128;
    constexpr int PART = BN / 4;                                 // columns a thread adds up
    constexpr int UW = BW * 16 / GROUP, UA = BN * 16 / GROUP;    // fours of floats a thread
    extern __shared__ uint8_t raw_smem[];
    __shared__ __align__(8) uint64_t bars[8];                    // full[2], empty[2], ready[2], drained[2]
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t w_kind[BW], a_kind[BN];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~(uintptr_t)1023);
    const uint32_t base = tc_smem(smem), bar = tc_smem(bars);
    const uint32_t full = bar, empty = bar + 16, ready = bar + 32, drained = bar + 48;
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int rank = SPLIT ? blockIdx.x % cluster : 0;
    // the last tile of W may cover rows of the one before again
    const int m0 = (SPLIT ? blockIdx.x / cluster : blockIdx.x) * BN, n0 = min((int)blockIdx.y * BW, N - BW);

    const int slice = slice_blocks(K), blocks = (K + BK - 1) / BK, slices = (blocks + slice - 1) / slice;
    const int per = SPLIT ? (slices + cluster - 1) / cluster : slices;
    const int s0 = min(rank * per, slices), my_slices = min(per, slices - s0);
    const int kb0 = s0 * slice, kb1 = min(blocks, (s0 + my_slices) * slice);

    // Splitters: four numbers of row r; a thread keeps its place in k and walks down the rows, 16 apart.
    // Rows of A past the matrix are never stored, so the last one stands in for them; numbers past K are
    // made zeros before they are used.
    const int stage = (tid / GROUP) & 1, c = tid & 15, r = (tid % GROUP) >> 4;
    ulonglong2 w_next[UW], a_next[UA];
    const float *w_at, *a_at;
    const bool inside = m0 + BN <= M;
    auto look_at = [&](int kb) {
        const int k = min(kb * BK + c * 4, K - 4);
        w_at = W + (size_t)(n0 + r) * ldw + k;
        a_at = A + (size_t)(inside ? m0 + r : 0) * lda + k;
    };
    // (read past L1, which the stages leave little of)
    auto load_w = [&](int u) {
        asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0, %1}, [%2];"
                     : "=l"(w_next[u].x), "=l"(w_next[u].y)
                     : "l"(w_at + (size_t)u * 16 * ldw));
    };
    auto load_a = [&](int u) {
        const size_t row = inside ? u * 16 : min(m0 + r + u * 16, M - 1);
        a_next[u] = __ldg(reinterpret_cast<const ulonglong2*>(a_at + row * lda));
    };
    if (tid < WORKERS) {
        look_at(min(kb0 + stage, blocks - 1));
#pragma unroll
        for (int u = 0; u < UW; ++u) load_w(u);
#pragma unroll
        for (int u = 0; u < UA; ++u) load_a(u);
    }

    if (tid == WORKERS) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(full + i * 8, GROUP / 32);
            mbar_init(empty + i * 8, 1);
            mbar_init(ready + i * 8, 1);
            mbar_init(drained + i * 8, WORKERS / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < BW + BN; i += THREADS) (i < BW ? w_kind[i] : a_kind[i - BW]) = 0;
    if (warp == ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;

    // one lane asks for its warp, and arrives for it
    auto wait = [&](uint32_t at, uint32_t parity) {
        const int ok = lane == 0 ? mbar_wait(at, parity) : 0;
        return __shfl_sync(0xffffffffu, ok, 0) != 0;
    };
    auto arrive = [&](uint32_t at) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(at) : "memory");
    };

    if (tid < WORKERS) {
        const uint32_t place = (uint32_t)(r * 128 + (((c >> 1) ^ (r & 7)) << 4) + (c & 1) * 8);
        auto put = [&](uint8_t* to, int plane, const ulonglong2 v, pair_t& t) {
            uint2 h, m, l;
            split2(v.x, h.x, m.x, l.x, t);
            split2(v.y, h.y, m.y, l.y, t);
            *reinterpret_cast<uint2*>(to) = h;
            *reinterpret_cast<uint2*>(to + plane) = m;
            *reinterpret_cast<uint2*>(to + 2 * plane) = l;
        };
        uint32_t parity = 1;                                     // of a stage that was never filled
        auto fill = [&](int kb) {
            if (kb * BK + c * 4 >= K) {                          // a last block that ends inside
#pragma unroll
                for (int u = 0; u < UW; ++u) w_next[u] = make_ulonglong2(0, 0);
#pragma unroll
                for (int u = 0; u < UA; ++u) a_next[u] = make_ulonglong2(0, 0);
            }
            const bool ok = wait(empty + stage * 8, parity);
            parity ^= 1;
            uint8_t* to = smem + stage * STAGE + place;
            // a number's place is free for a later block's as soon as its parts are made
            look_at(min(kb + 2, blocks - 1));
            pair_t t = 0;
#pragma unroll
            for (int u = 0; u < UW; ++u) {
                put(to + u * 16 * 128, W_PLANE, w_next[u], t);
                load_w(u);
            }
#pragma unroll
            for (int u = 0; u < UA; ++u) {
                put(to + 3 * W_PLANE + u * 16 * 128, A_PLANE, a_next[u], t);
                load_a(u);
            }
            if (!isfinite(__uint_as_float((uint32_t)t) + __uint_as_float((uint32_t)(t >> 32)))) {
                const int k = kb * BK + c * 4;
                mark(W + (size_t)(n0 + r) * ldw + k, (size_t)16 * ldw, UW, &w_kind[r]);
                mark(A + (size_t)(m0 + r) * lda + k, (size_t)16 * lda, (min(BN, M - m0) - r + 15) / 16, &a_kind[r]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            arrive(full + stage * 8);
            return ok;
        };
        // this thread's columns of its row of a slice whose accumulators begin at a column
        constexpr int STEP = PART % 8 == 0 ? 8 : 4;
        const int row = (warp & 3) * 32 + lane, part = warp >> 2, n = n0 + row;
        const uint32_t my_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + part * PART;
        auto sums = [&](int b, auto&& use) {
#pragma unroll
            for (int j = 0; j < PART; j += STEP) {
                float lead[STEP], rest[STEP], more[STEP];
                tc_ld(my_tmem + b * 3 * BN + j, lead);
                tc_ld(my_tmem + b * 3 * BN + BN + j, rest);
                tc_ld(my_tmem + b * 3 * BN + 2 * BN + j, more);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < STEP; ++i) use(j + i, lead[i] + (rest[i] + more[i]));
            }
        };
        bool ok = true;
        if constexpr (!SPLIT) {
            float total[PART];
#pragma unroll
            for (int j = 0; j < PART; ++j) total[j] = 0.f;
            int done = 0, left = slice;                          // slices added up, blocks to the next one
            auto drain = [&]() {
                const int b = done & 1;
                ok = ok && wait(ready + b * 8, (done >> 1) & 1);
                tc_fence_after_sync();
                sums(b, [&](int j, float v) { total[j] += v; });
                tc_fence_before_sync();
                arrive(drained + b * 8);
                ++done;
            };
            for (int kb = kb0 + stage; kb < kb1 && ok; kb += 2) {
                ok = fill(kb);
                // the slice before this block's, while this one's products run
                if (left == 0) {
                    drain();
                    left = slice;
                }
                left -= 2;
            }
            while (done < my_slices && ok) drain();
            asm volatile("bar.sync 1, 512;" ::: "memory");       // all marks are made
#pragma unroll
            for (int j = 0; j < PART; ++j) {
                const int m = m0 + part * PART + j;
                if (m < M) {
                    if (!isfinite(total[j]))
                        total[j] = not_finite(w_kind[row] | a_kind[part * PART + j], A + (size_t)m * lda,
                                              W + (size_t)n * ldw, K);
                    C[(size_t)m * ldc + n] = total[j];
                }
            }
        } else {
            for (int kb = kb0 + stage; kb < kb1 && ok; kb += 2) ok = fill(kb);
            ok = ok && wait(ready, 0);
            tc_fence_after_sync();
            float* out = reinterpret_cast<float*>(smem);         // [slice][column][row], in the stages' place
            for (int s = 0; s < my_slices; ++s)
                sums(s, [&](int j, float v) { out[(s * BN + part * PART + j) * BW + row] = v; });
        }
        if (!ok) atomicExch(error, 28);
        tc_fence_before_sync();
    } else {
        if (lane == 0) {
            constexpr uint32_t all = instr_desc_bf16(BW, 3 * BN), two = instr_desc_bf16(BW, 2 * BN);
            constexpr uint32_t one = instr_desc_bf16(BW, BN);
            bool ok = true;
            const int mine = kb1 - kb0;
            int left = slice, at = 0, st = 0;                    // blocks of the slice to come, slices begun
            uint32_t lead = tmem, parity = 0;
            bool there = false;                                  // this block is known to be there
            for (int it = 0; it < mine; ++it) {
                const bool first = left == slice;
                // a buffer that was never used is free: the wait for the phase before its first passes
                if (!SPLIT && first) ok = mbar_wait(drained + (at & 1) * 8, ((at >> 1) & 1) ^ 1);
                if (!there) ok = ok && mbar_wait(full + st * 8, parity);
                if (!ok) break;
                const int next = st ^ 1;
                const uint32_t next_parity = parity ^ (next == 0);
                // asked before the products are issued: the answer takes some 500 cycles where the splitters
                // keep shared memory busy
                there = it + 1 < mine && is_over(full + next * 8, next_parity);
                tc_fence_after_sync();
                const uint64_t w = smem_desc_sw128(base + st * STAGE), a = smem_desc_sw128(base + st * STAGE + 3 * W_PLANE);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) {
                    tc_mma(lead, w + k * 2, a + k * 2, all, !first || k > 0);                    // high x (high | middle | low)
                    tc_mma(lead + BN, w + k * 2 + (W_PLANE >> 4), a + k * 2, two, 1);            // middle x (high | middle)
                    tc_mma(lead + BN, w + k * 2 + 2 * (W_PLANE >> 4), a + k * 2, one, 1);        // low x high
                }
                tc_commit(empty + st * 8);
                if (--left == 0 || it + 1 == mine) {
                    if (!SPLIT || it + 1 == mine) tc_commit(ready + (SPLIT ? 0 : at & 1) * 8);
                    left = slice;
                    ++at;
                    lead = SPLIT ? lead + 3 * BN : tmem + (at & 1) * 3 * BN;
                }
                st = next;
                parity = next_parity;
            }
            if (!ok) atomicExch(error, 29);
        }
        __syncwarp();
    }
    if (SPLIT) {
        cg::cluster_group cl = cg::this_cluster();
        float* part = reinterpret_cast<float*>(smem);
        cl.sync();
        if (tid < WORKERS) {
            const int row = tid % BW, n = n0 + row;
            for (int col = rank * 4 + tid / BW; col < BN && m0 + col < M; col += 4 * cluster) {
                float v = 0.f;
                int s = 0;
                for (int q = 0; q < cluster; ++q) {
                    const float* from = cl.map_shared_rank(part, q) + col * BW + row;
                    for (int i = 0; i < per && s < slices; ++i, ++s) v += from[i * BN * BW];
                }
                if (!isfinite(v)) {
                    uint32_t kind = 0;
                    for (int q = 0; q < cluster; ++q)
                        kind |= cl.map_shared_rank(w_kind, q)[row] | cl.map_shared_rank(a_kind, q)[col];
                    v = not_finite(kind, A + (size_t)(m0 + col) * lda, W + (size_t)n * ldw, K);
                }
                C[(size_t)(m0 + col) * ldc + n] = v;
            }
        }
        cl.sync();
    }
    __syncthreads();
    if (warp == ISSUER) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
}

int slices_of(int K) { return ((K + BK - 1) / BK + slice_blocks(K) - 1) / slice_blocks(K); }

template <int BN, bool SPLIT>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int cluster,
           int* error, cudaStream_t s) {
    constexpr int smem = smem_bytes(BN);
    auto kernel = sgemm_parts_kernel<BN, SPLIT>;
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int slices = slices_of(K), per = (slices + cluster - 1) / cluster;
    uint32_t cols = 32;
    while (cols < (uint32_t)(3 * BN * (SPLIT ? per : 2))) cols *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((M + BN - 1) / BN * cluster), (unsigned)((N + BW - 1) / BW));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)cluster, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, A, W, C, M, N, K, lda, ldw, ldc, cluster, cols, error);
    return launch_status();
}

// Whether BN columns and a cluster of this size hold all slices of a CTA: in tensor memory (512 columns)
// and, as floats, in the stages' shared memory.
bool fits(int bn, int cluster, int slices) {
    if (cluster == 1) return true;
    const int per = (slices + cluster - 1) / cluster;
    return 3 * bn * per <= 512 && per * bn * BW * 4 <= 2 * stage_bytes(bn) &&
           (cluster - 1) * per < slices;
}

}  // namespace

bool sgemm_parts_takes(const float* A, const float* W, int N, int K, int lda, int ldw) {
    return N >= BW && K >= 512 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}

int sgemm_parts(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int bn,
                int cluster, int* error, cudaStream_t s) {
    const int slices = slices_of(K);
    if (bn <= 0) {
        // Microseconds, from measured products: 6 for the start and end of a tile, 1.1 (BN 16) to 1.5
        // (BN 80) a k-block, 4 for adding up a cluster's sums; clusters of 4 and 8 leave SMs of a
        // GPC over.  It gives 18 for [1, 2048] x [3072, 2048] (measured: 19), 45 for [50, 8192] x [2048, 8192] (45),
        // 53 for [448, 2048] x [3072, 2048] (55).
        const int sms = device_sm_count();
        double best = 1e30;
        for (int b : {16, 32, 48, 64, 80})
            for (int c : {1, 2, 4, 8}) {
                if (!fits(b, c, slices)) continue;
                const int per = (slices + c - 1) / c;
                const long long ctas = (long long)((M + b - 1) / b) * ((N + BW - 1) / BW) * c;
                const int there = c == 8 ? sms * 3 / 4 : c == 4 ? sms * 7 / 8 : sms;
                const double block = 0.9 + 0.0075 * b > 1.1 ? 0.9 + 0.0075 * b : 1.1;
                const double t = (double)((ctas + there - 1) / there) * (per * slice_blocks(K) * block + 6.0) +
                                 (c > 1 ? 4.0 : 0.0);
                if (t < best) best = t, bn = b, cluster = c;
            }
    } else if (!fits(bn, cluster, slices)) {
        return -1;
    }
#define CASE(B)                                                                                                   \
    case B:                                                                                                       \
        return cluster > 1 ? launch<B, true>(A, W, C, M, N, K, lda, ldw, ldc, cluster, error, s)                  \
                           : launch<B, false>(A, W, C, M, N, K, lda, ldw, ldc, 1, error, s);
    switch (bn) {
        CASE(16)
        CASE(32)
        CASE(48)
        CASE(64)
        CASE(80)
    }
#undef CASE
    return -1;
}

// The same with the columns of a tile and the CTAs that share K given, for measurements and tests.
MSTAR_API int mstar_sgemm_parts(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                int ldc, int bn, int cluster, int* error, void* stream) {
    if (!sgemm_parts_takes(A, W, N, K, lda, ldw)) return -1;
    return sgemm_parts(A, W, C, M, N, K, lda, ldw, ldc, bn, cluster, error, (cudaStream_t)stream);
}
