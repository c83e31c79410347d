// C[M,N] = A[M,K] * W[N,K]^T in 32 bits on the fifth-generation tensor cores.
//
// A float is the sum of three bfloat16 numbers, its 24 bits eight at a time.  Of the nine products of such
// parts the six that are 2^-16 or more of the whole are made (tcgen05.mma kind::f16): the leading
// one into one accumulator, the others into two more, since a tensor-core accumulator is cut off rather
// than rounded and every sum into it costs half a bit of its last place, all on the same side where products have one
// sign.  After 128 positions of K, however long it is, the three are read out of tensor memory and added, rounded
// to nearest, to the sums in registers.  Error against 64 bits (2-norm over 2-norm; the FMA kernel of gemm_f32.cu in
// brackets): normal operands 1.3e-7 (3.9e-7) at K = 1,024, 1.4e-7 (1.1e-6) at 8,192, 1.6e-7 (2.1e-6) at 28,672; operands of
// one sign 1.75e-7 at every K (2.3e-7, 7.1e-7, 1.3e-6).  With sums of 512 positions at K = 8,192 those took 8.9e-7; with sums of 64
// they have 9.3e-8, and the product takes 1.4 times as long.
//
// A CTA has 128 rows of W (the M side of the product, lanes of tensor memory) and BN rows of A (the
// N side, columns).  Two groups of eight warps, one for the even and one for the odd k-blocks of 64,
// read both operands straight into registers, a block of their own ahead, cut them into their
// parts, put these into the group's stage in shared memory in the layout the products read (K-major,
// 128-byte swizzle) and add up the slices; one more warp issues the products.
//
// Every element is the sum, in this order, of its slices of K, which the two matrices' widths cut.  Where there are few
// tiles, the CTAs of a cluster share K slice by slice, keep each slice's sum and add them in the same
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
// Measured, against the FMA kernel: [448, 2048] x [3072, 2048] 55 (177) us, [50, 2048] x [16384, 2048] 44 (128),
// [7, 2048] x [16384, 2048] 39 (57), [1, 2048] x [3072, 2048] 17 (20); with a long K [256, 8192] x [3072, 8192] 150 (422), [1, 8192] x
// [3072, 8192] 41 (70).  One row of 4,100 to 9,400 columns and K up to 2,048 is slower: [1, 2048] x [5632, 2048] 25 (22).  What
// several slices cost a CTA that has them all: [448, 3072] x [3072, 3072] takes 89 us, 75 if K were one slice, since the sums that
// wait in shared memory leave L1 and registers short; a second set in registers 83, waiting in C for more than one
// slice 102.  Slower too: a warpgroup of its own for the sums, blocks of 32 in five stages (70 us where this takes 55), three
// stages of 64, leading products alone read out every 128 positions (the issuer's loop is what all wait for: 58).
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
// A tensor-core sum runs over a pair of k-blocks, 128 positions, whatever K is.  Pairs are added up in slices of K, which
// are what CTAs can share, and these in their order: a pair each up to K = 2,048; of a longer K as many as CTAs can
// share K with a tile each of W and no more rows of A than a tile has, on 148 SMs less what GPCs leave over.
__host__ __device__ constexpr bool is_long(int k) { return k > 2048; }
__host__ __device__ constexpr int pairs_of(int k) { return (k + 2 * BK - 1) / (2 * BK); }
int slices_of(int n, int k) {
    const int tiles = (n + BW - 1) / BW;
    return !is_long(k) ? pairs_of(k) : tiles <= 13 ? 8 : tiles <= 32 ? 4 : tiles <= 74 ? 2 : 1;
}
__host__ __device__ constexpr int slice_start(int s, int slices, int pairs) { return s * pairs / slices; }
// What a CTA does with the sums of pairs and slices: it has all of K and adds pairs to a sum in registers (ALL); of a long
// K in two slices the first one's sum waits in C for the second's (HALVES), of more they wait in shared memory
// (OUTSIDE; few registers are left).  CTAs that share K have an accumulator a pair and read none before the end
// (RAW), or where these do not fit keep the slices' sums in tensor memory behind two accumulators (KEPT).
enum Mode { ALL, HALVES, OUTSIDE, RAW, KEPT };
constexpr int W_PLANE = BW * 128;     // bytes of a part of the W tile

__host__ __device__ constexpr int stage_bytes(int bn) { return 3 * (W_PLANE + bn * 128); }
constexpr int smem_bytes(int bn, Mode mode) { return 2 * stage_bytes(bn) + (mode == OUTSIDE ? bn * BW * 4 : 0) + 1024; }

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

__device__ __forceinline__ void tc_st(uint32_t taddr, const float (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(taddr), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3])
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

template <int BN, Mode MODE>
__global__ void __launch_bounds__(THREADS, 1)
sgemm_parts_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N,
                   int K, int lda, int ldw, int ldc, int cluster, int slices, uint32_t tmem_cols, int* error) {
    constexpr bool SPLIT = MODE == RAW || MODE == KEPT;
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

    const int blocks = (K + BK - 1) / BK, pairs = pairs_of(K);
    const int per = SPLIT ? (slices + cluster - 1) / cluster : slices;
    const int s0 = rank * per, my_slices = min(per, slices - s0);
    const int pair0 = SPLIT ? slice_start(s0, slices, pairs) : 0;
    const int my_pairs = SPLIT ? slice_start(s0 + my_slices, slices, pairs) - pair0 : pairs;
    const int kb0 = 2 * pair0, kb1 = min(blocks, kb0 + 2 * my_pairs);

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
        // this thread's columns of its row of a pair with this accumulator
        constexpr int STEP = PART == 8 ? 8 : 4;                  // (of 16 columns at once more would be spilled)
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
        float total[PART];
#pragma unroll
        for (int j = 0; j < PART; ++j) total[j] = 0.f;
        int done = 0;                                            // pairs added up
        bool second = false;                                     // a block of this thread's is under way
        int s = 0, s_end = 0;                                    // of a long K: the slice, its end
        if (MODE == HALVES || MODE == OUTSIDE || MODE == KEPT) s_end = slice_start(s0 + 1, slices, pairs) - pair0;
        float* outside = reinterpret_cast<float*>(smem + 2 * STAGE) + part * PART * BW + row;      // [column][row]
        const uint32_t kept = my_tmem + 6 * BN;
        auto drain = [&]() {
            const int b = done & 1;
            ok = ok && wait(ready + b * 8, (done >> 1) & 1);
            tc_fence_after_sync();
            sums(b, [&](int j, float v) { total[j] += v; });
            tc_fence_before_sync();
            arrive(drained + b * 8);
            ++done;
            if constexpr (MODE == HALVES) {
                if (done != s_end) return;
                // (where the last tile of W is shifted back the tile before has these rows)
                const int first = m0 + (warp >> 2) * PART, rows = n0 + row < (int)blockIdx.y * BW ? 0 : M - first;
                float* at = C + (size_t)first * ldc + n0 + row;
#pragma unroll
                for (int j = 0; j < PART; ++j) {
                    if (j < rows) *at = total[j];
                    at += ldc;
                    total[j] = 0.f;
                }
            }
            if constexpr (MODE == OUTSIDE || MODE == KEPT) {
                if (done != s_end) return;
#pragma unroll
                for (int j = 0; j < PART; j += 4) {
                    const float v[4] = {total[j], total[j + 1], total[j + 2], total[j + 3]};
                    if constexpr (MODE == KEPT) tc_st(kept + s * BN + j, v);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if constexpr (MODE == OUTSIDE) outside[(j + i) * BW] = (s == 0 ? 0.f : outside[(j + i) * BW]) + v[i];
                        total[j + i] = 0.f;
                    }
                }
                ++s;
                s_end = slice_start(s0 + s + 1, slices, pairs) - pair0;
            }
        };
        for (int kb = kb0 + stage; kb < kb1 && ok; kb += 2) {
            ok = fill(kb);
            // the pair before this block's, while this one's products run
            if (MODE != RAW && second) drain();
            second = true;
        }
        if constexpr (MODE != RAW)
            while (done < my_pairs && ok) drain();
        if constexpr (!SPLIT) {
            asm volatile("bar.sync 1, 512;" ::: "memory");       // all marks are made
#pragma unroll
            for (int j = 0; j < PART; ++j) {
                const int m = m0 + part * PART + j;
                if (m < M && (MODE != HALVES || n >= (int)blockIdx.y * BW)) {
                    float v = MODE == OUTSIDE ? outside[j * BW] : total[j];
                    if (MODE == HALVES) v = C[(size_t)m * ldc + n] + v;
                    if (!isfinite(v))
                        v = not_finite(w_kind[row] | a_kind[part * PART + j], A + (size_t)m * lda, W + (size_t)n * ldw, K);
                    C[(size_t)m * ldc + n] = v;
                }
            }
        } else {
            // [slice][column][row], in the stages' place: their last products are done
            float* out = reinterpret_cast<float*>(smem) + part * PART * BW + row;
            if constexpr (MODE == RAW) {
                ok = ok && wait(ready, 0);
                tc_fence_after_sync();
                for (int i = 0, at = 0; i < my_slices; ++i) {
                    const int end = slice_start(s0 + i + 1, slices, pairs) - pair0;
                    if (end == at + 1) {
                        sums(at++, [&](int j, float v) { out[(i * BN + j) * BW] = v; });
                        continue;
                    }
                    for (; at < end; ++at) sums(at, [&](int j, float v) { total[j] += v; });
#pragma unroll
                    for (int j = 0; j < PART; ++j) {
                        out[(i * BN + j) * BW] = total[j];
                        total[j] = 0.f;
                    }
                }
            } else {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                for (int i = 0; i < my_slices; ++i)
#pragma unroll
                    for (int j = 0; j < PART; j += 4) {
                        float v[4];
                        tc_ld(kept + i * BN + j, v);
                        tc_wait_ld();
#pragma unroll
                        for (int x = 0; x < 4; ++x) out[(i * BN + j + x) * BW] = v[x];
                    }
            }
        }
        if (!ok) atomicExch(error, 28);
        tc_fence_before_sync();
    } else {
        if (lane == 0) {
            constexpr uint32_t all = instr_desc_bf16(BW, 3 * BN), two = instr_desc_bf16(BW, 2 * BN);
            constexpr uint32_t one = instr_desc_bf16(BW, BN);
            bool ok = true;
            const int mine = kb1 - kb0;
            int left = 2, at = 0, st = 0;                        // blocks of the pair to come, pairs begun
            uint32_t lead = tmem, parity = 0;
            bool there = false;                                  // this block is known to be there
            for (int it = 0; it < mine; ++it) {
                const bool first = left == 2;
                // a buffer that was never used is free: the wait for the phase before its first passes
                if (MODE != RAW && first) ok = mbar_wait(drained + (at & 1) * 8, ((at >> 1) & 1) ^ 1);
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
                    if (MODE != RAW || it + 1 == mine) tc_commit(ready + (MODE == RAW ? 0 : at & 1) * 8);
                    left = 2;
                    ++at;
                    lead = MODE == RAW ? lead + 3 * BN : tmem + (at & 1) * 3 * BN;
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

// Columns of tensor memory that a CTA takes (512 there are).
int columns(int bn, int per_slices, int per_pairs, Mode mode) {
    return bn * (mode == RAW ? 3 * per_pairs : mode == KEPT ? 6 + per_slices : 6);
}
// The way for this many columns of a tile and CTAs that share K, or -1: the slices have to fit, also as floats in the
// stages' shared memory, and no CTA may be without one.
int mode_of(int bn, int cluster, int N, int K) {
    const int slices = slices_of(N, K), pairs = pairs_of(K), per = (slices + cluster - 1) / cluster;
    if (cluster == 1) return !is_long(K) || slices == 1 ? ALL : slices == 2 ? HALVES : OUTSIDE;
    if (per * bn * BW * 4 > 2 * stage_bytes(bn) || (cluster - 1) * per >= slices) return -1;
    const int per_pairs = (per * pairs + slices - 1) / slices;
    return columns(bn, per, per_pairs, RAW) <= 512 ? RAW : columns(bn, per, per_pairs, KEPT) <= 512 ? KEPT : -1;
}

template <int BN, Mode MODE>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int cluster,
           int* error, cudaStream_t s) {
    constexpr int smem = smem_bytes(BN, MODE);
    auto kernel = sgemm_parts_kernel<BN, MODE>;
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int slices = slices_of(N, K), per = (slices + cluster - 1) / cluster;
    const int need = columns(BN, per, (per * pairs_of(K) + slices - 1) / slices, MODE);
    uint32_t cols = 32;
    while ((int)cols < need) cols *= 2;
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
    cudaLaunchKernelEx(&cfg, kernel, A, W, C, M, N, K, lda, ldw, ldc, cluster, slices, cols, error);
    return launch_status();
}

}  // namespace

bool sgemm_parts_takes(const float* A, const float* W, int N, int K, int lda, int ldw) {
    return N >= BW && K >= (N > 74 * BW ? 512 : 1024) && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}

int sgemm_parts(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int bn,
                int cluster, int* error, cudaStream_t s) {
    const int blocks = (K + BK - 1) / BK;
    if (bn <= 0) {
        // Microseconds, from measured products: 6 for the start and end of a tile, 1.1 (BN 16) to 1.5
        // (BN 80) a k-block, 4 for adding up a cluster's sums; clusters of 4 and 8 leave SMs of a
        // GPC over.  Of 60 products of 1 to 1,000 rows it chose one that was slower than the best by 10 % twice.
        const int sms = device_sm_count();
        double best = 1e30;
        for (int b : {16, 32, 48, 64, 80})
            for (int c : {1, 2, 4, 8}) {
                if (mode_of(b, c, N, K) < 0) continue;
                const long long ctas = (long long)((M + b - 1) / b) * ((N + BW - 1) / BW) * c;
                const int there = c == 8 ? sms * 3 / 4 : c == 4 ? sms * 7 / 8 : sms;
                const double block = 0.9 + 0.0075 * b > 1.1 ? 0.9 + 0.0075 * b : 1.1;
                const double t = (double)((ctas + there - 1) / there) * ((double)blocks / c * block + 6.0) +
                                 (c > 1 ? 4.0 : 0.0);
                if (t < best) best = t, bn = b, cluster = c;
            }
    }
    const int mode = mode_of(bn, cluster, N, K);
#define GO(B, MODE) \
    if (bn == B && mode == MODE) return launch<B, MODE>(A, W, C, M, N, K, lda, ldw, ldc, cluster, error, s);
#define CASE(B) GO(B, ALL) GO(B, HALVES) GO(B, OUTSIDE) GO(B, RAW) GO(B, KEPT)
    CASE(16)
    CASE(32)
    CASE(48)
    CASE(64)
    GO(80, ALL) GO(80, HALVES) GO(80, OUTSIDE) GO(80, RAW)          // (80 columns leave no tensor memory to keep slices in)
#undef CASE
#undef GO
    return -1;
}

// The same with the columns of a tile and the CTAs that share K given, for measurements and tests.
MSTAR_API int mstar_sgemm_parts(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                int ldc, int bn, int cluster, int* error, void* stream) {
    if (!sgemm_parts_takes(A, W, N, K, lda, ldw)) return -1;
    return sgemm_parts(A, W, C, M, N, K, lda, ldw, ldc, bn, cluster, error, (cudaStream_t)stream);
}
