// Attention of prompt portions on the fifth-generation tensor cores (tcgen05) for the attentions
// whose probabilities are not rounded to bfloat16, in two forms that share everything but where
// their keys and values come from:
//
//   paged    the window attention of attention_sink.cu (kept first keys, chunks, soft cap, sink,
//            score bias, sigmoid weights, gates) over the paged cache, key and value size 64 or 128;
//            rows are (token, query head of the group) pairs;
//   latent   the latent attention of attention_latent.cu for prompts: the keys and values of every
//            head are made from the latents first (one product, below), so that a query and a key
//            meet in dim + rot features and a probability and a value in dim, instead of the
//            rank + rot and rank features of the folded form; rows are tokens of one head.
//
// What is float in those kernels goes through the tensor cores in as many bfloat16 parts (a head and
// remainders) as there, and the parts' products meet in the float accumulator: the probabilities of both
// forms in three (24 bits: P = P0 + P1 + P2, all times V), and, of the latent form, the keys in two, as the
// folded query (q K0 + q K1; the rotated key features and the queries are bfloat16 numbers).  The latent
// form's values have two as well ((P0 + P1 + P2) V0 + (P0 + P1) V1; the folded form rounds its weighted sum
// of latents to one).
//
// The CTA is that of attention_prefill_tc.cu: 128 rows, tiles of 64 keys, a key and a value producer
// warp (TMA, two stages each), a warp that issues S = Q K^T a tile ahead into one of two buffers in
// tensor memory, 128 softmax threads of a row each that write P over S, a warp that issues O += P V.
// What differs: two parts of P fill the whole of their S buffer (64 columns), the third lies behind them
// where the CTA's share of tensor memory has room (96 columns a buffer) and in shared memory where not
// (keys and values of 128 in the paged form: two CTAs an SM), each row masks by its own range, scores pass the cap, and the tiles that hold keys no row of the CTA sees (before a
// window, past the last key) have those keys' values zeroed in shared memory before the product, so
// that what lies there, other requests' numbers or none, cannot reach a sum.
//
// With few row tiles the keys of a tile are shared among `splits` CTAs whose unnormalised partials
// (o, maximum, sum) a second kernel merges.  Every mbarrier wait is bounded; a timeout is recorded
// in the error word.
//
// Bound, in the paged form with a cap, by the softmax warps' arithmetic (2,048 tokens with 16 / 4 heads
// of 128: 72 us; 59 with probabilities in two parts, which are 16 bits; the mma.sync kernel 233; tanh from
// the exponential unit alone instead of its series where scores are small, and running maxima under a low
// cap, cost 9 us), in the latent form by the tensor pipe (33 us of products for 2,048 tokens and 16 heads of
// 128 + 64 where the kernel takes 61, and 52 with two parts; making the keys and values 28; the folded form
// on mma.sync, 3.4 times the work, 1,912).
#include <string.h>

#include "attention_tc_util.cuh"
#include "common.cuh"
#include "mma_util.cuh"

#define PA_ROWS 128
#define PA_KEYS 64
#define PA_THREADS 256  // 4 softmax warps, the S-issuing warp, the key warp, the O-issuing warp, the value warp
#define PA_BLOCK (PA_KEYS * 128)    // bytes of 64 keys x 64 features
// As in attention_prefill_tc.cu: a row's reference maximum follows the tile maxima only when they
// exceed it by more than 2^8.
#define PA_MAX_SLACK 8.0f
#define PA_NO_MAX (-1e30f)          // reference maximum of a row that has seen no key

struct PromptArgs {
    const int* block_table;
    const int* qo_indptr;
    const int* kv_len;
    bf16* out;
    float* scratch;
    const float* gate;      // null, or one number a head or (gate_features) a feature
    const float* sink;      // null, or one number a query head
    const float* bias;      // null, or one number a query head
    int bt_stride, nq, nkv, page_size, first_entry, entries;
    int window, keep_first, chunk;      // 0: none
    int splits, row_tiles, fold, gate_stride, gate_features, gate_vec;
    float scale_log2e;
    float cap_in, cap_log2e;            // 2 log2(e) scale / cap and cap log2(e)
    float cap_z;                        // scale / cap
    int cap_bounds;                     // the cap is low enough to be every row's reference maximum
    int rot_x;                          // latent form: first rotated feature of a latent row
    int out_heads;                      // heads of a row of `out` (the launch may write some of them)
};

__device__ __forceinline__ float pa_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two floats in a register pair, and operations on both at once.
typedef unsigned long long pa_f2;
__device__ __forceinline__ pa_f2 pa_pack(float lo, float hi) {
    return (pa_f2)__float_as_uint(lo) | ((pa_f2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float pa_lo(pa_f2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float pa_hi(pa_f2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ pa_f2 pa_mul2(pa_f2 a, pa_f2 b) {
    pa_f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ pa_f2 pa_fma2(pa_f2 a, pa_f2 b, pa_f2 c) {
    pa_f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ pa_f2 pa_add2(pa_f2 a, pa_f2 b) {
    pa_f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// tanh for |z| <= 1/2 by its Taylor series to z^13 (the next term is under 1e-7 of the result there)
__device__ __forceinline__ pa_f2 pa_tanh2(pa_f2 z) {
    const pa_f2 u = pa_mul2(z, z);
    const auto c = [](double v) { return pa_pack((float)v, (float)v); };
    pa_f2 p = pa_fma2(u, c(21844.0 / 6081075.0), c(-1382.0 / 155925.0));
    p = pa_fma2(u, p, c(62.0 / 2835.0));
    p = pa_fma2(u, p, c(-17.0 / 315.0));
    p = pa_fma2(u, p, c(2.0 / 15.0));
    p = pa_fma2(u, p, c(-1.0 / 3.0));
    return pa_fma2(pa_mul2(z, u), p, z);
}
// the lowest n bits of 32 (none for n <= 0, all for n >= 32)
__device__ __forceinline__ uint32_t pa_first(int n) { return n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u; }
// Takes the bfloat16 heads off a pair of floats: returns them packed and leaves the remainders (exact).
__device__ __forceinline__ uint32_t pa_take_part(pa_f2& x) {
    const __nv_bfloat162 head2 = __floats2bfloat162_rn(pa_lo(x), pa_hi(x));
    const uint32_t bits = *reinterpret_cast<const uint32_t*>(&head2);
    x = pa_fma2(pa_pack(__uint_as_float(bits << 16), __uint_as_float(bits & 0xffff0000u)), pa_pack(-1.f, -1.f), x);
    return bits;
}
__device__ __forceinline__ float pa_sigmoid(float g) { return 1.f / (1.f + expf(-g)); }

// The latent form's keys lie request after request: those of entry e (of the launch) start at row
// pa_latent_base(e), its first one at position pa_latent_first(e), a multiple of the key tile.
__host__ __device__ __forceinline__ int pa_latent_first(int past, int window) {
    return window > 0 && past >= window ? (past - window + 1) / PA_KEYS * PA_KEYS : 0;
}
__device__ __forceinline__ int pa_latent_base(const int* qo_indptr, const int* kv_len, int first_entry, int e,
                                              int window) {
    int base = 0;
    for (int i = first_entry; i < first_entry + e; ++i)
        base += kv_len[i] - pa_latent_first(kv_len[i] - (qo_indptr[i + 1] - qo_indptr[i]), window);
    return base;
}

template <int HD, bool LATENT> struct PromptShape {
    static constexpr int NB = HD / 64;                       // 64-feature blocks of a value
    static constexpr int QB = LATENT ? NB + 1 : NB;          // ... of a query (plain features, rotated ones)
    static constexpr int KB = LATENT ? 2 * NB + 1 : NB;      // ... of a key: heads, remainders, rotated
    static constexpr int VB = LATENT ? 2 * NB : NB;          // ... of a value: heads, remainders
    static constexpr int Q_BYTES = QB * PA_ROWS * 128, K_BYTES = KB * PA_BLOCK, V_BYTES = VB * PA_BLOCK;
    // the third part of P: behind the others in tensor memory, or (one buffer) in shared memory
    static constexpr bool P2_SMEM = !LATENT && HD == 128;
    static constexpr int P_COLS = P2_SMEM ? 64 : 96;         // tensor-memory columns of an S / P buffer
    static constexpr int TMEM_COLS = 2 * P_COLS + HD <= 256 ? 256 : 512;
    static constexpr int P2_BYTES = P2_SMEM ? PA_ROWS * 128 : 0;
    static constexpr int SMEM = Q_BYTES + 2 * (K_BYTES + V_BYTES) + P2_BYTES + 128;
    // no more CTAs on an SM than its 512 TMEM columns serve (two of 256, or one of 512)
    static constexpr int SMEM_LAUNCH = SMEM < 77 * 1024 ? 77 * 1024 : SMEM;
    static_assert(TMEM_COLS == 256 || SMEM_LAUNCH > 114 * 1024, "two CTAs would want more tensor memory than there is");
};

template <int HD, bool LATENT, bool CAP, bool SIGMOID>
__global__ void __launch_bounds__(PA_THREADS, PromptShape<HD, LATENT>::TMEM_COLS == 256 ? 2 : 1)
prompt_attention_kernel(const __grid_constant__ CUtensorMap kv_map, const __grid_constant__ CUtensorMap rot_map,
                        const __grid_constant__ CUtensorMap q_map, PromptArgs a, int* __restrict__ error_word) {
    using Shape = PromptShape<HD, LATENT>;
    constexpr int NB = Shape::NB, QB = Shape::QB, KB = Shape::KB, VB = Shape::VB;
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    unsigned char* q_s = smem_dyn;
    unsigned char* k_s = q_s + Shape::Q_BYTES;          // [2 stages]
    unsigned char* v_s = k_s + 2 * Shape::K_BYTES;      // [2 stages]
    unsigned char* p2_s = v_s + 2 * Shape::V_BYTES;     // (the third part of P, where it lies here)
    uint64_t* bars = reinterpret_cast<uint64_t*>(p2_s + Shape::P2_BYTES);
    // k_full[2], v_full[2]: a stage's copies have landed.  k_empty[2]: S of the stage's tile is done.
    // v_empty[2]: O += P V of the stage's tile is done.  s_full[2]: S of a tile is done.  p_ready[2]:
    // P of a tile is written (one arrival per softmax thread).  One phase per two tiles.
    const uint32_t k_full = tc_smem(bars + 0), v_full = tc_smem(bars + 2), k_empty = tc_smem(bars + 4),
                   v_empty = tc_smem(bars + 6), p_ready = tc_smem(bars + 8), s_full = tc_smem(bars + 10),
                   q_ready = tc_smem(bars + 12);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);

    // grid: x (split, kv head, row tile), the last row tile first (the most keys, where there are no chunks); z
    // the entry.  `fold`: all
    // CTAs run at once, two an SM: from this rank on the order is turned round, so that the CTA that
    // shares its SM with the longest is the shortest.
    int rank = blockIdx.x;
    const int split = rank % a.splits;
    rank /= a.splits;
    if (a.fold > 0 && rank >= a.fold) rank = a.fold + a.row_tiles * a.nkv - 1 - rank;
    const int kvh = rank % a.nkv, tile = a.row_tiles - 1 - rank / a.nkv;
    const int e = a.first_entry + blockIdx.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = a.nq / a.nkv;
    const int TPT = PA_ROWS / G, RPT = TPT * G;         // tokens and rows of a tile
    const int q_start = a.qo_indptr[e];
    const int q_len = a.qo_indptr[e + 1] - q_start;
    const int tok0 = tile * TPT;
    if (tok0 >= q_len) return;
    if ((tc_smem(smem_dyn) & 1023u) != 0) {             // the swizzled tiles need this alignment
        if (tid == 0) atomicExch(error_word, 22);
        return;
    }
    const int past = a.kv_len[e] - q_len;
    const int hi = past + min(q_len, tok0 + TPT);       // keys below hi are visible to some row
    // the oldest key that the window (or chunk) of a cache position holds
    auto window_lo = [&](int cp) {
        return a.chunk > 0 ? cp / a.chunk * a.chunk : a.window > 0 ? max(0, cp - a.window + 1) : 0;
    };
    const int lo = window_lo(past + tok0);
    // tiles of keys: those of the kept first keys that lie before the window's, then the window's
    const int lo_tile = lo / PA_KEYS;
    const int kept_tiles = min((min(a.keep_first, lo) + PA_KEYS - 1) / PA_KEYS, lo_tile);
    const int all_tiles = kept_tiles + (hi + PA_KEYS - 1) / PA_KEYS - lo_tile;
    const int per_split = (all_tiles + a.splits - 1) / a.splits;
    const int first_tile = split * per_split;
    const int ntiles = max(0, min(all_tiles, first_tile + per_split) - first_tile);
    auto tile_key = [&](int j) {
        const int t = first_tile + j;
        return (t < kept_tiles ? t : lo_tile + t - kept_tiles) * PA_KEYS;
    };

    if (tid == 0) {
        for (int i = 0; i < 13; ++i) mbar_init(tc_smem(bars + i), i == 8 || i == 9 ? 128 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid >= RPT && tid < PA_ROWS) {
        // rows of the tile that the copy of the query rows leaves out (128 is no multiple of G)
        for (int c = 0; c < QB * 8; ++c)
            *reinterpret_cast<uint4*>(q_s + (c >> 3) * (PA_ROWS * 128) + tid * 128 + (c & 7) * 16) =
                make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         tc_smem(tmem_slot)),
                     "r"((uint32_t)Shape::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pt_fence_before();
    __syncthreads();
    pt_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_sp = tmem;                      // S / P: two buffers of P_COLS columns
    const uint32_t tmem_o = tmem + 2 * Shape::P_COLS;   // O: HD columns

    if (warp == 5 || warp == 7) {
        // ------------------------------------------- TMA producers: warp 5 the keys, 7 the values
        const int which = warp == 7;
        const uint32_t full0 = which ? v_full : k_full, empty0 = which ? v_empty : k_empty;
        const uint32_t bytes = which ? Shape::V_BYTES : Shape::K_BYTES;
        const uint32_t dst0 = tc_smem(which ? v_s : k_s);
        if (which == 0 && lane == 0 && ntiles > 0) {
            // the query rows: tokens tok0 .. tok0+TPT-1 (past the last row of the batch: zeros)
            mbar_expect_tx(q_ready, (uint32_t)(QB * RPT * 128));
            for (int b = 0; b < QB; ++b)
                pt_tma_load_4d(tc_smem(q_s + b * (PA_ROWS * 128)), &q_map, q_ready, b * 64, 0, kvh, q_start + tok0);
        }
        bool ok = true;
        int asked = 0;                                  // tiles whose copies have been asked for
        if (LATENT) {
            const int row0 = pa_latent_base(a.qo_indptr, a.kv_len, a.first_entry, blockIdx.z, a.window) -
                             pa_latent_first(past, a.window);
            const int blocks = which ? VB : KB;
            for (int j = 0; j < ntiles; ++j) {
                const int s = j & 1;
                asked = j + 1;
                if (lane < blocks) {
                    if (!mbar_wait(empty0 + 8 * s, (((uint32_t)j >> 1) & 1u) ^ 1u)) {
                        atomicExch(error_word, 23);
                        ok = false;
                    } else {
                        // (bytes may land before lane 0 has announced them: the phase has one arrival)
                        if (lane == 0) mbar_expect_tx(full0 + 8 * s, bytes);
                        const uint32_t dst = dst0 + (uint32_t)s * bytes + (uint32_t)lane * PA_BLOCK;
                        const int row = row0 + tile_key(j);
                        if (!which && lane == 2 * NB)   // the rotated features, shared by the heads
                            tma_load_2d(dst, &rot_map, full0 + 8 * s, a.rot_x, row);
                        else                            // [head keys | remainders | head values | remainders]
                            pt_tma_load_4d(dst, &kv_map, full0 + 8 * s, (which * 2 * NB + lane) * 64, kvh, row, 0);
                    }
                }
                if (!__all_sync(0xffffffffu, ok)) break;
            }
        } else {
            // lanes fetch 32 block-table entries at a time; lane NB p + h waits for the stage and copies
            // block h of page p (at most 8 pages x 2 blocks)
            const int* bt = a.block_table + (size_t)e * a.bt_stride;
            const int ps = a.page_size, ps_log = 31 - __clz(ps);
            const int last_page = (hi - 1) >> ps_log;
            const int per_tile = ps < PA_KEYS ? PA_KEYS >> ps_log : 1;
            const int box_rows = ps < PA_KEYS ? ps : PA_KEYS;
            const int p = lane / NB, h = lane % NB;
            const int page_rows = 2 * a.nkv * ps, row0 = (which * a.nkv + kvh) * ps;
            int mine = 0, have_from = -1;               // lanes hold pages have_from .. +31
            for (int j = 0; j < ntiles; ++j) {
                const int s = j & 1;
                asked = j + 1;
                const int key0 = tile_key(j);
                const int base_page = key0 >> ps_log;
                if (have_from < 0 || base_page + per_tile > have_from + 32) {
                    have_from = base_page;
                    // pages past the last and pages given back: some page, its keys are masked and
                    // its values zeroed
                    mine = max(0, bt[min(base_page + lane, last_page)]);
                }
                const int page = __shfl_sync(0xffffffffu, mine, (base_page + p - have_from) & 31);
                if (p < per_tile) {
                    if (!mbar_wait(empty0 + 8 * s, (((uint32_t)j >> 1) & 1u) ^ 1u)) {
                        atomicExch(error_word, 23);
                        ok = false;
                    } else {
                        if (lane == 0) mbar_expect_tx(full0 + 8 * s, bytes);
                        tma_load_2d(dst0 + (uint32_t)s * bytes + (uint32_t)(h * PA_BLOCK + p * box_rows * 128), &kv_map,
                                    full0 + 8 * s, h * 64, page * page_rows + row0 + (key0 & (ps - 1)));
                    }
                }
                if (!__all_sync(0xffffffffu, ok)) break;
            }
        }
        // no copy outlives the CTA, whatever became of its reader
        if (lane == 0) {
            if (which == 0 && ntiles > 0) mbar_wait(q_ready, 0);
            for (int j = max(0, asked - 2); j < asked; ++j) mbar_wait(full0 + 8 * (j & 1), ((uint32_t)j >> 1) & 1u);
        }
    } else if (warp == 4) {
        // ------------------------------------------------ S = Q K^T, a tile ahead of the softmax
        if (lane == 0 && ntiles > 0) {
            constexpr uint32_t idesc_s = pt_idesc(PA_ROWS, PA_KEYS, 0);
            const uint32_t q_addr = tc_smem(q_s);
            bool q_there = mbar_wait(q_ready, 0);
            if (!q_there) atomicExch(error_word, 24);
            int j = 0;
            for (; j < ntiles && q_there; ++j) {
                const int s = j & 1;
                const uint32_t parity = ((uint32_t)j >> 1) & 1u;
                // the buffer is free once O += P V of tile j-2, which read P from it, is done
                if (!mbar_wait(k_full + 8 * s, parity) ||
                    (j >= 2 && !mbar_wait(v_empty + 8 * s, parity ^ 1u))) {
                    atomicExch(error_word, 24);
                    break;
                }
                pt_fence_after();
                const uint32_t k_addr = tc_smem(k_s) + (uint32_t)s * Shape::K_BYTES;
#pragma unroll
                for (int b = 0; b < KB; ++b) {
                    // key block b meets query block b; the remainders (latent form) the same blocks again
                    const int qb = b < NB ? b : b < 2 * NB ? b - NB : NB;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        pt_mma(tmem_sp + (uint32_t)s * Shape::P_COLS,
                               pt_desc(q_addr + (uint32_t)qb * (PA_ROWS * 128) + (uint32_t)kk * 32, 16, 1024),
                               pt_desc(k_addr + (uint32_t)b * PA_BLOCK + (uint32_t)kk * 32, 16, 1024), idesc_s,
                               (b | kk) != 0);
                }
                pt_commit(s_full + 8 * s);
                pt_commit(k_empty + 8 * s);
            }
            // ... nor a product
            if (j > 0) mbar_wait(k_empty + 8 * ((j - 1) & 1), ((uint32_t)(j - 1) >> 1) & 1u);
        }
    } else if (warp == 6) {
        // ------------------------------------------------ O += P V, V the N-major operand
        constexpr uint32_t idesc_o = pt_idesc(PA_ROWS, HD, 1);
        int j = 0;
        for (; j < ntiles; ++j) {
            const int s = j & 1;
            const uint32_t parity = ((uint32_t)j >> 1) & 1u;
            if (!pt_wait_warp(v_full + 8 * s, parity)) {
                if (lane == 0) atomicExch(error_word, 25);
                break;
            }
            const uint32_t v_addr = tc_smem(v_s) + (uint32_t)s * Shape::V_BYTES;
            const int key0 = tile_key(j);
            if (key0 + PA_KEYS > hi || (key0 < lo && key0 + PA_KEYS > a.keep_first)) {
                // values of keys that no row of the CTA sees
                for (int r = lane; r < PA_KEYS; r += 32) {
                    const int key = key0 + r;
                    if (key < hi && (key >= lo || key < a.keep_first)) continue;
                    for (int c = 0; c < VB * 8; ++c)
                        *reinterpret_cast<uint4*>(v_s + s * Shape::V_BYTES + (c >> 3) * PA_BLOCK + r * 128 + (c & 7) * 16) =
                            make_uint4(0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            // the softmax threads have replaced S by P and rescaled O where needed
            if (!pt_wait_warp(p_ready + 8 * s, parity)) {
                if (lane == 0) atomicExch(error_word, 25);
                break;
            }
            if (lane == 0) {
                pt_fence_after();
                const uint32_t p0 = tmem_sp + (uint32_t)s * Shape::P_COLS;
                // 4 k-steps of 16 keys (8 columns of packed P); V rows are keys, 8-key groups 1024 bytes
                // apart, the 64-feature blocks 8192 bytes apart
#pragma unroll
                for (int part = 0; part < (LATENT ? 5 : 3); ++part) {   // P0 V0, P1 V0, P2 V0, P0 V1, P1 V1
                    const uint32_t p = p0 + (uint32_t)(part % 3) * 32;
                    const uint32_t v = v_addr + (part >= 3 ? (uint32_t)NB * PA_BLOCK : 0u);
#pragma unroll
                    for (int kk = 0; kk < PA_KEYS / 16; ++kk) {
                        const uint64_t vd = pt_desc(v + (uint32_t)kk * 16 * 128, PA_BLOCK, 1024);
                        if (Shape::P2_SMEM && part == 2)
                            pt_mma(tmem_o, pt_desc(tc_smem(p2_s) + (uint32_t)kk * 32, 16, 1024), vd, idesc_o, 1);
                        else
                            pt_mma_ts(tmem_o, p + (uint32_t)kk * 8, vd, idesc_o, (j | part | kk) != 0);
                    }
                }
                pt_commit(v_empty + 8 * s);     // the values are consumed, O holds tiles 0..j
            }
            __syncwarp();
        }
        if (lane == 0 && j > 0) mbar_wait(v_empty + 8 * ((j - 1) & 1), ((uint32_t)(j - 1) >> 1) & 1u);
    } else if (warp < 4) {
        // ------------------------------------------------------ softmax, one row per thread
        const int r = tid;                              // row of the tile = TMEM lane
        const int tok = tok0 + min(r, RPT - 1) / G, head = kvh * G + r % G;
        const bool valid = r < RPT && tok < q_len;
        const int cp = past + min(tok, q_len - 1);      // newest key this row sees
        const int row_lo = window_lo(cp);               // ... and the oldest one (kept ones aside)
        const int cp_min = past + tok0, lo_max = window_lo(past + min(q_len, tok0 + TPT) - 1);
        const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
        const float scale = a.scale_log2e;
        const float bias = a.bias != nullptr && r < RPT ? a.bias[head] * 1.4426950408889634f : 0.f;
        // m: the reference maximum, in base-2 units; a low cap serves every row without a search
        float m = SIGMOID ? 0.f : CAP && a.cap_bounds ? a.cap_log2e + bias : PA_NO_MAX, l = 0.f;
        bool ok = true;
        for (int j = 0; j < ntiles; ++j) {
            const uint32_t parity = ((uint32_t)j >> 1) & 1u;
            if (!pt_wait_warp(s_full + 8 * (j & 1), parity)) {
                if (lane == 0) atomicExch(error_word, 26);
                ok = false;
                break;
            }
            pt_fence_after();
            const uint32_t sp = tmem_sp + lane_off + (uint32_t)(j & 1) * Shape::P_COLS;
            uint32_t s[2][32];
            pt_ld32(sp, s[0]);
            pt_ld32(sp + 32, s[1]);
            pt_wait_ld();
            const int key0 = tile_key(j);
            // the keys of the tile that the row sees, a bit each (tiles that every row sees whole: not asked)
            const bool edge = !(key0 + PA_KEYS - 1 <= cp_min && (key0 >= lo_max || key0 + PA_KEYS <= a.keep_first));
            uint32_t seen[2] = {0xffffffffu, 0xffffffffu};
            if (edge) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k0 = key0 + 32 * h;
                    seen[h] = pa_first(cp + 1 - k0) & (~pa_first(row_lo - k0) | pa_first(a.keep_first - k0));
                }
            }
            // scores in base-2 units, capped and biased where the options ask for it:
            // cap tanh(x / cap) = cap (1 - 2 / (2^(2 log2(e) x / cap) + 1)), or, where all of the scores that the
            // row sees in the tile lie within half of the cap, by a polynomial, which leaves the exponential
            // unit to the probabilities (what bounds the kernel otherwise: three operations a score instead of
            // one).  Each row decides for itself by what it sees, so that its bits depend on nothing else.
            if (CAP) {
                float big = 0.f;
                if (edge) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            big = fmaxf(big, seen[h] >> i & 1u ? fabsf(__uint_as_float(s[h][i])) : 0.f);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        big = fmaxf(big, fmaxf(fabsf(__uint_as_float(s[0][i])), fabsf(__uint_as_float(s[1][i]))));
                }
                if (big * a.cap_z <= 0.5f) {
                    const pa_f2 to_z = pa_pack(a.cap_z, a.cap_z), cap2 = pa_pack(a.cap_log2e, a.cap_log2e),
                                bias2 = pa_pack(bias, bias);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const pa_f2 x = pa_pack(__uint_as_float(s[h][i]), __uint_as_float(s[h][i + 1]));
                            const pa_f2 v = pa_fma2(pa_tanh2(pa_mul2(x, to_z)), cap2, bias2);
                            s[h][i] = __float_as_uint(pa_lo(v));
                            s[h][i + 1] = __float_as_uint(pa_hi(v));
                        }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float x = __uint_as_float(s[h][i]);
                            s[h][i] = __float_as_uint(
                                fmaf(pa_rcp(pt_ex2(x * a.cap_in) + 1.f), -2.f * a.cap_log2e, a.cap_log2e) + bias);
                        }
                }
                __syncwarp();
            } else if (SIGMOID) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 32; ++i) s[h][i] = __float_as_uint(fmaf(__uint_as_float(s[h][i]), scale, bias));
            }
            if (edge) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!(seen[h] >> i & 1u)) s[h][i] = 0xff800000u;    // -inf
            }
            const float unit = CAP || SIGMOID ? 1.f : scale;
            float alpha = 1.f;
            if (!SIGMOID && !(CAP && a.cap_bounds)) {
                float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    mx0 = fmaxf(mx0, __uint_as_float(s[0][i]));
                    mx1 = fmaxf(mx1, __uint_as_float(s[1][i]));
                }
                float mx = fmaxf(mx0, mx1) * unit;      // unit > 0
                if (!CAP) mx += bias;
                if (mx > m + PA_MAX_SLACK) {
                    alpha = pt_ex2(m - mx);
                    m = mx;
                }
            }
            const float shift = CAP || SIGMOID ? -m : bias - m;
            pa_f2 sum2 = 0ull;
            const pa_f2 unit2 = pa_pack(unit, unit), shift2 = pa_pack(shift, shift);
            // P over this row's S, 16 keys at a time: columns 0..31 the heads, 32..63 the remainders, 64..95 theirs
            // (or a row of shared memory, below); column c of each holds keys 2 c, 2 c + 1
            uint32_t p2[4][8];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t p0[8], p1[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = 16 * (h & 1) + 2 * i;
                    pa_f2 x = pa_pack(__uint_as_float(s[h >> 1][k]), __uint_as_float(s[h >> 1][k + 1]));
                    if (SIGMOID) {
                        x = pa_pack(pa_rcp(1.f + pt_ex2(-pa_lo(x))), pa_rcp(1.f + pt_ex2(-pa_hi(x))));
                    } else {
                        x = pa_fma2(x, unit2, shift2);
                        x = pa_pack(pt_ex2(pa_lo(x)), pt_ex2(pa_hi(x)));
                        sum2 = pa_add2(sum2, x);
                    }
                    p0[i] = pa_take_part(x);
                    p1[i] = pa_take_part(x);
                    p2[h][i] = pa_take_part(x);
                }
                pt_st8(sp + 8 * h, p0);
                pt_st8(sp + 32 + 8 * h, p1);
                if (!Shape::P2_SMEM) pt_st8(sp + 64 + 8 * h, p2[h]);
            }
            l = l * alpha + (pa_lo(sum2) + pa_hi(sum2));
            const bool rescale = !SIGMOID && j > 0 && __any_sync(0xffffffffu, alpha != 1.f);
            if (rescale || (Shape::P2_SMEM && j > 0)) {
                // O += P V of tile j-1 must be done before O is rescaled, and has read the third part of its P
                if (!pt_wait_warp(v_empty + 8 * ((j - 1) & 1), ((uint32_t)(j - 1) >> 1) & 1u)) {
                    if (lane == 0) atomicExch(error_word, 27);
                    ok = false;
                    break;
                }
                pt_fence_after();
            }
            if (rescale) {
#pragma unroll 1
                for (int c0 = 0; c0 < HD; c0 += 32) {
                    uint32_t o[32];
                    pt_ld32(tmem_o + lane_off + (uint32_t)c0, o);
                    pt_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    pt_st32(tmem_o + lane_off + (uint32_t)c0, o);
                }
            }
            if (Shape::P2_SMEM) {
                // a row of 128 bytes, its 16-byte pieces where the 128-byte swizzle wants them
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(p2_s + r * 128 + ((c ^ (r & 7)) << 4)) =
                        make_uint4(p2[c >> 1][4 * (c & 1)], p2[c >> 1][4 * (c & 1) + 1], p2[c >> 1][4 * (c & 1) + 2],
                                   p2[c >> 1][4 * (c & 1) + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            pt_wait_st();
            pt_fence_before();
            mbar_arrive(p_ready + 8 * (j & 1));
        }
        if (ok && ntiles > 0 &&
            !pt_wait_warp(v_empty + 8 * ((ntiles - 1) & 1), ((uint32_t)(ntiles - 1) >> 1) & 1u)) {
            if (lane == 0) atomicExch(error_word, 27);
            ok = false;
        }
        pt_fence_after();
        // ---------------------------------------------------------------- epilogue
        // (`ok` is the same in all lanes of a warp; rows past the entry's last token are read with the
        // others, the load being a warp's, and not stored)
        if (ok) {
            const size_t row = (size_t)(q_start + tok) * a.nq + head;
            bf16* out = a.out + ((size_t)(q_start + tok) * a.out_heads + head) * HD;
            const float* gate = nullptr;
            float inv = 1.f;
            if (a.splits == 1 && valid) {
                if (!SIGMOID) {
                    if (a.sink != nullptr) l += exp2f(a.sink[head] * 1.4426950408889634f - m);
                    inv = 1.f / l;
                }
                if (a.gate != nullptr) {
                    gate = a.gate + (size_t)(q_start + tok) * a.gate_stride + (a.gate_features ? head * HD : head);
                    if (!a.gate_features) inv *= pa_sigmoid(*gate);
                }
            }
#pragma unroll 1
            for (int c0 = 0; c0 < HD; c0 += 32) {
                uint32_t o[32];
                if (ntiles > 0) {
                    pt_ld32(tmem_o + lane_off + (uint32_t)c0, o);
                    pt_wait_ld();
                }
                if (!valid) continue;
                if (ntiles == 0) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0u;
                }
                if (a.splits > 1) {                     // rows of HD + 2 floats: 8-byte pieces
                    float2* dst = reinterpret_cast<float2*>(a.scratch + (row * a.splits + split) * (HD + 2) + c0);
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        dst[i] = make_float2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float f[8];
                    if (a.gate != nullptr && a.gate_features) {
                        if (a.gate_vec) {
                            load8(gate + c0 + 8 * i, f);
                        } else {
#pragma unroll
                            for (int t = 0; t < 8; ++t) f[t] = gate[c0 + 8 * i + t];
                        }
#pragma unroll
                        for (int t = 0; t < 8; ++t) f[t] = over_one_plus_bf16(inv, expf(-f[t]));
                    } else {
#pragma unroll
                        for (int t = 0; t < 8; ++t) f[t] = inv;
                    }
#pragma unroll
                    for (int t = 0; t < 8; ++t) f[t] *= __uint_as_float(o[8 * i + t]);
                    store8(out + c0 + 8 * i, f);
                }
            }
            if (a.splits > 1 && valid) {
                // (sigmoid weights: the merge's quotient is by the one split that says 1)
                const bool none = !SIGMOID && m == PA_NO_MAX;
                *reinterpret_cast<float2*>(a.scratch + (row * a.splits + split) * (HD + 2) + HD) =
                    make_float2(none ? -INFINITY : m, SIGMOID ? (split == 0 ? 1.f : 0.f) : l);
            }
        }
    }
    pt_fence_before();
    __syncthreads();
    if (warp == 4) {
        pt_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)Shape::TMEM_COLS)
                     : "memory");
    }
}

// A warp a (token, head) row: the partials of the splits (at most 32), weighted by 2^(m_s - max m).
template <int HD>
__global__ void __launch_bounds__(128)
prompt_merge_kernel(PromptArgs a, int row0, int rows) {
    const int row = row0 + (blockIdx.x * 128 + threadIdx.x) / 32, lane = threadIdx.x & 31;
    if (row >= row0 + rows) return;
    const int tok = row / a.nq, head = row - tok * a.nq;
    const float* base = a.scratch + (size_t)row * a.splits * (HD + 2);
    float m = -INFINITY, l = 0.f;
    if (lane < a.splits) {
        m = base[lane * (HD + 2) + HD];
        l = base[lane * (HD + 2) + HD + 1];
    }
    const float M = warp_max(m);
    const float w = m == -INFINITY ? 0.f : exp2f(m - M);
    float L = warp_sum(l * w);
    if (a.sink != nullptr) L += exp2f(a.sink[head] * 1.4426950408889634f - M);
    const float* gate = a.gate == nullptr ? nullptr
                                          : a.gate + (size_t)tok * a.gate_stride + (a.gate_features ? head * HD : head);
    float sum[HD / 32];
#pragma unroll
    for (int i = 0; i < HD / 32; ++i) sum[i] = 0.f;
#pragma unroll 4
    for (int s = 0; s < a.splits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, s);
#pragma unroll
        for (int i = 0; i < HD / 32; ++i) sum[i] = fmaf(base[s * (HD + 2) + i * 32 + lane], ws, sum[i]);
    }
#pragma unroll
    for (int i = 0; i < HD / 32; ++i) {
        const float g = gate == nullptr ? 1.f : pa_sigmoid(gate[a.gate_features ? i * 32 + lane : 0]);
        a.out[((size_t)tok * a.out_heads + head) * HD + i * 32 + lane] = __float2bfloat16_rn(sum[i] / L * g);
    }
}

template <int HD, bool LATENT, bool CAP, bool SIGMOID>
static int launch_prompt(const CUtensorMap& kv_map, const CUtensorMap& rot_map, const CUtensorMap& q_map,
                         PromptArgs a, int row0, int rows, int* error_word, cudaStream_t stream) {
    constexpr int smem = PromptShape<HD, LATENT>::SMEM_LAUNCH;
    auto kernel = prompt_attention_kernel<HD, LATENT, CAP, SIGMOID>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        // several CTAs per SM need nearly all of the SM's shared memory
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long n = (long long)a.row_tiles * a.nkv * a.splits;
    const int sms = device_sm_count();
    a.fold = smem < 114 * 1024 && a.entries == 1 && a.splits == 1 && n > sms && n <= 2 * sms ? sms : 0;
    kernel<<<dim3((unsigned)n, 1, a.entries), PA_THREADS, smem, stream>>>(kv_map, rot_map, q_map, a, error_word);
    if (a.splits > 1) prompt_merge_kernel<HD><<<(rows + 3) / 4, 128, 0, stream>>>(a, row0, rows);
    return launch_status();
}

// rows of [heads][features] queries as [token][kv head][head of the group][feature]; a box is a tile's
// rows of one kv head and 64 features (features past the last: zeros)
static int prompt_q_map(CUtensorMap* map, const void* q, int q_stride, int q_head, int q_rows, int nkv, int G,
                        int features) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (encode == nullptr) return -3;
    const cuuint64_t dims[4] = {(cuuint64_t)features, (cuuint64_t)G, (cuuint64_t)nkv, (cuuint64_t)q_rows};
    const cuuint64_t strides[3] = {(cuuint64_t)q_head * 2, (cuuint64_t)G * q_head * 2, (cuuint64_t)q_stride * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)G, 1, (cuuint32_t)(PA_ROWS / G)};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(q), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -4;
}

// Entries [0, entries) of the batch, the paged form.  `kv_map`: the cache's tensor map (key and value
// size hd = 64 or 128, page size 8..64 dividing 64, or 128 or 256); q: `tokens` dense rows of nq * hd;
// out: [tokens, nq * hd]; scratch: float [tokens * nq * splits * (hd + 2)] when splits > 1 (at most
// 32).  Returns 0, a CUDA error code, -1 when the shape is refused, -3 / -4 when a tensor map cannot
// be made.  `error_word` receives 22..27 if a wait ran out (22: shared memory off its alignment).
MSTAR_API int mstar_sink_attention_prompt(const void* kv_map, const void* q, int q_stride, void* out,
                                          const int* block_table, int bt_stride, const int* qo_indptr,
                                          const int* kv_len, int entries, int tokens, int max_q_len, int nq,
                                          int nkv, int hd, int page_size, int window, int keep_first, float scale,
                                          int splits, float* scratch, const float* gate, int gate_stride,
                                          int gate_features, float softcap, const float* sink, int chunk,
                                          int sigmoid, const float* bias, int* error_word, void* stream) {
    if (entries <= 0 || max_q_len <= 0) return 0;
    if (chunk < 0 || (chunk > 0 && window > 0) || (sigmoid && sink != nullptr)) return -1;
    if ((hd != 64 && hd != 128) || !(scale > 0.f) || nkv <= 0 || nq % nkv != 0 || kv_map == nullptr ||
        entries > 65535 || splits < 1 || splits > 32 || (splits > 1 && scratch == nullptr))
        return -1;
    if (!((page_size >= 8 && page_size <= 64 && PA_KEYS % page_size == 0) || page_size == 128 || page_size == 256))
        return -1;
    const int G = nq / nkv;
    if (G > PA_ROWS || (((uintptr_t)q | (uintptr_t)out) & 15) != 0 || q_stride % 8 != 0) return -1;
    CUtensorMap map, q_map;
    memcpy(&map, kv_map, sizeof(map));
    const int rc = prompt_q_map(&q_map, q, q_stride, hd, tokens, nkv, G, hd);
    if (rc != 0) return rc;
    PromptArgs a = {};
    a.block_table = block_table;
    a.qo_indptr = qo_indptr;
    a.kv_len = kv_len;
    a.out = (bf16*)out;
    a.scratch = scratch;
    a.gate = gate;
    a.sink = sink;
    a.bias = bias;
    a.bt_stride = bt_stride;
    a.nq = nq;
    a.nkv = nkv;
    a.out_heads = nq;
    a.page_size = page_size;
    a.entries = entries;
    a.window = window;
    a.keep_first = window > 0 ? keep_first : 0;
    a.chunk = chunk;
    a.splits = splits;
    a.row_tiles = (max_q_len + PA_ROWS / G - 1) / (PA_ROWS / G);
    a.gate_stride = gate_stride;
    a.gate_features = gate != nullptr && gate_features;
    a.gate_vec = gate_stride % 4 == 0 && ((uintptr_t)gate & 15) == 0;
    a.scale_log2e = scale * 1.4426950408889634f;
    a.cap_in = softcap > 0.f ? 2.f * 1.4426950408889634f * scale / softcap : 0.f;
    a.cap_log2e = softcap * 1.4426950408889634f;
    a.cap_z = softcap > 0.f ? scale / softcap : 0.f;
    // probabilities then lie within 2^(-2 cap) of 1: far from what a float, and the remainders 2^-9 and 2^-18 below
    // it, hold
    a.cap_bounds = softcap > 0.f && a.cap_log2e <= 48.f;
    if ((long long)a.row_tiles * nkv * splits > 2147483647LL) return -1;
    cudaStream_t s = (cudaStream_t)stream;
#define GO(HD, CAP, SIG) launch_prompt<HD, false, CAP, SIG>(map, map, q_map, a, 0, tokens * nq, error_word, s)
#define GO_HD(HD)                                                                                 \
    (softcap > 0.f ? (sigmoid ? GO(HD, true, true) : GO(HD, true, false))                         \
                   : (sigmoid ? GO(HD, false, true) : GO(HD, false, false)))
    return hd == 64 ? GO_HD(64) : GO_HD(128);
#undef GO_HD
#undef GO
}

// ------------------------------------------------------------------ the latent form's keys and values
// rows[pa_latent_base(e) + key - first] = the cache row of `key`, for the keys that entry e's tokens see
// (first: pa_latent_first); `chunks` pieces of 16 bytes a row.  Grid: x pieces of the keys, y the entry.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const uint4* __restrict__ cache, const int* __restrict__ block_table, int bt_stride,
                     const int* __restrict__ qo_indptr, const int* __restrict__ kv_len, uint4* __restrict__ rows,
                     int first_entry, int window, int page_size, int chunks) {
    const int e = first_entry + blockIdx.y;
    const int n = kv_len[e], first = pa_latent_first(n - (qo_indptr[e + 1] - qo_indptr[e]), window);
    const size_t base = pa_latent_base(qo_indptr, kv_len, first_entry, blockIdx.y, window);
    const int* bt = block_table + (size_t)e * bt_stride;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    for (int key = first + blockIdx.x * 8 + (threadIdx.x >> 5); key < n; key += gridDim.x * 8) {
        // (a page before the window may have been given back)
        const int page = bt[key / page_size];
        const uint4* src = cache + ((size_t)max(page, 0) * page_size + key % page_size) * chunks;
        uint4* dst = rows + (base + key - first) * chunks;
        for (int c = threadIdx.x & 31; c < chunks; c += 32) dst[c] = page < 0 ? none : src[c];
    }
}

// parts[row][head][k head | k remainder | v head | v remainder] from the float products
// keys[row][head][dim] and values, rows `ld` floats apart; eight features a thread.
__global__ void __launch_bounds__(256)
latent_split_kernel(const float* __restrict__ keys, const float* __restrict__ values, bf16* __restrict__ parts,
                    int ld, long long pieces, int heads, int dim) {
    const int per_head = dim / 8, per_row = 2 * heads * per_head;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < pieces; i += (long long)gridDim.x * 256) {
        const long long row = i / per_row;
        const int at = (int)(i - row * per_row), which = at / (heads * per_head);
        const int head = at / per_head - which * heads, d = at % per_head * 8;
        float v[8], rest[8];
        load8((which ? values : keys) + row * ld + head * dim + d, v);
#pragma unroll
        for (int k = 0; k < 8; ++k) rest[k] = v[k] - __bfloat162float(__float2bfloat16_rn(v[k]));
        bf16* dst = parts + ((row * heads + head) * 4 + 2 * which) * dim + d;
        store8(dst, v);
        store8(dst + dim, rest);
    }
}

// The rows of the cache that entries [first_entry, first_entry + entries) see, one after another (how
// many there are the caller knows from the lengths; `most` bounds those of one entry).
MSTAR_API int mstar_latent_gather(const void* cache, const int* block_table, int bt_stride, const int* qo_indptr,
                                  const int* kv_len, void* rows, int first_entry, int entries, int most, int window,
                                  int page_size, int features, void* stream) {
    if (entries <= 0 || most <= 0) return 0;
    if (features % 8 != 0 || entries > 65535 || (((uintptr_t)cache | (uintptr_t)rows) & 15) != 0) return -1;
    latent_gather_kernel<<<dim3((most + 7) / 8, entries), 256, 0, (cudaStream_t)stream>>>(
        (const uint4*)cache, block_table, bt_stride, qo_indptr, kv_len, (uint4*)rows, first_entry, window, page_size,
        features / 8);
    return launch_status();
}

MSTAR_API int mstar_latent_split(const float* keys, const float* values, int ld, void* parts, int rows, int heads,
                                 int dim, void* stream) {
    if (rows <= 0) return 0;
    if (dim % 8 != 0 || ld % 4 != 0 || (((uintptr_t)keys | (uintptr_t)values | (uintptr_t)parts) & 15) != 0) return -1;
    const long long pieces = (long long)rows * 2 * heads * (dim / 8);
    const long long blocks = (pieces + 255) / 256, most = (long long)device_sm_count() * 16;
    latent_split_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, (cudaStream_t)stream>>>(
        keys, values, (bf16*)parts, ld, pieces, heads, dim);
    return launch_status();
}

// Entries [first_entry, first_entry + entries), the latent form.  q: `tokens` rows (the whole step's), head
// h's dim plain and rot rotated features at h * q_head; parts: [key_rows][heads][4 * dim] and latents:
// [key_rows][rank + rot], made by the two functions above; out: [tokens, out_heads * dim], of which the
// entries' rows (rows_from .. + rows) and the first `heads` heads are written; gate: null or one number a head.
MSTAR_API int mstar_latent_attention_prompt(const void* q, int q_stride, int q_head, int tokens, const void* parts,
                                            const void* latents, int key_rows, void* out, const int* qo_indptr,
                                            const int* kv_len, int first_entry, int entries, int max_q_len,
                                            int rows_from, int rows, int heads, int out_heads, int dim, int rank, int rot, int window,
                                            float scale, int splits, float* scratch, const float* gate,
                                            int gate_stride, int* error_word, void* stream) {
    if (entries <= 0 || max_q_len <= 0) return 0;
    if ((dim != 64 && dim != 128) || rot <= 0 || rot > 64 || rot % 8 != 0 || rank % 8 != 0 || !(scale > 0.f) ||
        heads <= 0 || entries > 65535 || key_rows <= 0 || splits < 1 || splits > 32 || (splits > 1 && scratch == nullptr))
        return -1;
    if ((((uintptr_t)q | (uintptr_t)out | (uintptr_t)parts | (uintptr_t)latents) & 15) != 0 || q_stride % 8 != 0 ||
        q_head % 8 != 0)
        return -1;
    CUtensorMap kv_map, rot_map, q_map;
    int rc = prompt_q_map(&q_map, q, q_stride, q_head, tokens, heads, 1, dim + rot);
    if (rc != 0) return rc;
    EncodeTiledFn encode = encode_tiled_fn();
    {
        const cuuint64_t dims[4] = {(cuuint64_t)4 * dim, (cuuint64_t)heads, (cuuint64_t)key_rows, 1};
        const cuuint64_t strides[3] = {(cuuint64_t)dim * 8, (cuuint64_t)heads * dim * 8,
                                       (cuuint64_t)key_rows * heads * dim * 8};
        const cuuint32_t box[4] = {64, 1, PA_KEYS, 1};
        const cuuint32_t elem[4] = {1, 1, 1, 1};
        if (encode(&kv_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(parts), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -4;
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)(rank + rot), (cuuint64_t)key_rows};
        const cuuint64_t strides[1] = {(cuuint64_t)(rank + rot) * 2};
        const cuuint32_t box[2] = {64, PA_KEYS};
        const cuuint32_t elem[2] = {1, 1};
        if (encode(&rot_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(latents), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -4;
    }
    PromptArgs a = {};
    a.qo_indptr = qo_indptr;
    a.kv_len = kv_len;
    a.out = (bf16*)out;
    a.scratch = scratch;
    a.gate = gate;
    a.nq = a.nkv = heads;
    a.out_heads = out_heads;
    a.first_entry = first_entry;
    a.entries = entries;
    a.window = window;
    a.splits = splits;
    a.row_tiles = (max_q_len + PA_ROWS - 1) / PA_ROWS;
    a.gate_stride = gate_stride;
    a.scale_log2e = scale * 1.4426950408889634f;
    a.rot_x = rank;
    cudaStream_t s = (cudaStream_t)stream;
    return dim == 64 ? launch_prompt<64, true, false, false>(kv_map, rot_map, q_map, a, rows_from * heads, rows * heads, error_word, s)
                     : launch_prompt<128, true, false, false>(kv_map, rot_map, q_map, a, rows_from * heads, rows * heads, error_word, s);
}
