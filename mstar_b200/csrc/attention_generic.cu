// Paged grouped-query attention for any mix of prompt portions and decoded tokens,
// in float arithmetic: on CUDA cores, and for prompt portions of floats by bfloat16 parts on the tensor cores (below).  It is
// the attention of the true 32-bit path and the fallback of the bfloat16 path for shapes the tensor-core kernels refuse.
//
// Semantics (mstar/engine/cache_manager.py:653-701 for the call, scale 1/sqrt(hd)
// as in mstar/utils/attention.py:116-117): query head i uses key/value head
// i / (nq/nkv); the token whose key sits at cache position p sees keys lo..p with
// lo = max(0, p - window + 1) (window 0: lo = 0), which is the causal mask aligned
// to the end of the sequence; softmax statistics and the output sum are float.
//
// One block per (token, kv head) handles the whole group of query heads, streaming
// the keys and values of that head through shared memory in tiles of 32 keys with
// an online softmax.  The keys of the current step are already in the cache.
//
// Floats with a head_dim of 64 or 128 take the kernels below: prompt portions one whose blocks share a tile of
// keys among 64 rows, single tokens one whose warps read their keys straight from the cache.
#include "common.cuh"
#include "mma_util.cuh"

#define ATT_TILE 32
#define ATT_THREADS 128
#define ATT_MAX_ACC 32

struct AttnArgs {
    int nq, nkv, hd, page_size, bt_stride, window;
    int q_stride;  // elements between consecutive tokens in q
    float scale;
};

template <typename A>
__global__ void __launch_bounds__(ATT_THREADS)
paged_attention_generic_kernel(const A* __restrict__ q, A* __restrict__ out,
                               const A* __restrict__ kv_cache, const int* __restrict__ block_table,
                               const int* __restrict__ token_req, const int* __restrict__ cache_pos,
                               AttnArgs a) {
    extern __shared__ float smem[];
    const int t = blockIdx.x, kvh = blockIdx.y;
    const int hd = a.hd, G = a.nq / a.nkv;
    const int ldk = hd + 1;
    float* qs = smem;                        // [G][hd]
    float* tile = qs + G * hd;               // [ATT_TILE][hd+1]
    float* sc = tile + ATT_TILE * ldk;       // [G][ATT_TILE]
    float* m_s = sc + G * ATT_TILE;          // [G]
    float* l_s = m_s + G;                    // [G]
    float* alpha_s = l_s + G;                // [G]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hi = cache_pos[t] + 1;
    const int lo = (a.window > 0 && hi > a.window) ? hi - a.window : 0;
    const int* bt = block_table + (size_t)token_req[t] * a.bt_stride;
    const size_t page_elems = (size_t)2 * a.nkv * a.page_size * hd;
    const size_t head_off = (size_t)kvh * a.page_size * hd;
    const size_t v_off = (size_t)a.nkv * a.page_size * hd;

    const A* qrow = q + (size_t)t * a.q_stride + (size_t)kvh * G * hd;
    for (int i = tid; i < G * hd; i += ATT_THREADS) qs[i] = to_float(qrow[i]);
    for (int i = tid; i < G; i += ATT_THREADS) {
        m_s[i] = -INFINITY;
        l_s[i] = 0.f;
    }
    float acc[ATT_MAX_ACC];
#pragma unroll
    for (int k = 0; k < ATT_MAX_ACC; ++k) acc[k] = 0.f;
    const int n_out = G * hd;
    __syncthreads();

    for (int base = lo; base < hi; base += ATT_TILE) {
        // ---- keys of this tile -> shared (zero rows beyond hi)
        for (int idx = tid; idx < ATT_TILE * hd; idx += ATT_THREADS) {
            const int j = idx / hd, d = idx - j * hd;
            const int key = base + j;
            float v = 0.f;
            if (key < hi) {
                const int page = bt[key / a.page_size];
                const int slot = key % a.page_size;
                v = to_float(kv_cache[(size_t)page * page_elems + head_off + (size_t)slot * hd + d]);
            }
            tile[j * ldk + d] = v;
        }
        __syncthreads();
        // ---- scores
        for (int idx = tid; idx < G * ATT_TILE; idx += ATT_THREADS) {
            const int g = idx / ATT_TILE, j = idx - g * ATT_TILE;
            float s = -INFINITY;
            if (base + j < hi) {
                const float* qv = qs + g * hd;
                const float* kv = tile + j * ldk;
                float dot = 0.f;
                for (int d = 0; d < hd; ++d) dot = fmaf(qv[d], kv[d], dot);
                s = dot * a.scale;
            }
            sc[idx] = s;
        }
        __syncthreads();
        // ---- online softmax statistics, one warp per query head
        for (int g = warp; g < G; g += ATT_THREADS / 32) {
            const float s = sc[g * ATT_TILE + lane];
            const float m_old = m_s[g];
            const float m_new = fmaxf(m_old, warp_max(s));  // key `base` is always valid
            const float p = expf(s - m_new);                 // exp(-inf) = 0 for masked keys
            const float psum = warp_sum(p);
            sc[g * ATT_TILE + lane] = p;
            if (lane == 0) {
                const float al = expf(m_old - m_new);        // 0 on the first tile
                alpha_s[g] = al;
                l_s[g] = l_s[g] * al + psum;
                m_s[g] = m_new;
            }
        }
        __syncthreads();
        // ---- values of this tile -> shared (reusing the key buffer)
        for (int idx = tid; idx < ATT_TILE * hd; idx += ATT_THREADS) {
            const int j = idx / hd, d = idx - j * hd;
            const int key = base + j;
            float v = 0.f;
            if (key < hi) {
                const int page = bt[key / a.page_size];
                const int slot = key % a.page_size;
                v = to_float(kv_cache[(size_t)page * page_elems + v_off + head_off + (size_t)slot * hd + d]);
            }
            tile[j * ldk + d] = v;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ATT_MAX_ACC; ++k) {
            const int o = tid + k * ATT_THREADS;
            if (o < n_out) {
                const int g = o / hd, d = o - g * hd;
                const float* p = sc + g * ATT_TILE;
                float sum = acc[k] * alpha_s[g];
#pragma unroll 8
                for (int j = 0; j < ATT_TILE; ++j) sum = fmaf(p[j], tile[j * ldk + d], sum);
                acc[k] = sum;
            }
        }
        __syncthreads();
    }

    A* orow = out + (size_t)t * a.nq * hd + (size_t)kvh * G * hd;
#pragma unroll
    for (int k = 0; k < ATT_MAX_ACC; ++k) {
        const int o = tid + k * ATT_THREADS;
        if (o < n_out) {
            const int g = o / hd;
            orow[o] = from_float<A>(acc[k] / l_s[g]);
        }
    }
}

// ------------------------------------------------------------------ float prompt portions
// The same attention for float tokens that come in runs of one request: a block takes 64 rows
// (token, head of the group) of one kv head and walks their keys in tiles of 64, so that a key
// is fetched once for all of them.  Thread (ty, tx) of 16 x 16 owns rows ty + 16 i from the
// scores to the output: 4 x 4 scores of a tile (packed FMAs over pairs of features), a row's
// maximum and sum by shuffles among its 16 threads, then 4 rows x HD / 16 output columns
// (packed FMAs over pairs of columns).  Only the probabilities pass through shared memory; the
// next tile's keys are fetched under the softmax and the sum, its values under the scores.
// Two groups of 256 threads take the even and the odd tiles, each with stages of its own, and are added up at
// the end: a block alone on its SM, as most are in a batch of short prompts, is a chain of loads, scores, softmax
// and sums a tile.  Of a tile, scores are made for the sixteens of keys that a row of the block sees, and only
// the few keys that some rows see and others don't are taken one by one (the last tile of every row is such a one).
// Tiles start at multiples of 64 keys whatever the block's rows are, and a tile that a row does
// not see leaves its sums as they are, so a row's result does not depend on what else is in the
// batch.  Bound by the shared loads that feed the FMA pipe (of 16 bytes, no bank met twice).  It makes the rows (`bad`) that
// the tensor cores (below, both sides measured) cannot, for operands that are not finite.
#define AR_ROWS 64
#define AR_KEYS 64
#define AR_THREADS 256                         // of a group
#define AR_GROUPS 2

__device__ __forceinline__ void ar_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long ar_pack(float lo, float hi) {
    return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float ar_lo(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float ar_hi(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

// O += P V of four keys of a tile.  MASKED: a key that a row does not see is left out (a probability of zero
// would still make a NaN of a value that is not finite).
template <int HD, bool MASKED>
__device__ __forceinline__ void ar_output(unsigned long long (&acc)[4][HD / 32], const float* p_s,
                                          const float* v_s, int ty, int tx, int j, int key0, const int (&lo_r)[4],
                                          const int (&hi_r)[4]) {
    constexpr int PL = AR_KEYS + 4;
    float4 p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(p_s + (ty + 16 * i) * PL + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
        unsigned long long v[HD / 32];
#pragma unroll
        for (int c = 0; c < HD / 32; ++c)
            v[c] = *reinterpret_cast<const unsigned long long*>(v_s + (j + jj) * HD + 2 * tx + 32 * c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (MASKED && !(key0 + j + jj >= lo_r[i] && key0 + j + jj < hi_r[i])) continue;
            const float pj = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
            const unsigned long long pp = ar_pack(pj, pj);
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) ar_fma2(acc[i][c], pp, v[c]);
        }
    }
}

template <int HD>
__device__ __noinline__ void ar_block_fma(const float* __restrict__ q, float* __restrict__ out,
                                          const float* __restrict__ kv_cache, const int* __restrict__ block_table,
                                          const int* __restrict__ token_req, const int* __restrict__ cache_pos,
                                          const AttnArgs& a, int num_tokens, unsigned long long bad) {
    constexpr int QL = HD + 4, PL = AR_KEYS + 4;   // floats between rows: 16-byte reads of 8 rows
    extern __shared__ __align__(16) float ar_smem[];
    float* q_s = ar_smem;                          // [ROWS][QL]
    constexpr int BUFS = AR_KEYS * QL + AR_KEYS * HD + AR_ROWS * PL;   // floats of a group
    const int group = threadIdx.x / AR_THREADS;
    float* k_s = q_s + AR_ROWS * QL + group * BUFS;    // [KEYS][QL]
    float* v_s = k_s + AR_KEYS * QL;               // [KEYS][HD]
    float* p_s = v_s + AR_KEYS * HD;               // [ROWS][PL]
    const int tid = threadIdx.x % AR_THREADS, tx = tid & 15, ty = tid >> 4;
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(AR_THREADS) : "memory"); };
    const int kvh = blockIdx.x;
    const int G = a.nq / a.nkv, TPB = AR_ROWS / G;
    // (the tokens with the most keys first)
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * TPB;
    const int ntok = min(TPB, num_tokens - t0), nrows = ntok * G;
    const size_t page_elems = (size_t)2 * a.nkv * a.page_size * HD;
    const size_t v_off = (size_t)a.nkv * a.page_size * HD;
    const float* head_base = kv_cache + (size_t)kvh * a.page_size * HD;

    for (int c = threadIdx.x; c < AR_ROWS * (HD / 4); c += AR_GROUPS * AR_THREADS) {
        const int r = c / (HD / 4), d = (c % (HD / 4)) * 4;
        const bool ok = r < nrows;
        const float* src = q;
        if (ok) src += (size_t)(t0 + r / G) * a.q_stride + (size_t)(kvh * G + r % G) * HD + d;
        cp_async_16(smem_u32(q_s + r * QL + d), src, ok ? 16 : 0);
    }
    cp_async_commit();

    for (int s0 = 0; s0 < ntok;) {
        // tokens s0 .. s1-1 of the block belong to one request
        const int req = token_req[t0 + s0];
        if ((bad >> (s0 * G) & ((2ull << (G - 1)) - 1)) == 0) {        // nothing to make for this token
            ++s0;
            continue;
        }
        int s1 = s0, lo_min = 0x7fffffff, hi_max = 0;      // the keys that any of them sees
        int full_lo = 0, full_hi = 0x7fffffff;             // ... and those that all of them see
        for (; s1 < ntok && token_req[t0 + s1] == req; ++s1) {
            const int hi = cache_pos[t0 + s1] + 1;
            const int lo = (a.window > 0 && hi > a.window) ? hi - a.window : 0;
            lo_min = min(lo_min, lo);
            hi_max = max(hi_max, hi);
            full_lo = max(full_lo, lo);
            full_hi = min(full_hi, hi);
        }
        const int* bt = block_table + (size_t)req * a.bt_stride;
        int lo_r[4], hi_r[4];                      // the keys that this thread's rows see
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + 16 * i, tk = r / G;
            lo_r[i] = hi_r[i] = 0;                 // a row of another request: idle
            if (r < nrows && tk >= s0 && tk < s1) {
                hi_r[i] = cache_pos[t0 + tk] + 1;
                lo_r[i] = (a.window > 0 && hi_r[i] > a.window) ? hi_r[i] - a.window : 0;
            }
        }
        auto load = [&](bool values, int key0) {
#pragma unroll
            for (int c = tid; c < AR_KEYS * (HD / 4); c += AR_THREADS) {
                const int j = c / (HD / 4), d = (c % (HD / 4)) * 4, key = key0 + j;
                const bool ok = key >= lo_min && key < hi_max;
                const float* src = kv_cache;
                if (ok)
                    src = head_base + (size_t)bt[key / a.page_size] * page_elems + (values ? v_off : 0) +
                          (size_t)(key % a.page_size) * HD + d;
                cp_async_16(smem_u32(values ? v_s + j * HD + d : k_s + j * QL + d), src, ok ? 16 : 0);
            }
            cp_async_commit();
        };
        float m[4], l[4];
        unsigned long long acc[4][HD / 32];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            m[i] = -INFINITY;
            l[i] = 0.f;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) acc[i][c] = 0ull;
        }
        const int tile0 = lo_min / AR_KEYS;
        const int first = (tile0 + ((tile0 ^ group) & 1)) * AR_KEYS;       // even tiles: group 0
        if (first < hi_max) load(false, first);
        else cp_async_commit();
        if (first < hi_max) load(true, first);
        else cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();                           // the queries are there
        for (int key0 = first; key0 < hi_max; key0 += AR_GROUPS * AR_KEYS) {
            cp_async_wait<1>();                    // the keys are there
            group_sync();
            unsigned long long s2[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
            const int sixteens = (min(AR_KEYS, hi_max - key0) + 15) / 16;      // of keys that anyone sees
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                ulonglong2 qv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(q_s + (ty + 16 * i) * QL + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j >= sixteens) break;
                    const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(k_s + (tx + 16 * j) * QL + d);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        ar_fma2(s2[i][j], qv[i].x, kv.x);
                        ar_fma2(s2[i][j], qv[i].y, kv.y);
                    }
                }
            }
            group_sync();                          // the keys are done with
            if (key0 + AR_GROUPS * AR_KEYS < hi_max) load(false, key0 + AR_GROUPS * AR_KEYS);
            else cp_async_commit();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float s[4], mx = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = key0 + tx + 16 * j;
                    s[j] = key >= lo_r[i] && key < hi_r[i] ? (ar_lo(s2[i][j]) + ar_hi(s2[i][j])) * a.scale
                                                           : -INFINITY;
                    mx = fmaxf(mx, s[j]);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m[i], mx);
                const bool none = m_new == -INFINITY;          // the row has seen no key yet
                const float alpha = none ? 1.f : expf(m[i] - m_new);
                m[i] = m_new;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float p = none ? 0.f : expf(s[j] - m_new);
                    sum += p;
                    p_s[(ty + 16 * i) * PL + tx + 16 * j] = p;
                }
                l[i] = l[i] * alpha + sum;
                const unsigned long long aa = ar_pack(alpha, alpha);
#pragma unroll
                for (int c = 0; c < HD / 32; ++c)
                    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][c]) : "l"(aa));
            }
            cp_async_wait<1>();                    // the values are there
            group_sync();
            // four keys at a time, of which all are seen by all rows but at the ends
            const int j1 = min(AR_KEYS, hi_max - key0), j0 = max(0, lo_min - key0) & ~3;
            const int m0 = min(j1, max(j0, (max(0, full_lo - key0) + 3) & ~3));
            const int m1 = max(m0, min(j1, full_hi - key0) & ~3);
            for (int j = j0; j < m0; j += 4) ar_output<HD, true>(acc, p_s, v_s, ty, tx, j, key0, lo_r, hi_r);
#pragma unroll 2
            for (int j = m0; j < m1; j += 4) ar_output<HD, false>(acc, p_s, v_s, ty, tx, j, key0, lo_r, hi_r);
            for (int j = m1; j < j1; j += 4) ar_output<HD, true>(acc, p_s, v_s, ty, tx, j, key0, lo_r, hi_r);
            group_sync();                          // the values and the probabilities are done with
            if (key0 + AR_GROUPS * AR_KEYS < hi_max) load(true, key0 + AR_GROUPS * AR_KEYS);
            else cp_async_commit();
        }
        // the odd tiles' sums pass through the place of their values, the rows' statistics through that of
        // their probabilities; the even ones' group adds them up
        float* other_v = q_s + AR_ROWS * QL + BUFS + AR_KEYS * QL;
        float2* other_ml = reinterpret_cast<float2*>(other_v + AR_KEYS * HD);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
            if (group == 0) continue;
            const int r = ty + 16 * i;
            if (tx == 0) other_ml[r] = make_float2(m[i], l[i]);
#pragma unroll
            for (int c = 0; c < HD / 32; ++c)
                *reinterpret_cast<unsigned long long*>(other_v + r * HD + 2 * tx + 32 * c) = acc[i][c];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + 16 * i;
            if (group != 0 || hi_r[i] == 0 || !(bad >> r & 1)) continue;
            const float2 ml = other_ml[r];
            const float top = fmaxf(m[i], ml.x);
            const float w0 = expf(m[i] - top), w1 = expf(ml.x - top);      // (a group that saw no key: 0)
            const float sum = fmaf(l[i], w0, ml.y * w1);
            float* dst = out + (size_t)(t0 + r / G) * a.nq * HD + (size_t)(kvh * G + r % G) * HD + 2 * tx;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) {
                const float2 v = *reinterpret_cast<const float2*>(other_v + r * HD + 2 * tx + 32 * c);
                *reinterpret_cast<float2*>(dst + 32 * c) =
                    make_float2(fmaf(ar_lo(acc[i][c]), w0, v.x * w1) / sum, fmaf(ar_hi(acc[i][c]), w0, v.y * w1) / sum);
            }
        }
        __syncthreads();                           // the sums have been read
        s0 = s1;
    }
}

// ------------------------------------------------------------------ the same on the tensor cores
// A float is the sum of three bfloat16 numbers, its 24 bits eight at a time; of the nine products of such parts the
// six of 2^-16 or more of the whole are made by mma.sync m16n8k16, the leading one into a sum of its own, since
// the tensor core cuts its sums off instead of rounding them; a tile's P V is summed by itself and then added.
// A block takes the same 64 rows.  Its two groups of eight warps take the even and the odd tiles, in a group a
// warp takes 16 rows and one half of a tile's keys, and keeps maxima, sums and output of its own; the four
// shares of a row are added up at the end in their order.  A tile's keys and values are fetched into registers under
// the products of the tile before it, cut into their parts and put into shared memory by the whole group;
// probabilities go from the scores' registers into the products' without passing through memory.
// Operands that are not finite leave no sum behind in their parts (infinity less infinity): zeros stand in for those of a
// key or value, and the rows that see one, or whose result is not finite (an own query, products of finite numbers
// past the largest float), are made again with plain FMAs, no others, so that a row's result does not depend on
// what else is in the batch.
// Bound by latencies where prompts are short (of a block's 10 us with one tile the queries take 1.2, the first
// keys 2, the tile 3, the shares 2) and by the warp-level tensor path and the splitting where they are long.  448
// prompt tokens with 32 / 8 heads of 64 (requests of 256 and 192): 26.5 us, with FMAs 33, and 41 in one group with
// whole tiles; 1,500 tokens: 211, 283, 283; one of 250 tokens on 250 cached keys, 24 / 8 heads of 128: 72, 89, 121;
// 2,000 tokens: 695, 876, 1,258.  512 threads leave 128 registers each: 160 (HD 64) and 300 (128) bytes of them are spilled.
// Error against 64 bits, FMAs in brackets: 256 tokens of normal numbers 1.2e-7 (1.9e-7) with heads of 64 and 1.8e-7 (2.2e-7)
// of 128, 2,000 tokens 1.5e-7 (3.6e-7) and 2.2e-7 (3.9e-7), values of one sign 7.4e-8 (4.7e-7); tokens that see two keys
// of even weight 2.8e-8 (2.7e-8).
template <int HD> __host__ __device__ constexpr int ap_keys() { return HD == 64 ? 64 : 32; }     // of a tile
template <int HD> __host__ __device__ constexpr int ap_smem() {
    return 3 * 2 * (HD + 8) * (AR_ROWS + AR_GROUPS * 2 * ap_keys<HD>());
}

// Two floats as three pairs of bfloat16 numbers; false if one of them is not finite (or too large for its part).
__device__ __forceinline__ bool ap_split(float x, float y, uint32_t (&p)[3]) {
    p[0] = pack_bf16(x, y);
    const float rx = x - __uint_as_float(p[0] << 16), ry = y - __uint_as_float(p[0] & 0xffff0000u);
    p[1] = pack_bf16(rx, ry);
    const float sx = rx - __uint_as_float(p[1] << 16), sy = ry - __uint_as_float(p[1] & 0xffff0000u);
    p[2] = pack_bf16(sx, sy);
    return isfinite(sx + sy);
}

// Zeros for the parts of four floats if one of them is not finite, and a bit set.  (Out of line: this is rare.)
__device__ __noinline__ void ap_zero(bf16* to, int plane, const float* v, unsigned long long* bad, int bit) {
    uint32_t p[3];
    if (ap_split(v[0], v[1], p) && ap_split(v[2], v[3], p)) return;
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(to + i * plane) = make_uint2(0u, 0u);
    atomicOr(bad, 1ull << bit);
}
// The row, if it sees one of these keys.
__device__ __noinline__ void ap_mark(unsigned long long keys, int key0, int lo, int hi, int row, unsigned long long* bad) {
    for (int key = max(lo - key0, 0); key < min(hi - key0, 64); ++key)
        if (keys >> key & 1) atomicOr(bad, 1ull << row);
}

template <int HD>
__global__ void __launch_bounds__(AR_GROUPS * AR_THREADS)
attention_rows_f32_kernel(const float* __restrict__ q, float* __restrict__ out,
                          const float* __restrict__ kv_cache, const int* __restrict__ block_table,
                          const int* __restrict__ token_req, const int* __restrict__ cache_pos,
                          AttnArgs a, int num_tokens) {
    constexpr int KEYS = ap_keys<HD>(), HALF = KEYS / 2, LD = HD + 8;
    constexpr int NT = HALF / 8, KT = HALF / 16, VT = HD / 8;          // a warp's tiles of scores, of keys, of columns
    constexpr int QPLANE = AR_ROWS * LD, KPLANE = KEYS * LD;             // bfloat16 numbers of a part
    constexpr int U = KEYS * (HD / 4) / AR_THREADS;                      // fours of floats a thread fetches
    extern __shared__ __align__(16) float ar_smem[];
    bf16* q_p = reinterpret_cast<bf16*>(ar_smem);                        // [3][ROWS][LD]
    const int group = threadIdx.x / AR_THREADS, tid = threadIdx.x % AR_THREADS;
    bf16* k_p = q_p + 3 * QPLANE + group * 6 * KPLANE;                   // [3][KEYS][LD]
    bf16* v_p = k_p + 3 * KPLANE;
    const int lane = tid & 31, warp = tid >> 5, rt = warp & 3, half = warp >> 2;
    const int g = lane >> 2, c4 = lane & 3;
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(AR_THREADS) : "memory"); };
    // a group's sync that tells it whether this holds for any thread
    auto any_of_group = [&](bool here) {
        uint32_t any;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                     "barrier.cta.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                     : "=r"(any) : "r"((uint32_t)here), "r"(1 + group), "n"(AR_THREADS) : "memory");
        return any != 0;
    };
    const int kvh = blockIdx.x;
    const int G = a.nq / a.nkv, TPB = AR_ROWS / G;
    // (the tokens with the most keys first)
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * TPB;
    const int ntok = min(TPB, num_tokens - t0), nrows = ntok * G;
    const size_t page_elems = (size_t)2 * a.nkv * a.page_size * HD;
    const size_t v_off = (size_t)a.nkv * a.page_size * HD;
    const float* head_base = kv_cache + (size_t)kvh * a.page_size * HD;
    // rows to make again; keys of a tile that are not finite, while the rows that see them are marked
    __shared__ unsigned long long bad_rows, bad_keys[AR_GROUPS];
    if (threadIdx.x == 0) bad_rows = bad_keys[0] = bad_keys[1] = 0ull;
    auto put = [&](bf16* to, int plane, const float4 v) {
        uint32_t x[3], y[3];
        bool finite = ap_split(v.x, v.y, x);
        finite = ap_split(v.z, v.w, y) && finite;
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(to + i * plane) = make_uint2(x[i], y[i]);
        return finite;
    };
    // (a query that is not finite spoils its own row alone, whose result tells)
    for (int c = threadIdx.x; c < AR_ROWS * (HD / 4); c += AR_GROUPS * AR_THREADS) {
        const int r = c / (HD / 4), d = (c % (HD / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nrows)
            v = *reinterpret_cast<const float4*>(q + (size_t)(t0 + r / G) * a.q_stride + (size_t)(kvh * G + r % G) * HD + d);
        put(q_p + r * LD + d, QPLANE, v);
    }
    __syncthreads();

    for (int s0 = 0; s0 < ntok;) {
        // tokens s0 .. s1-1 of the block belong to one request; every warp looks at them all, a token a lane (one
        // after the other 16 of them took 3 us)
        const int req = token_req[t0 + s0];
        int s1 = s0, lo_min = 0x7fffffff, hi_max = 0;
        for (bool more = true; more && s1 < ntok;) {
            const int tk = s1 + lane;
            const bool same = tk < ntok && token_req[t0 + min(tk, ntok - 1)] == req;
            const int run = __ffs(~__ballot_sync(0xffffffffu, same)) - 1;          // (-1: all 32)
            const bool in = run < 0 || lane < run;
            const int hi = in ? cache_pos[t0 + tk] + 1 : 0;
            const int lo = !in ? 0x7fffffff : (a.window > 0 && hi > a.window) ? hi - a.window : 0;
            lo_min = min(lo_min, (int)__reduce_min_sync(0xffffffffu, (unsigned)lo));
            hi_max = max(hi_max, (int)__reduce_max_sync(0xffffffffu, (unsigned)hi));
            more = run < 0;
            s1 += run < 0 ? 32 : run;
        }
        const int* bt = block_table + (size_t)req * a.bt_stride;
        int lo_r[2], hi_r[2];                      // the keys that this thread's rows see
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = rt * 16 + g + 8 * i, tk = r / G;
            lo_r[i] = hi_r[i] = 0;                 // a row of another request: idle
            if (r < nrows && tk >= s0 && tk < s1) {
                hi_r[i] = cache_pos[t0 + tk] + 1;
                lo_r[i] = (a.window > 0 && hi_r[i] > a.window) ? hi_r[i] - a.window : 0;
            }
        }
        const int warp_hi = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(hi_r[0], hi_r[1]));
        float4 k_next[U], v_next[U];
        auto fetch = [&](int key0) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int c = tid + u * AR_THREADS, key = key0 + c / (HD / 4), d = (c % (HD / 4)) * 4;
                k_next[u] = v_next[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (key >= lo_min && key < hi_max) {
                    const float* src = head_base + (size_t)bt[key / a.page_size] * page_elems +
                                       (size_t)(key % a.page_size) * HD + d;
                    k_next[u] = *reinterpret_cast<const float4*>(src);
                    v_next[u] = *reinterpret_cast<const float4*>(src + v_off);
                }
            }
        };
        float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[VT][4];
#pragma unroll
        for (int v = 0; v < VT; ++v) o[v][0] = o[v][1] = o[v][2] = o[v][3] = 0.f;
        const int tile0 = lo_min / KEYS;
        const int first = (tile0 + ((tile0 ^ group) & 1)) * KEYS;       // even tiles: group 0
        if (first < hi_max) fetch(first);
        for (int key0 = first; key0 < hi_max; key0 += AR_GROUPS * KEYS) {
            group_sync();                          // the tile before is done with
            bool finite = true;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int c = tid + u * AR_THREADS, at = c / (HD / 4) * LD + (c % (HD / 4)) * 4;
                finite = put(k_p + at, KPLANE, k_next[u]) && finite;
                finite = put(v_p + at, KPLANE, v_next[u]) && finite;
            }
            if (any_of_group(!finite)) {
#pragma unroll 1
                for (int c = tid; c < KEYS * (HD / 4); c += AR_THREADS) {
                    const int key = c / (HD / 4), d = (c % (HD / 4)) * 4, there = key0 + key;
                    if (there < lo_min || there >= hi_max) continue;
                    const float* src = head_base + (size_t)bt[there / a.page_size] * page_elems +
                                       (size_t)(there % a.page_size) * HD + d;
                    ap_zero(k_p + key * LD + d, KPLANE, src, &bad_keys[group], key);
                    ap_zero(v_p + key * LD + d, KPLANE, src + v_off, &bad_keys[group], key);
                }
                group_sync();
                const unsigned long long keys = bad_keys[group];
                ap_mark(keys, key0, lo_r[0], hi_r[0], rt * 16 + g, &bad_rows);
                ap_mark(keys, key0, lo_r[1], hi_r[1], rt * 16 + g + 8, &bad_rows);
                group_sync();
                if (tid == 0) bad_keys[group] = 0ull;
            }
            if (key0 + AR_GROUPS * KEYS < hi_max) fetch(key0 + AR_GROUPS * KEYS);
            const int mine = key0 + half * HALF;                         // this warp's first key
            if (mine >= warp_hi || mine + HALF <= lo_min) continue;
            float s[NT][4], rest[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = rest[n][i] = 0.f;
            const uint32_t q_at = smem_u32(q_p + (rt * 16 + (lane & 15)) * LD + (lane >> 4) * 8);
            const uint32_t k_at = smem_u32(k_p + (half * HALF + (lane & 7) + (lane >> 4) * 8) * LD + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int k = 0; k < HD / 16; ++k) {
                uint32_t A[3][4];
#pragma unroll
                for (int i = 0; i < 3; ++i) ldmatrix_x4(A[i], q_at + (i * QPLANE + k * 16) * 2);
#pragma unroll
                for (int n = 0; n < NT; n += 2)
#pragma unroll
                    for (int i = 2; i >= 0; --i) {
                        uint32_t B[4];
                        ldmatrix_x4(B, k_at + (i * KPLANE + n * 8 * LD + k * 16) * 2);
#pragma unroll
                        for (int j = 2 - i; j >= 0; --j) {
                            float (&x)[4] = i + j == 0 ? s[n] : rest[n];
                            float (&y)[4] = i + j == 0 ? s[n + 1] : rest[n + 1];
                            mma_bf16_16816(x, A[j], B[0], B[1]);
                            mma_bf16_16816(y, A[j], B[2], B[3]);
                        }
                    }
            }
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int key = mine + n * 8 + 2 * c4 + (i & 1), r = i >> 1;
                    s[n][i] = key >= lo_r[r] && key < hi_r[r] ? (s[n][i] + rest[n][i]) * a.scale : -INFINITY;
                    mx[r] = fmaxf(mx[r], s[n][i]);
                }
            float alpha[2];
            bool none[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
                const float m_new = fmaxf(m[r], mx[r]);
                none[r] = m_new == -INFINITY;                  // the row has seen no key yet
                alpha[r] = none[r] ? 1.f : expf(m[r] - m_new);
                m[r] = m_new;
                l[r] *= alpha[r];
            }
            uint32_t P[3][KT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float x = none[r] ? 0.f : expf(s[n][2 * r] - m[r]), y = none[r] ? 0.f : expf(s[n][2 * r + 1] - m[r]);
                    l[r] += x + y;
                    uint32_t p[3];
                    ap_split(x, y, p);
#pragma unroll
                    for (int i = 0; i < 3; ++i) P[i][n / 2][(n & 1) * 2 + r] = p[i];
                }
            const uint32_t v_at = smem_u32(v_p + (half * HALF + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + (lane >> 4) * 8);
#pragma unroll
            for (int v = 0; v < VT; v += 2) {
                float x[2][4], y[2][4];
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[n][i] = y[n][i] = 0.f;
#pragma unroll
                for (int k = 0; k < KT; ++k)
#pragma unroll
                    for (int i = 2; i >= 0; --i) {
                        uint32_t B[4];
                        ldmatrix_x4_trans(B, v_at + (i * KPLANE + k * 16 * LD + v * 8) * 2);
#pragma unroll
                        for (int j = 2 - i; j >= 0; --j) {
                            mma_bf16_16816(i + j == 0 ? x[0] : y[0], P[j][k], B[0], B[1]);
                            mma_bf16_16816(i + j == 0 ? x[1] : y[1], P[j][k], B[2], B[3]);
                        }
                    }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[v + n][i] = fmaf(o[v + n][i], alpha[i >> 1], x[n][i] + y[n][i]);
            }
        }
        // the shares of all warps but the first four pass through the tiles' place
        constexpr int OLD = HD + 8;                // floats between rows of a share: eight rows meet no bank twice
        float* shares = reinterpret_cast<float*>(q_p + 3 * QPLANE);      // [3][ROWS][OLD]
        float2* share_ml = reinterpret_cast<float2*>(shares + 3 * AR_ROWS * OLD);    // [3][ROWS]
        const int share = group * 2 + half - 1;
        __syncthreads();                           // all tiles are done with
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
            l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
            if (share < 0) continue;
            const int row = share * AR_ROWS + rt * 16 + g + 8 * r;
            if (c4 == 0) share_ml[row] = make_float2(m[r], l[r]);
#pragma unroll
            for (int v = 0; v < VT; ++v)
                *reinterpret_cast<float2*>(shares + row * OLD + v * 8 + 2 * c4) = make_float2(o[v][2 * r], o[v][2 * r + 1]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (share >= 0 || hi_r[r] == 0) continue;
            const int row = rt * 16 + g + 8 * r;
            float2 ml[3];
            float top = m[r];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                ml[i] = share_ml[i * AR_ROWS + row];
                top = fmaxf(top, ml[i].x);
            }
            const float w[4] = {expf(m[r] - top), expf(ml[0].x - top), expf(ml[1].x - top), expf(ml[2].x - top)};  // (no key: 0)
            float sum = l[r] * w[0], all = 0.f;
#pragma unroll
            for (int i = 0; i < 3; ++i) sum = fmaf(ml[i].y, w[i + 1], sum);
            float* dst = out + (size_t)(t0 + row / G) * a.nq * HD + (size_t)(kvh * G + row % G) * HD + 2 * c4;
#pragma unroll
            for (int v = 0; v < VT; ++v) {
                float x = o[v][2 * r] * w[0], y = o[v][2 * r + 1] * w[0];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float2 f = *reinterpret_cast<const float2*>(shares + (i * AR_ROWS + row) * OLD + v * 8 + 2 * c4);
                    x = fmaf(f.x, w[i + 1], x);
                    y = fmaf(f.y, w[i + 1], y);
                }
                x /= sum;
                y /= sum;
                all += x + y;
                *reinterpret_cast<float2*>(dst + v * 8) = make_float2(x, y);
            }
            if (!isfinite(all)) atomicOr(&bad_rows, 1ull << row);
        }
        __syncthreads();                           // the shares have been read
        s0 = s1;
    }
    if (const unsigned long long bad = bad_rows)      // (written before the last sync)
        ar_block_fma<HD>(q, out, kv_cache, block_table, token_req, cache_pos, a, num_tokens, bad);
}

// ------------------------------------------------------------------ float single tokens
// One token's attention, a block for four query heads of a kv head (blockIdx.z: which four of its
// group): scores of up to 512 keys into shared memory, their softmax statistics, then the values.  HD / 16
// lanes share a key, HD / 4 a value, each 16 bytes at a time, so a warp has 8 to 16 rows in flight
// and nothing is staged; warps take the keys in turn and their sums are added at the end in a fixed
// order: a row's result does not depend on what else is in the batch.  Bound by the latency of three
// dependent rounds of loads (table, keys, values).  20 tokens on 100 to 200 keys with 32 / 8 heads of
// 64: 156 us with the kernel above (keys of 32 staged by one load a thread at a time), 13 us here.
#define AT_THREADS 256
#define AT_KEYS 512

template <int HD>
__global__ void __launch_bounds__(AT_THREADS)
attention_token_f32_kernel(const float* __restrict__ q, float* __restrict__ out,
                           const float* __restrict__ kv_cache, const int* __restrict__ block_table,
                           const int* __restrict__ token_req, const int* __restrict__ cache_pos, AttnArgs a) {
    constexpr int WARPS = AT_THREADS / 32;
    constexpr int KL = HD / 16, KEYS = 32 / KL;    // lanes a key, keys a warp at a time
    constexpr int VL = HD / 4, VALS = 32 / VL;     // lanes a value row
    constexpr int U = 4;                           // rows a lane has in flight
    __shared__ float4 s_s[AT_KEYS];                // scores, then probabilities, of the four heads
    __shared__ size_t at_s[AT_KEYS];               // where a key's row begins
    __shared__ float4 stat_s[2];                   // per head: the factor for older sums, the sum
    __shared__ float4 acc_s[WARPS][4][HD / 4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x, kvh = blockIdx.y, G = a.nq / a.nkv, g0 = blockIdx.z * 4, heads = min(4, G - g0);
    const int hi = cache_pos[t] + 1;
    const int lo = (a.window > 0 && hi > a.window) ? hi - a.window : 0;
    const int* bt = block_table + (size_t)token_req[t] * a.bt_stride;
    const size_t page_elems = (size_t)2 * a.nkv * a.page_size * HD;
    const size_t v_off = (size_t)a.nkv * a.page_size * HD;
    const float* head_base = kv_cache + (size_t)kvh * a.page_size * HD;

    // this lane's part of the queries: floats 4 (KL i + lane % KL) ..
    const int kl = lane % KL, vl = lane % VL;
    ulonglong2 qv[4][4];
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            qv[h][i] = *reinterpret_cast<const ulonglong2*>(
                q + (size_t)t * a.q_stride + (size_t)(kvh * G + g0 + min(h, heads - 1)) * HD + (i * KL + kl) * 4);

    float m = -INFINITY, l = 0.f;                  // of head `warp`, in the first four warps
    unsigned long long acc[4][2];
#pragma unroll
    for (int h = 0; h < 4; ++h) acc[h][0] = acc[h][1] = 0ull;

    for (int base = lo; base < hi; base += AT_KEYS) {
        const int n = min(AT_KEYS, hi - base);
        for (int j = tid; j < n; j += AT_THREADS) {
            const int key = base + j, page = key / a.page_size;
            at_s[j] = (size_t)bt[page] * page_elems + (size_t)(key - page * a.page_size) * HD;
        }
        __syncthreads();
        for (int j0 = warp * KEYS + lane / KL; j0 < n; j0 += WARPS * KEYS * 2) {
            ulonglong2 kv[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float* row = head_base + at_s[min(j0 + u * WARPS * KEYS, n - 1)];
#pragma unroll
                for (int i = 0; i < 4; ++i) kv[u][i] = *reinterpret_cast<const ulonglong2*>(row + (i * KL + kl) * 4);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float dot[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    unsigned long long d = 0ull;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        ar_fma2(d, qv[h][i].x, kv[u][i].x);
                        ar_fma2(d, qv[h][i].y, kv[u][i].y);
                    }
                    dot[h] = ar_lo(d) + ar_hi(d);
                }
                // (lanes of a key leave the loop together, those of one warp may not)
                const unsigned mask = ((KL == 32 ? 0u : 1u << KL) - 1u) << (lane & ~(KL - 1));
#pragma unroll
                for (int h = 0; h < 4; ++h)
#pragma unroll
                    for (int o = KL / 2; o > 0; o >>= 1) dot[h] += __shfl_xor_sync(mask, dot[h], o);
                if (kl == 0 && j0 + u * WARPS * KEYS < n)
                    s_s[j0 + u * WARPS * KEYS] =
                        make_float4(dot[0] * a.scale, dot[1] * a.scale, dot[2] * a.scale, dot[3] * a.scale);
            }
        }
        __syncthreads();
        if (warp < 4) {
            float* s = reinterpret_cast<float*>(s_s) + warp;
            float mx = -INFINITY;
            for (int j = lane; j < n; j += 32) mx = fmaxf(mx, s[4 * j]);
            const float m_new = fmaxf(m, warp_max(mx));
            float sum = 0.f;
            for (int j = lane; j < n; j += 32) {
                const float p = expf(s[4 * j] - m_new);
                sum += p;
                s[4 * j] = p;
            }
            const float alpha = expf(m - m_new);   // 0 on the first round
            l = l * alpha + warp_sum(sum);
            m = m_new;
            if (lane == 0) {
                reinterpret_cast<float*>(stat_s)[warp] = alpha;
                reinterpret_cast<float*>(stat_s)[4 + warp] = l;
            }
        }
        __syncthreads();
        const float4 al = stat_s[0];
        const float alpha[4] = {al.x, al.y, al.z, al.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const unsigned long long f = ar_pack(alpha[h], alpha[h]);
            asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[h][0]) : "l"(f));
            asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[h][1]) : "l"(f));
        }
        for (int j0 = warp * VALS + lane / VL; j0 < n; j0 += WARPS * VALS * U) {
            ulonglong2 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                v[u] = *reinterpret_cast<const ulonglong2*>(head_base + v_off + at_s[min(j0 + u * WARPS * VALS, n - 1)] +
                                                            vl * 4);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j0 + u * WARPS * VALS >= n) break;
                const float4 p4 = s_s[j0 + u * WARPS * VALS];
                const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const unsigned long long pp = ar_pack(p[h], p[h]);
                    ar_fma2(acc[h][0], pp, v[u].x);
                    ar_fma2(acc[h][1], pp, v[u].y);
                }
            }
        }
        __syncthreads();                           // scores and places are done with
    }
    // the two value rows of a warp (HD 64), then the warps, in order
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        float r[4] = {ar_lo(acc[h][0]), ar_hi(acc[h][0]), ar_lo(acc[h][1]), ar_hi(acc[h][1])};
        if (VALS == 2)
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] += __shfl_xor_sync(0xffffffffu, r[i], 16);
        if (lane < VL) acc_s[warp][h][vl] = make_float4(r[0], r[1], r[2], r[3]);
    }
    __syncthreads();
    for (int i = tid; i < heads * HD; i += AT_THREADS) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) sum += reinterpret_cast<const float*>(acc_s[w])[i];
        out[(size_t)t * a.nq * HD + (size_t)(kvh * G + g0) * HD + i] =
            sum / reinterpret_cast<const float*>(stat_s)[4 + i / HD];
    }
}

template <int HD>
static int launch_rows_f32(const float* q, float* out, const float* kv, const int* block_table,
                           const int* token_req, const int* cache_pos, const AttnArgs& a, int num_tokens,
                           cudaStream_t s) {
    constexpr int fma = (int)sizeof(float) * (AR_ROWS * (HD + 4) +
                                              AR_GROUPS * (AR_KEYS * (HD + 4) + AR_KEYS * HD + AR_ROWS * (AR_KEYS + 4)));
    constexpr int smem = fma > ap_smem<HD>() ? fma : ap_smem<HD>();
    static_assert(smem - 6 * AR_ROWS * (HD + 8) >= 3 * AR_ROWS * ((HD + 8) * 4 + 8), "room for the shares");
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(attention_rows_f32_kernel<HD>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int per_block = AR_ROWS / (a.nq / a.nkv);
    attention_rows_f32_kernel<HD><<<dim3(a.nkv, (num_tokens + per_block - 1) / per_block),
                                     AR_GROUPS * AR_THREADS, smem, s>>>(
        q, out, kv, block_table, token_req, cache_pos, a, num_tokens);
    return launch_status();
}

// `portions`: the tokens come in runs of one request.  Returns 0, a CUDA error code, or -1 when
// the shape is refused (group * head_dim > 4096 or head_dim > 256).
MSTAR_API int mstar_paged_attention_generic(const void* q, int q_stride, void* out,
                                            const void* kv_cache, const int* block_table,
                                            int bt_stride, const int* token_req,
                                            const int* cache_pos, int num_tokens, int nq, int nkv,
                                            int hd, int page_size, int window, float scale,
                                            int act_dtype, int portions, void* stream) {
    if (num_tokens <= 0) return 0;
    if (nkv <= 0 || nq % nkv != 0) return -1;
    const int G = nq / nkv;
    if (G * hd > ATT_MAX_ACC * ATT_THREADS || hd > 256) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    AttnArgs a{nq, nkv, hd, page_size, bt_stride, window, q_stride, scale};
    const bool rows_of_16 = act_dtype == MSTAR_F32 && (hd == 64 || hd == 128) && q_stride % 4 == 0 &&
                            (((uintptr_t)q | (uintptr_t)kv_cache | (uintptr_t)out) & 15) == 0;
    if (portions && rows_of_16 && G <= AR_ROWS && num_tokens <= 65535) {
        return hd == 64 ? launch_rows_f32<64>((const float*)q, (float*)out, (const float*)kv_cache, block_table,
                                              token_req, cache_pos, a, num_tokens, s)
                        : launch_rows_f32<128>((const float*)q, (float*)out, (const float*)kv_cache, block_table,
                                               token_req, cache_pos, a, num_tokens, s);
    }
    if (rows_of_16 && nkv <= 65535) {
        const dim3 grid(num_tokens, nkv, (G + 3) / 4);
        auto kernel = hd == 64 ? attention_token_f32_kernel<64> : attention_token_f32_kernel<128>;
        kernel<<<grid, AT_THREADS, 0, s>>>((const float*)q, (float*)out, (const float*)kv_cache, block_table, token_req,
                                           cache_pos, a);
        return launch_status();
    }
    const size_t smem = sizeof(float) * ((size_t)G * hd + (size_t)ATT_TILE * (hd + 1) +
                                         (size_t)G * ATT_TILE + 3 * (size_t)G);
    dim3 grid(num_tokens, nkv);
    static size_t configured_f32 = 0, configured_bf16 = 0;  // largest size set so far
    if (act_dtype == MSTAR_F32) {
        if (smem > 48 * 1024 && smem > configured_f32) {
            cudaFuncSetAttribute(paged_attention_generic_kernel<float>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            configured_f32 = smem;
        }
        paged_attention_generic_kernel<float><<<grid, ATT_THREADS, smem, s>>>(
            (const float*)q, (float*)out, (const float*)kv_cache, block_table, token_req, cache_pos, a);
    } else {
        if (smem > 48 * 1024 && smem > configured_bf16) {
            cudaFuncSetAttribute(paged_attention_generic_kernel<bf16>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            configured_bf16 = smem;
        }
        paged_attention_generic_kernel<bf16><<<grid, ATT_THREADS, smem, s>>>(
            (const bf16*)q, (bf16*)out, (const bf16*)kv_cache, block_table, token_req, cache_pos, a);
    }
    return launch_status();
}
