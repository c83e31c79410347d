// Routed experts: choosing the experts of a token, and the experts' gated feed-forwards on
// the rows that chose them.
//
//   scores  s = sigmoid(z) or softmax(z) over a token's float router logits z
//   chosen  the `top` largest scores (the lower index wins a tie), weight w = s, or s divided
//           by the sum of the chosen scores when `renormalize`
//           With a `choice_bias` the largest of s + bias are chosen; the weights stay s.
//           With `groups` > 0 the experts form that many equal groups of neighbours, a group
//           counts as its largest choice score, and only experts of the best `keep` groups can
//           be chosen.  `renorm_eps` is added to the sum the chosen scores are divided by;
//           `weight_scale` multiplies the weights at the end.
//   expert  y = W_down (silu(W_gate u) * (W_up u)),  u = w x (`scale_input`) or u = x with
//           w multiplying y; without a gate (`gated` 0) y = W_down relu(W_up u)^2; `gated` 2
//           takes the clamped swish of common.cuh (limit, alpha) for the SiLU and the product
//   out[t] = sum over the chosen experts (+ `add[t]`, the shared expert's output, times
//           sigmoid(add_gate[t]) where there is such a gate)
// A chosen index at or beyond `real` (the experts that have matrices) is an identity
// expert: it adds w x[t].
//
// Expert matrices are stacked expert after expert: gate_up [experts][2 * ff][width] (gate
// rows first; [experts][ff][width] without a gate), down [experts][width][ff].
//
// These are the kernels for a step's rows as they come (token by token, each row streaming
// the weights of its experts): dot products on CUDA cores, float sums in a fixed order, so a
// row's result does not depend on what else is in the batch.  Scaling the input by w is done
// on the sums (W (w x) = w (W x)), which is the same number without rounding w x first.
#include "common.cuh"

// ------------------------------------------------------------------ choice
// A warp per token: lane l holds the logits of experts l, l + 32, ... (up to 32 of them, so up
// to 1,024 experts); the largest logit not chosen yet is found `top` times by a warp-wide
// comparison of (value, index), the lower index winning a tie.  Scores are monotone in the
// logits, so the choice is made on the logits.
#define RT_PER_LANE 32
#define RT_MAX_GROUPS 1024

// The index of the largest value of a warp's lanes (a lane offers value bz at index be), the lower
// index winning a tie; an index of 0x7fffffff is no candidate.  Two integer reductions on keys that
// order as the floats do.
__device__ __forceinline__ int rt_warp_best(float bz, int be) {
    const unsigned bits = __float_as_uint(bz + 0.f);                 // (-0 and 0 are equal)
    const unsigned key = be == 0x7fffffff ? 0u : (bits & 0x80000000u) ? ~bits : bits | 0x80000000u;
    const unsigned most = __reduce_max_sync(0xffffffffu, key);
    return (int)__reduce_min_sync(0xffffffffu, key == most ? (unsigned)be : 0x7fffffffu);
}

// The choice where it cannot be read off the logits alone: choice scores s + bias are made once
// and kept in shared memory, and, with groups, the experts of all but the best `keep` groups are
// closed.  A warp per token; the scores of a row lie at dynamic shared memory [warp][experts], the
// groups' after all warps' scores ([warp][groups]).
__global__ void route_choice_kernel(const float* __restrict__ logits, const float* __restrict__ choice_bias,
                                     int* __restrict__ chosen, float* __restrict__ weight, int tokens,
                                     int experts, int top, int softmax, int renormalize, int ld,
                                     int groups, int keep, float renorm_eps, float weight_scale) {
    extern __shared__ float rt_sm[];
    logits = pdl_after(logits, pdl_wait());
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int t = blockIdx.x * nwarps + warp;
    if (t >= tokens) return;
    const float* z = logits + (size_t)t * ld;
    float* choice = rt_sm + (size_t)warp * experts;
    float* best = rt_sm + (size_t)nwarps * experts + (size_t)warp * groups;
    float zmax = -INFINITY, denom = 1.f;
    if (softmax) {
        for (int e = lane; e < experts; e += 32) zmax = fmaxf(zmax, z[e]);
        zmax = warp_max(zmax);
        denom = 0.f;
        for (int e = lane; e < experts; e += 32) denom += expf(z[e] - zmax);
        denom = warp_sum(denom);
    }
    auto score = [&](float v) { return softmax ? expf(v - zmax) / denom : 1.f / (1.f + expf(-v)); };
    for (int e = lane; e < experts; e += 32)
        choice[e] = score(z[e]) + (choice_bias != nullptr ? choice_bias[e] : 0.f);
    __syncwarp();
    const int per = groups > 0 ? experts / groups : experts;
    // bit i: expert lane + 32 i cannot be chosen (any more)
    unsigned closed = 0u;
    if (groups > 0 && keep < groups) {
        for (int g = lane; g < groups; g += 32) {
            float m = choice[g * per];
            for (int j = 1; j < per; ++j) m = fmaxf(m, choice[g * per + j]);
            best[g] = m;
        }
        __syncwarp();
        unsigned open_groups = 0u;              // bit i: group lane + 32 i is kept
        for (int k = 0; k < keep; ++k) {
            float bz = -INFINITY;
            int be = 0x7fffffff;
            for (int i = 0, g = lane; g < groups; ++i, g += 32)
                if (!((open_groups >> i) & 1u) && (be == 0x7fffffff || best[g] > bz)) {
                    bz = best[g];
                    be = g;
                }
            be = rt_warp_best(bz, be);
            if ((be & 31) == lane) open_groups |= 1u << (be >> 5);
        }
        // the mark of a kept group goes where every lane reads it
        __syncwarp();
        for (int i = 0, g = lane; g < groups; ++i, g += 32) best[g] = (open_groups >> i) & 1u ? 1.f : 0.f;
        __syncwarp();
        for (int i = 0, e = lane; e < experts; ++i, e += 32)
            if (best[e / per] == 0.f) closed |= 1u << i;
    }
    float total = 0.f;
    for (int k = 0; k < top; ++k) {
        float bz = -INFINITY;
        int be = 0x7fffffff;
        for (int i = 0, e = lane; e < experts; ++i, e += 32)
            if (!((closed >> i) & 1u) && (be == 0x7fffffff || choice[e] > bz)) {
                bz = choice[e];
                be = e;
            }
        be = rt_warp_best(bz, be);
        if ((be & 31) == lane) closed |= 1u << (be >> 5);
        const float s = score(z[be]);
        total += s;
        if (lane == 0) {
            chosen[(size_t)t * top + k] = be;
            weight[(size_t)t * top + k] = s;
        }
    }
    if (lane == 0) {
        const float div = renormalize ? total + renorm_eps : 1.f;
        for (int k = 0; k < top; ++k)
            weight[(size_t)t * top + k] = weight[(size_t)t * top + k] / div * weight_scale;
    }
}

__global__ void route_topk_kernel(const float* __restrict__ logits,
                                  int* __restrict__ chosen,
                                  float* __restrict__ weight, int tokens, int experts, int top,
                                  int softmax, int renormalize, int ld) {
    logits = pdl_after(logits, pdl_wait());
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= tokens) return;
    const float* z = logits + (size_t)t * ld;
    float zmax = -INFINITY, denom = 1.f;
    if (softmax) {
        for (int e = lane; e < experts; e += 32) zmax = fmaxf(zmax, z[e]);
        zmax = warp_max(zmax);
        denom = 0.f;
        for (int e = lane; e < experts; e += 32) denom += expf(z[e] - zmax);
        denom = warp_sum(denom);
    }
    unsigned taken = 0u;                       // bit i: expert lane + 32 i is chosen
    float total = 0.f;
    for (int k = 0; k < top; ++k) {
        float bz = -INFINITY;
        int be = 0x7fffffff;
        for (int i = 0; i < RT_PER_LANE; ++i) {
            const int e = lane + 32 * i;
            if (e >= experts) break;
            if (!((taken >> i) & 1u)) {
                const float v = z[e];                 // scores are monotone in the logits
                if (be == 0x7fffffff || v > bz) {
                    bz = v;
                    be = e;
                }
            }
        }
        be = rt_warp_best(bz, be);
        if ((be & 31) == lane) taken |= 1u << (be >> 5);
        const float zb = z[be];
        const float s = softmax ? expf(zb - zmax) / denom : 1.f / (1.f + expf(-zb));
        total += s;
        if (lane == 0) {
            chosen[(size_t)t * top + k] = be;
            weight[(size_t)t * top + k] = s;
        }
    }
    if (renormalize && lane == 0)
        for (int k = 0; k < top; ++k) weight[(size_t)t * top + k] /= total;
}

MSTAR_API int mstar_route_topk(const float* logits, const float* choice_bias, int* chosen,
                               float* weight, int tokens, int experts, int top, int softmax,
                               int renormalize, int ld, int groups, int keep, float renorm_eps,
                               float weight_scale, void* stream) {
    if (tokens <= 0) return 0;
    if (ld < experts) return -1;
    if (experts <= 0 || top <= 0 || top > experts || experts > 32 * RT_PER_LANE) return -1;
    if (groups > 0 && (groups > RT_MAX_GROUPS || experts % groups || keep <= 0 || keep > groups ||
                       top > experts / groups * keep))
        return -1;
    if (groups > 0 || choice_bias != nullptr || renorm_eps != 0.f || weight_scale != 1.f) {
        // four warps' scores: at most 4 * (1,024 + 1,024) floats
        const size_t smem = sizeof(float) * 4 * (size_t)(experts + (groups > 0 ? groups : 0));
        mstar_launch(route_choice_kernel, dim3((tokens + 3) / 4), dim3(128), smem, (cudaStream_t)stream,
                     logits, choice_bias, chosen, weight, tokens, experts, top, softmax, renormalize,
                     ld, groups, keep, renorm_eps, weight_scale);
        return launch_status();
    }
    mstar_launch(route_topk_kernel, dim3((tokens + 3) / 4), dim3(128), 0, (cudaStream_t)stream,
                 logits, chosen, weight, tokens, experts, top, softmax, renormalize, ld);
    return launch_status();
}

// ------------------------------------------------------------------ gate / up
// One block per (row = token x choice, slice of 32 hidden units); a warp per hidden unit,
// lanes along the width.
#define RE_THREADS 256
#define RE_UNITS 32

template <typename A, bool GATED>
__global__ void __launch_bounds__(RE_THREADS)
expert_gate_up_kernel(const A* __restrict__ x, const A* __restrict__ w_gate_up,
                      const int* __restrict__ chosen, const float* __restrict__ weight,
                      float* __restrict__ act, int width, int ff, int top, int scale_input,
                      int real, int clamped, float limit, float alpha) {
    extern __shared__ float xs[];            // [width]
    const int row = blockIdx.x, t = row / top;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long waited = pdl_wait();
    x = pdl_after(x, waited);
    chosen = pdl_after(chosen, waited);
    weight = pdl_after(weight, waited);
    for (int i = threadIdx.x; i < width; i += RE_THREADS) xs[i] = to_float(x[(size_t)t * width + i]);
    __syncthreads();
    const int e = chosen[row];
    if (e >= real) return;                     // an identity expert has no hidden units
    const float w = scale_input ? weight[row] : 1.f;
    const A* base = w_gate_up + (size_t)e * (GATED ? 2 : 1) * ff * width;
    // rows start at multiples of `width` elements: 8-element loads where that is aligned
    const bool vec = width % 8 == 0 && ((uintptr_t)w_gate_up & 31) == 0;
    // a warp takes four hidden units at a time: eight rows of weights stream side by side
    const int u_end = min(ff, (int)(blockIdx.y + 1) * RE_UNITS);
    for (int u0 = blockIdx.y * RE_UNITS + warp * 4; u0 < u_end; u0 += (RE_THREADS / 32) * 4) {
        float sg[4] = {0.f, 0.f, 0.f, 0.f}, su[4] = {0.f, 0.f, 0.f, 0.f};
        if (vec) {
            for (int c = lane; c < (width >> 3); c += 32) {
                float a8[4][8], b8[4][8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int u = min(u0 + k, ff - 1);          // a unit past the end repeats the last
                    load8(base + (size_t)u * width + 8 * c, a8[k]);
                    if (GATED) load8(base + (size_t)(ff + u) * width + 8 * c, b8[k]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float xv = xs[8 * c + i];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        sg[k] = fmaf(a8[k][i], xv, sg[k]);
                        if (GATED) su[k] = fmaf(b8[k][i], xv, su[k]);
                    }
                }
            }
        } else {
            for (int i = lane; i < width; i += 32) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int u = min(u0 + k, ff - 1);
                    sg[k] = fmaf(to_float(base[(size_t)u * width + i]), xs[i], sg[k]);
                    if (GATED) su[k] = fmaf(to_float(base[(size_t)(ff + u) * width + i]), xs[i], su[k]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float g = warp_sum(sg[k]) * w;
            float v;
            if (GATED) {
                const float up = warp_sum(su[k]) * w;
                v = clamped ? clamped_swish(g, up, limit, alpha) : g / (1.f + expf(-g)) * up;
            } else {
                const float r = fmaxf(g, 0.f);
                v = r * r;
            }
            if (lane == 0 && u0 + k < u_end) act[(size_t)row * ff + u0 + k] = v;
        }
    }
}

// ------------------------------------------------------------------ down (+ sum, + shared)
template <typename A>
__global__ void __launch_bounds__(RE_THREADS)
expert_down_kernel(const float* __restrict__ act, const A* __restrict__ w_down,
                   const int* __restrict__ chosen, const float* __restrict__ weight,
                   const A* __restrict__ add, A* __restrict__ out, int width, int ff, int top,
                   int scale_input, const A* __restrict__ x, int real, const float* add_gate,
                   int gate_stride) {
    extern __shared__ float as[];            // [top][ff]
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long waited = pdl_wait();
    act = pdl_after(act, waited);
    add = pdl_after(add, waited);
    x = pdl_after(x, waited);
    add_gate = pdl_after(add_gate, waited);
    const float share = add_gate == nullptr ? 1.f : 1.f / (1.f + expf(-add_gate[(size_t)t * gate_stride]));
    for (int i = threadIdx.x; i < top * ff; i += RE_THREADS)
        as[i] = chosen[(size_t)t * top + i / ff] < real ? act[(size_t)t * top * ff + i] : 0.f;
    __syncthreads();
    const bool vec = ff % 8 == 0 && ((uintptr_t)w_down & 31) == 0;
    const int c_end = min(width, (int)(blockIdx.y + 1) * RE_UNITS);
    for (int c0 = blockIdx.y * RE_UNITS + warp * 4; c0 < c_end; c0 += (RE_THREADS / 32) * 4) {
        float total[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < top; ++k) {
            const int e = chosen[(size_t)t * top + k];
            if (e >= real) {                   // identity expert: w x[t]
                const float wk = weight[(size_t)t * top + k];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    total[q] += wk * to_float(x[(size_t)t * width + min(c0 + q, width - 1)]);
                continue;
            }
            const A* wexp = w_down + (size_t)e * width * ff;
            float s4[4] = {0.f, 0.f, 0.f, 0.f};
            if (vec) {
                for (int c2 = lane; c2 < (ff >> 3); c2 += 32) {
                    float a8[4][8];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        load8(wexp + (size_t)min(c0 + q, width - 1) * ff + 8 * c2, a8[q]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float av = as[k * ff + 8 * c2 + i];
#pragma unroll
                        for (int q = 0; q < 4; ++q) s4[q] = fmaf(a8[q][i], av, s4[q]);
                    }
                }
            } else {
                for (int j = lane; j < ff; j += 32) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        s4[q] = fmaf(to_float(wexp[(size_t)min(c0 + q, width - 1) * ff + j]), as[k * ff + j], s4[q]);
                }
            }
            const float wk = scale_input ? 1.f : weight[(size_t)t * top + k];
#pragma unroll
            for (int q = 0; q < 4; ++q) total[q] += warp_sum(s4[q]) * wk;
        }
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = c0 + q;
                if (c < c_end) {
                    float v = total[q];
                    if (add != nullptr) v += share * to_float(add[(size_t)t * width + c]);
                    out[(size_t)t * width + c] = from_float<A>(v);
                }
            }
        }
    }
}

// x [tokens, width], chosen / weight [tokens, top]; `act`: float scratch [tokens * top, ff];
// `add`: nullptr or [tokens, width]; out [tokens, width].  Returns 0, a CUDA error code, or
// -1 when a row does not fit shared memory.
MSTAR_API int mstar_experts_by_row(const void* x, const void* w_gate_up, const void* w_down,
                                   const int* chosen, const float* weight, float* act,
                                   const void* add, void* out, int act_dtype, int tokens,
                                   int width, int ff, int top, int scale_input, int gated,
                                   int real, float limit, float alpha, const float* add_gate,
                                   int gate_stride, void* stream) {
    if (tokens <= 0) return 0;
    if (width <= 0 || ff <= 0 || top <= 0) return -1;
    if ((size_t)width * 4 > 48 * 1024 || (size_t)top * ff * 4 > 48 * 1024) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 g1(tokens * top, (ff + RE_UNITS - 1) / RE_UNITS), g2(tokens, (width + RE_UNITS - 1) / RE_UNITS);
#define GO(A, GATED)                                                                              \
    mstar_launch((expert_gate_up_kernel<A, GATED>), g1, dim3(RE_THREADS), sizeof(float) * width, s, \
                 (const A*)x, (const A*)w_gate_up, chosen, weight, act, width, ff, top,            \
                 scale_input, real, (int)(gated == 2), limit, alpha)
    if (act_dtype == MSTAR_F32) {
        if (gated) { GO(float, true); } else { GO(float, false); }
        mstar_launch((expert_down_kernel<float>), g2, dim3(RE_THREADS), sizeof(float) * top * ff, s,
                     (const float*)act, (const float*)w_down, chosen, weight, (const float*)add,
                     (float*)out, width, ff, top, scale_input, (const float*)x, real, add_gate, gate_stride);
    } else {
        if (gated) { GO(bf16, true); } else { GO(bf16, false); }
        mstar_launch((expert_down_kernel<bf16>), g2, dim3(RE_THREADS), sizeof(float) * top * ff, s,
                     (const float*)act, (const bf16*)w_down, chosen, weight, (const bf16*)add,
                     (bf16*)out, width, ff, top, scale_input, (const bf16*)x, real, add_gate, gate_stride);
    }
#undef GO
    return launch_status();
}

// ====================================================================== grouped by expert
// For many rows (prompt portions) the rows are sorted by expert, and every expert's rows go
// through its matrices as tiles of a tensor-core GEMM (tcgen05, bfloat16, float sums in TMEM):
//   1. experts_sort: counting sort of the rows (token x choice) by expert; the list of row
//      tiles (expert, first sorted row), one per 128 rows of a group.
//   2. grouped GEMM, gated: act[p] = silu(w G) * (w U), G and U the products of the gathered
//      token rows with the expert's gate and up rows (bfloat16 out, sorted order).
//   3. grouped GEMM, plain: y[p] = act[p] W_down[e]^T (float out, sorted order).
//   4. experts_combine: out[t] = sum over a token's choices, in the order of the choices,
//      of (w) y[pos] (+ add[t]).
// A row's numbers depend on its own inputs only: the position of a row in its tile changes
// nothing, so the order inside a group need not be stable.
#include "mma_util.cuh"
#include "tma_util.cuh"
#include "tcgen05_util.cuh"

#define GG_BM 128
#define GG_BN 256                 // accumulator columns of a tile
#define GG_BK 64
#define GG_STAGES 4
#define GG_PART_ROWS 32           // rows of the weight boxes of a tile's part
// the producer warp, the MMA warp, four epilogue warps and, where token rows are gathered, four more
__host__ __device__ constexpr int gg_threads(bool gather) { return gather ? 320 : 192; }
#define GG_STORE_LD 36            // floats between rows of an epilogue warp's 32 x 32 staging tile
#define GG_A_BYTES (GG_BM * GG_BK * 2)
#define GG_STAGE_BYTES ((GG_BM + GG_BN) * GG_BK * 2)

// `experts`: all router outputs; tiles are made for the first `real` of them only.  One block of
// 1,024 threads, a thread an expert between the two passes over the rows: 7 us for 8,192 rows and 32
// experts (14 us with one thread making the list and rows asked for one at a time).
__global__ void __launch_bounds__(1024)
experts_sort_kernel(const int* __restrict__ chosen, int rows, int experts, int real,
                    int* __restrict__ order, int* __restrict__ pos, int* __restrict__ offsets,
                    int* __restrict__ tile_expert, int* __restrict__ tile_first,
                    int* __restrict__ num_tiles) {
    __shared__ int cursor[1024];
    __shared__ int warp_rows[32], warp_tiles[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cursor[tid] = 0;
    chosen = pdl_after(chosen, pdl_wait());
    __syncthreads();
    // A row's place in its group is what its expert's counter held before it.  A thread asks for its
    // rows eight at a time and keeps the first eight for the second pass; further ones leave their
    // place in pos.  (Lanes counting together by __match_any_sync were slower than the atomics.)
    int mine[8], place[8];
    for (int r0 = tid; r0 < rows; r0 += 8 * 1024) {
        int e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = r0 + i * 1024 < rows ? chosen[r0 + i * 1024] : -1;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = e[i] >= 0 ? atomicAdd(&cursor[e[i]], 1) : 0;
            if (r0 < 1024) {
                mine[i] = e[i];
                place[i] = at;
            } else if (e[i] >= 0) {
                pos[r0 + i * 1024] = at;
            }
        }
    }
    __syncthreads();
    // exclusive sums over the experts of the rows and of the tiles
    const int n = tid < experts ? cursor[tid] : 0;
    const int t = tid < real ? (n + GG_BM - 1) / GG_BM : 0;
    int rows_to = n, tiles_to = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, rows_to, o), b = __shfl_up_sync(0xffffffffu, tiles_to, o);
        if (lane >= o) {
            rows_to += a;
            tiles_to += b;
        }
    }
    if (lane == 31) {
        warp_rows[warp] = rows_to;
        warp_tiles[warp] = tiles_to;
    }
    __syncthreads();
    for (int w = 0; w < warp; ++w) {
        rows_to += warp_rows[w];
        tiles_to += warp_tiles[w];
    }
    const int first = rows_to - n, tile0 = tiles_to - t;
    if (tid < experts) {
        offsets[tid] = first;
        cursor[tid] = first;
        for (int i = 0; i < t; ++i) {
            tile_expert[tile0 + i] = tid;
            tile_first[tile0 + i] = first + i * GG_BM;
        }
    }
    if (tid == 1023) {
        offsets[experts] = rows_to;
        *num_tiles = tiles_to;
    }
    __syncthreads();
    for (int r0 = tid; r0 < rows; r0 += 8 * 1024) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + i * 1024;
            if (r >= rows) continue;
            const int at = r0 < 1024 ? cursor[mine[i]] + place[i] : cursor[chosen[r]] + pos[r];
            order[at] = r;
            pos[r] = at;
        }
    }
}

struct GroupedArgs {
    void* out;
    const int* order;
    const float* weight;
    const int* offsets;
    const int* tile_expert;
    const int* tile_first;
    const int* num_tiles;
    int N, K, top, n_tiles;       // N: output columns, n_tiles: column tiles of an expert
    int scale_input, clamped;
    float limit, alpha;
};

// Persistent CTAs walk over the tiles (row tile, column tile), a row tile's column tiles one after
// another.  A tile is 128 sorted rows of one expert x 256 rows of its matrix, K in blocks of 64:
//   warp 0     brings the expert's rows by TMA into a ring of four stages, two boxes of 128, and the
//              rows of the down product, which lie in order, as a third;
//   warps 6-9  bring token rows by cp.async (eight lanes a row of 128 bytes, swizzled as TMA would),
//              and tell a stage's barrier two k-blocks later, when they have landed.  (TMA's gather4
//              moved four rows in some 70 cycles, 32 of them a k-block: 128 us where this takes
//              52.)
//   warp 1     one lane issues tcgen05.mma (M 128, N 256, K 16) into one of two accumulators;
//   warps 2-5  turn an accumulator into output rows while the next tile's products run; float rows
//              pass through shared memory so that a store writes whole 128-byte rows.
// MODE 0: plain (down), A rows are act[p], out float.  1: gated gate/up, A rows are x[order[p] /
// top], columns 0..127 of the accumulator are gate rows and 128..255 the up rows of the same hidden
// units, out = act(w G) * (w U) in bfloat16.  2: up alone with relu^2, bfloat16 out.
// Rows of a tile past the group's last are computed from other rows and not stored.
//
// Bound by the operands' way from L2 (48 KB per 512 cycles of MMA and SM) and by the rows that fill
// up a group's last tile.  2,048 tokens x 4 of 32 experts of 512 at width 2,048: gate/up 52 us, down
// 31 us (operands alone: 26 and 9 us of MMA); as mma.sync tiles of 128 x 64 fed by cp.async they took
// 200 and 102 us.
template <int MODE>
__global__ void __launch_bounds__(gg_threads(MODE != 0), 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_part, const bf16* __restrict__ x, GroupedArgs a,
                    int* __restrict__ error_word) {
    constexpr bool GATED = MODE == 1, GATHER = MODE != 0;
    constexpr int OUT_COLS = GATED ? GG_BN / 2 : GG_BN;
    extern __shared__ unsigned char gg_smem[];
    // the swizzle pattern is a function of the address: stage buffers start on 1024 bytes
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(gg_smem) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_bar[GG_STAGES];
    __shared__ __align__(8) uint64_t empty_bar[GG_STAGES];
    __shared__ __align__(8) uint64_t acc_full[2];
    __shared__ __align__(8) uint64_t acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < GG_STAGES; ++s) {
            // the announcement of the TMA bytes, and every thread that gathers
            mbar_init(tc_smem(&full_bar[s]), GATHER ? 1 + 128 : 1);
            mbar_init(tc_smem(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tc_smem(&acc_full[b]), 1);
            mbar_init(tc_smem(&acc_empty[b]), 4);       // the four epilogue warps
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         tc_smem(&tmem_base_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;

    const unsigned long long waited = pdl_wait();
    const int* order = pdl_after(a.order, waited);
    const int* tile_expert = pdl_after(a.tile_expert, waited);
    const int* tile_first = pdl_after(a.tile_first, waited);
    const int* offsets = pdl_after(a.offsets, waited);
    const int total = *pdl_after(a.num_tiles, waited) * a.n_tiles;
    const int num_kb = (a.K + GG_BK - 1) / GG_BK;
    // Rounds of a tile a CTA; the tiles of a last round that would leave half of the CTAs idle or more are
    // cut into two or four parts along N (groups of some 256 rows have a third tile of a few rows as often as
    // not: 320 tiles on 148 SMs, three rounds for 2.2 rounds of work; the layer of 2,048 tokens 183 -> 179 us).
    // Unit u of this CTA: tile, columns per side and the first of them.
    const int grid = (int)gridDim.x, rounds = total / grid, rem = total - rounds * grid;
    const int parts = rem * 4 <= grid ? 4 : rem * 2 <= grid ? 2 : 1;
    const int units = rounds + ((int)blockIdx.x < rem * parts ? 1 : 0);
    struct Unit { int mt, n0, cols; };
    auto unit = [&](int u) {
        const bool last = u == rounds;
        const int t = u * grid + (last ? (int)blockIdx.x / parts : (int)blockIdx.x);
        Unit w;
        w.mt = t / a.n_tiles;
        w.cols = last ? OUT_COLS / parts : OUT_COLS;
        w.n0 = (t - w.mt * a.n_tiles) * OUT_COLS + (last ? (int)blockIdx.x % parts * w.cols : 0);
        return w;
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;                            // k-blocks loaded so far, over all tiles
            bool ok = true;
            for (int u = 0; u < units && ok; ++u) {
                const Unit w = unit(u);
                const int e = tile_expert[w.mt], p0 = tile_first[w.mt];
                // the expert's rows: gate rows n0.. and up rows N + n0.., or 256 rows from n0 on
                const int w0 = e * (GATED ? 2 : 1) * a.N + w.n0, w1 = w0 + (GATED ? a.N : GG_BN / 2);
                const bool whole = w.cols == OUT_COLS;
                const uint32_t b_bytes = (uint32_t)w.cols * (GATED ? 2 : 1) * GG_BK * 2;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % GG_STAGES;
                    if (!mbar_wait(tc_smem(&empty_bar[s]), ((it / GG_STAGES) & 1u) ^ 1u)) {
                        atomicExch(error_word, 19);
                        abort_flag = 1;
                        ok = false;
                        break;
                    }
                    const uint32_t bar = tc_smem(&full_bar[s]);
                    const uint32_t at = tc_smem(tiles + (size_t)s * GG_STAGE_BYTES);
                    mbar_expect_tx(bar, b_bytes + (GATHER ? 0 : GG_A_BYTES));
                    if (!GATHER) tma_load_2d(at, &map_a, bar, kb * GG_BK, p0);
                    if (whole) {
                        tma_load_2d(at + GG_A_BYTES, &map_b, bar, kb * GG_BK, w0);
                        tma_load_2d(at + GG_A_BYTES + GG_BN / 2 * GG_BK * 2, &map_b, bar, kb * GG_BK, w1);
                        continue;
                    }
                    for (int r = 0; r < w.cols; r += GG_PART_ROWS) {
                        tma_load_2d(at + GG_A_BYTES + r * GG_BK * 2, &map_part, bar, kb * GG_BK, w0 + r);
                        if (GATED)
                            tma_load_2d(at + GG_A_BYTES + (w.cols + r) * GG_BK * 2, &map_part, bar, kb * GG_BK, w1 + r);
                    }
                }
                if (*(volatile int*)&abort_flag) break;
            }
            // no copy outlives the CTA, whatever became of its reader
            for (uint32_t k = it > GG_STAGES ? it - GG_STAGES : 0; k < it; ++k)
                mbar_wait(tc_smem(&full_bar[k % GG_STAGES]), (k / GG_STAGES) & 1u);
        }
    } else if (GATHER && warp >= 6) {
        constexpr int LAG = 2;                          // k-blocks between asking and telling
        const int sub = lane >> 3, chunk = lane & 7;    // row of four, 16-byte piece of the row
        auto tell = [&](uint32_t done) {                // the MMA reads through the asynchronous proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&full_bar[done % GG_STAGES])) : "memory");
        };
        uint32_t it = 0;
        bool ok = true;
        for (int u = 0; u < units && ok; ++u) {
            const int mt = unit(u).mt;
            const int p0 = tile_first[mt], p_last = offsets[tile_expert[mt] + 1] - 1;
            const bf16* src[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                src[i] = x + (size_t)(order[min(p0 + (warp - 6) * 32 + i * 4 + sub, p_last)] / a.top) * a.K + chunk * 8;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it % GG_STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(tc_smem(&empty_bar[s]), ((it / GG_STAGES) & 1u) ^ 1u) &&
                                                 !*(volatile int*)&abort_flag);
                if (!ok) {
                    if (lane == 0 && !*(volatile int*)&abort_flag) {
                        atomicExch(error_word, 19);
                        abort_flag = 1;
                    }
                    break;
                }
                const uint32_t at = tc_smem(tiles + (size_t)s * GG_STAGE_BYTES);
                const bool in = kb * GG_BK + chunk * 8 < a.K;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = (warp - 6) * 32 + i * 4 + sub;
                    cp_async_16(at + r * 128 + ((chunk ^ (r & 7)) << 4), in ? src[i] + kb * GG_BK : x, in ? 16 : 0);
                }
                cp_async_commit();
                if (it >= LAG) {
                    cp_async_wait<LAG>();
                    tell(it - LAG);
                }
            }
        }
        cp_async_wait<0>();
        if (ok)
            for (uint32_t done = it > LAG ? it - LAG : 0; done < it; ++done) tell(done);
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0;
            int j = 0;                                  // tiles done by this CTA
            bool ok = true;
            for (int u = 0; u < units && ok; ++u, ++j) {
                const int b = j & 1;
                const uint32_t idesc = instr_desc_bf16(GG_BM, unit(u).cols * (GATED ? 2 : 1));
                if (!mbar_wait(tc_smem(&acc_empty[b]), (((uint32_t)j >> 1) & 1u) ^ 1u)) {
                    atomicExch(error_word, 20);
                    abort_flag = 1;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t tmem_d = tmem_base + (uint32_t)b * GG_BN;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % GG_STAGES;
                    if (!mbar_wait(tc_smem(&full_bar[s]), (it / GG_STAGES) & 1u)) {
                        atomicExch(error_word, 20);
                        abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_addr = tc_smem(tiles + (size_t)s * GG_STAGE_BYTES);
                    const uint32_t b_addr = a_addr + GG_A_BYTES;
#pragma unroll
                    for (int k4 = 0; k4 < GG_BK / 16; ++k4)
                        tc_mma(tmem_d, smem_desc_sw128(a_addr + k4 * 32), smem_desc_sw128(b_addr + k4 * 32),
                               idesc, (kb | k4) != 0 ? 1u : 0u);
                    tc_commit(tc_smem(&empty_bar[s]));
                }
                if (ok) tc_commit(tc_smem(&acc_full[b]));
            }
            // ... nor a product
            if (it > 0) mbar_wait(tc_smem(&empty_bar[(it - 1) % GG_STAGES]), ((it - 1) / GG_STAGES) & 1u);
        }
    } else {
        const int quarter = warp & 3;                   // the TMEM lanes this warp may touch
        int j = 0;
        for (int k = 0; k < units; ++k, ++j) {
            const int b = j & 1;
            const Unit w = unit(k);
            const int n0 = w.n0, e = tile_expert[w.mt], p = tile_first[w.mt] + quarter * 32 + lane;
            const int p_end = offsets[e + 1];
            const bool valid = p < p_end;
            float wgt = 1.f;
            if (GATHER && a.scale_input && valid) wgt = a.weight[order[p]];
            const bool ready = mbar_wait(tc_smem(&acc_full[b]), ((uint32_t)j >> 1) & 1u);
            // one outcome for the warp: the loads from tensor memory below are warp-wide
            if (!__all_sync(0xffffffffu, ready && !*(volatile int*)&abort_flag)) {
                if (!ready && lane == 0) {
                    atomicExch(error_word, 21);
                    abort_flag = 1;
                }
                break;
            }
            tc_fence_after_sync();
            const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)b * GG_BN;
#pragma unroll 1
            for (int c0 = 0; c0 < w.cols; c0 += 32) {
                uint32_t r[32], u[32];
                tc_ld32(tbase + (uint32_t)c0, r);
                if (GATED) tc_ld32(tbase + (uint32_t)(c0 + w.cols), u);
                tc_wait_ld();
                if (c0 + 32 == w.cols) {              // the accumulator is free, the stores follow
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&acc_empty[b])) : "memory");
                }
                if (MODE == 0) {
                    // through shared memory: eight lanes then store a row's 128 bytes (a lane a row
                    // would touch 32 rows a store: the stores, not the products, set the pace)
                    float* stage = reinterpret_cast<float*>(tiles + (size_t)GG_STAGES * GG_STAGE_BYTES) +
                                   quarter * 32 * GG_STORE_LD;
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<uint4*>(stage + lane * GG_STORE_LD + 4 * i) =
                            make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
                    __syncwarp();
                    const int n = n0 + c0 + (lane & 7) * 4;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = i * 4 + (lane >> 3);
                        const float4 v = *reinterpret_cast<const float4*>(stage + row * GG_STORE_LD + (lane & 7) * 4);
                        if (p - lane + row < p_end && n < a.N)
                            *reinterpret_cast<float4*>((float*)a.out + (size_t)(p - lane + row) * a.N + n) = v;
                    }
                    continue;
                }
                if (!valid) continue;
                // N is a multiple of 8: whole groups of 8 columns are inside or outside
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    const int n = n0 + c0 + c;
                    if (n >= a.N) break;
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float g = __uint_as_float(r[c + i]) * wgt;
                        if (GATED) {
                            const float up = __uint_as_float(u[c + i]) * wgt;
                            v[i] = a.clamped ? clamped_swish_bf16(g, up, a.limit, a.alpha) : silu_bf16(g) * up;
                        } else {
                            const float q = fmaxf(g, 0.f);
                            v[i] = q * q;
                        }
                    }
                    store8((bf16*)a.out + (size_t)p * a.N + n, v);
                }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                     : "memory");
    }
}

// A block a token, eight columns a thread: 16 us for 2,048 x 4 rows of 2,048 floats (67 MB, mostly in L2),
// 36 us a column a thread.  Four rows of y are asked for at once, the sum runs in the
// order of the choices.
template <typename A>
__global__ void __launch_bounds__(256)
experts_combine_kernel(const float* __restrict__ y, const int* __restrict__ pos,
                       const float* __restrict__ weight, const A* __restrict__ add, A* __restrict__ out,
                       int width, int top, int scale_input, const int* __restrict__ chosen,
                       const A* __restrict__ x, int real, const float* add_gate, int gate_stride) {
    const unsigned long long waited = pdl_wait();
    y = pdl_after(y, waited);
    pos = pdl_after(pos, waited);
    add = pdl_after(add, waited);
    add_gate = pdl_after(add_gate, waited);
    const int t = blockIdx.x;
    const float share = add_gate == nullptr ? 1.f : 1.f / (1.f + expf(-add_gate[(size_t)t * gate_stride]));
    for (int c = threadIdx.x * 8; c < width; c += 256 * 8) {
        float total[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < top; k0 += 4) {
            float v[4][8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (k0 + q >= top) continue;
                const size_t r = (size_t)t * top + k0 + q;
                // an identity expert: w x[t]
                if (chosen[r] >= real) load8(x + (size_t)t * width + c, v[q]);
                else load8(y + (size_t)pos[r] * width + c, v[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (k0 + q >= top) continue;
                const size_t r = (size_t)t * top + k0 + q;
                const float w = scale_input && chosen[r] < real ? 1.f : weight[r];
#pragma unroll
                for (int i = 0; i < 8; ++i) total[i] += v[q][i] * w;
            }
        }
        if (add != nullptr) {
            float s[8];
            load8(add + (size_t)t * width + c, s);
#pragma unroll
            for (int i = 0; i < 8; ++i) total[i] += share * s[i];
        }
        store8(out + (size_t)t * width + c, total);
    }
}

// [rows, K] bfloat16 row-major; box = box_rows x 64
static int gg_make_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return -3;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {GG_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -4;
}

template <int MODE>
static int launch_grouped(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mp, const void* x,
                          GroupedArgs a, int max_row_tiles, int* error_word, cudaStream_t s) {
    constexpr size_t smem = (size_t)GG_STAGES * GG_STAGE_BYTES + 1024 +
                            (MODE == 0 ? 4 * 32 * GG_STORE_LD * sizeof(float) : 0);
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(grouped_gemm_kernel<MODE>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int cols = MODE == 1 ? GG_BN / 2 : GG_BN;
    a.n_tiles = (a.N + cols - 1) / cols;
    const long long most = (long long)max_row_tiles * a.n_tiles * 4;      // (a tile may be cut into four)
    const int sms = device_sm_count();
    mstar_launch((grouped_gemm_kernel<MODE>), dim3((unsigned)(most < sms ? most : sms)), dim3(gg_threads(MODE != 0)),
                 smem, s, ma, mb, mp, (const bf16*)x, a, error_word);
    return launch_status();
}

// bfloat16 only.  `ints`: scratch of 2 * rows + experts + 2 + 2 * (rows / 128 + experts) ints;
// `act`: bfloat16 [rows, ff]; `y`: float [rows, width] (rows = tokens * top).  Returns 0, a CUDA
// error code, -1 when the shape is refused (width or ff no multiple of 8, over 1024 experts, an
// operand off 16 bytes), or -3 / -4 when a tensor map cannot be made.  `error_word` receives 19 to 21
// if a bounded wait ran out.
MSTAR_API int mstar_experts_grouped(const void* x, const void* w_gate_up, const void* w_down,
                                    const int* chosen, const float* weight, int* ints, void* act,
                                    float* y, const void* add, void* out, int tokens, int width,
                                    int ff, int top, int experts, int scale_input, int gated,
                                    int real, float limit, float alpha, const float* add_gate,
                                    int gate_stride, int* error_word, void* stream) {
    if (tokens <= 0) return 0;
    if (width % 8 != 0 || ff % 8 != 0 || experts <= 0 || experts > 1024 || top <= 0) return -1;
    if (((uintptr_t)x | (uintptr_t)w_gate_up | (uintptr_t)w_down | (uintptr_t)act | (uintptr_t)y |
         (uintptr_t)add | (uintptr_t)out) & 15)
        return -1;
    cudaStream_t s = (cudaStream_t)stream;
    const int rows = tokens * top;
    const int max_tiles = rows / GG_BM + experts;
    int* order = ints;
    int* pos = order + rows;
    int* offsets = pos + rows;
    int* num_tiles = offsets + experts + 1;
    int* tile_expert = num_tiles + 1;
    int* tile_first = tile_expert + max_tiles;
    CUtensorMap mgu, mact, mdn, mgu_part, mdn_part;
    int rc = gg_make_map(&mgu, w_gate_up, (long long)real * (gated ? 2 : 1) * ff, width, GG_BN / 2);
    if (rc == 0) rc = gg_make_map(&mact, act, rows, ff, GG_BM);
    if (rc == 0) rc = gg_make_map(&mdn, w_down, (long long)real * width, ff, GG_BN / 2);
    if (rc == 0) rc = gg_make_map(&mgu_part, w_gate_up, (long long)real * (gated ? 2 : 1) * ff, width, GG_PART_ROWS);
    if (rc == 0) rc = gg_make_map(&mdn_part, w_down, (long long)real * width, ff, GG_PART_ROWS);
    if (rc != 0) return rc;
    mstar_launch(experts_sort_kernel, dim3(1), dim3(1024), 0, s, chosen, rows, experts, real, order, pos,
                 offsets, tile_expert, tile_first, num_tiles);
    GroupedArgs a{act, order, weight, offsets, tile_expert, tile_first, num_tiles, ff, width, top, 0,
                  scale_input, (int)(gated == 2), limit, alpha};
    rc = gated ? launch_grouped<1>(mgu, mgu, mgu_part, x, a, max_tiles, error_word, s)
               : launch_grouped<2>(mgu, mgu, mgu_part, x, a, max_tiles, error_word, s);
    if (rc != 0) return rc;
    a.out = y;
    a.N = width;
    a.K = ff;
    rc = launch_grouped<0>(mact, mdn, mdn_part, nullptr, a, max_tiles, error_word, s);
    if (rc != 0) return rc;
    mstar_launch((experts_combine_kernel<bf16>), dim3(tokens), dim3(256), 0, s, (const float*)y, pos,
                 weight, (const bf16*)add, (bf16*)out, width, top, scale_input, chosen,
                 (const bf16*)x, real, add_gate, gate_stride);
    return launch_status();
}
