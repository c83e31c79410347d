// Gated delta rule: a matrix memory S [dim][vdim] per head that is decayed row by row,
// corrected towards the token's value along its key, and read with its query.
//
//   prepare  from the float fused projection row [q: G*D | k: G*D | v: H*VD | b: H | ...]:
//            a causal convolution over time on every q, k and v channel (taps weights a
//            channel, the last on the token itself; rows before a portion's start from the
//            request's state slot, which holds the last taps - 1 projected rows) and SiLU;
//            q and k heads to unit length (x / sqrt(sum x^2 + unit_eps)), q times D^-1/2;
//            beta = sigmoid(b);  decay = exp(-exp(A_log_h) * softplus(a + dt_bias)) per head
//            and key channel, a = the low-rank projection's output [H*D].  With one decay a
//            head (`head_decay`) a lies in the row behind b and the decays are [H].
//   scan     per head, token after token:  S = decay * S (rows);  u = beta (v - S^T k);
//            S += k u^T;  o = S^T q.  Computed as  r = (decay*S)^T k,  p = (decay*S)^T q,
//            u = beta (v - r),  o = p + (q . k) u:  the chain from token to token holds one
//            round of shuffles (r); the read-out's round runs beside the next token.
//   finish   o / rms(o per head) * weight * sigmoid(gate) (or silu(gate)), handed on in the
//            activation type.
//
// The scans also move the slot's convolution inputs on (they run after prepare has read them).
//
// A slot is [(taps - 1) * (2 G D + H VD) convolution inputs | S^T as [H][VD][D]], float.
// Everything here is float whatever the activation type.
#include "common.cuh"
#include "mma_util.cuh"
#include "tma_util.cuh"

// ------------------------------------------------------------------ prepare
struct DeltaPrepArgs {
    const float* proj;
    int row_stride;
    const void* conv_w;         // [2 G D + H VD][taps], weight type
    const float* a_proj;        // [tokens][H*D]; null: one decay a head, read from the row
    const float* dt_bias;       // [H*D], or [H]
    const float* a_exp;         // [H]: exp(A_log)
    const int* token_req;
    const int* qo_indptr;
    const int* slots;
    const float* state;
    long long state_stride;
    float* q;                   // [tokens][G*D]
    float* k;                   // [tokens][G*D]
    float* v;                   // [tokens][H*VD]
    float* beta;                // [tokens][H]
    float* decay;               // [tokens][H*D], or [tokens][H]
    int H, G, D, VD, taps;
    float unit_eps;
};

__device__ __forceinline__ float gd_softplus(float z) {
    return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
}

// The convolved and activated value of channel c of token t (the `local`-th of its portion).
template <typename W>
__device__ __forceinline__ float delta_conv_silu(const float* row, const float* slot, const W* cw,
                                                 int c, int channels, int local,
                                                 const DeltaPrepArgs& a) {
    const int keep = a.taps - 1;
    float y = 0.f;
    for (int j = 0; j < a.taps; ++j) {
        const int back = keep - j;                       // rows before this token
        const float u = back <= local ? *(row - (ptrdiff_t)back * a.row_stride + c)
                                      : slot[(size_t)(keep + local - back) * channels + c];
        y = fmaf(to_float(cw[(size_t)c * a.taps + j]), u, y);
    }
    return y / (1.f + expf(-y));
}

// The same for four channels c .. c + 3 at once, by 16-byte accesses.
template <typename W>
__device__ __forceinline__ void delta_conv_silu4(const float* row, const float* slot, const W* cw,
                                                 int c, int channels, int local,
                                                 const DeltaPrepArgs& a, float (&y)[4]) {
    const int keep = a.taps - 1;
    y[0] = y[1] = y[2] = y[3] = 0.f;
    if (a.taps == 4) {
        float w[16], u[4][4];
        if constexpr (sizeof(W) == 2) {
            load8(cw + (size_t)c * 4, reinterpret_cast<float (&)[8]>(w[0]));
            load8(cw + (size_t)c * 4 + 8, reinterpret_cast<float (&)[8]>(w[8]));
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                load4(cw + (size_t)c * 4 + 4 * i, reinterpret_cast<float (&)[4]>(w[4 * i]));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int back = 3 - j;
            load4(back <= local ? row - (ptrdiff_t)back * a.row_stride + c
                                : slot + (size_t)(3 + local - back) * channels + c, u[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = fmaf(w[4 * e + j], u[j][e], y[e]);
    } else {
        for (int j = 0; j < a.taps; ++j) {
            const int back = keep - j;
            float u[4];
            load4(back <= local ? row - (ptrdiff_t)back * a.row_stride + c
                                : slot + (size_t)(keep + local - back) * channels + c, u);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                y[e] = fmaf(to_float(cw[(size_t)(c + e) * a.taps + j]), u[e], y[e]);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = y[e] / (1.f + expf(-y[e]));
}

// A block per token, or, with few tokens, several: a token's work comes in units that a warp
// takes whole (a q head or a k head with its unit norm, the values of a head, the decays of a
// head with its write strength; with one decay a head, those of all heads), dealt out among the
// warps of gridDim.y blocks.  VEC: heads, rows and buffers allow 16-byte accesses.
template <typename W, bool VEC>
__global__ void __launch_bounds__(256) delta_prepare_kernel(DeltaPrepArgs a) {
    extern __shared__ float ch[];             // [warps][D] a q or k head after its convolution
    const int t = blockIdx.x;
    const int qk = a.G * a.D, vv = a.H * a.VD, channels = 2 * qk + vv;
    const W* cw = reinterpret_cast<const W*>(a.conv_w);
    const unsigned long long waited = pdl_wait();
    const float* proj = pdl_after(a.proj, waited);
    const float* a_proj = a.a_proj == nullptr ? nullptr : pdl_after(a.a_proj, waited);
    const float* state = pdl_after(a.state, waited);
    const int e = a.token_req[t];
    const int local = t - a.qo_indptr[e];
    const float* slot = a.taps > 1 ? state + (size_t)a.slots[e] * a.state_stride : nullptr;
    const float* row = proj + (size_t)t * a.row_stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float* mine = ch + (size_t)warp * a.D;
    const float q_scale = rsqrtf((float)a.D);
    const int units = 2 * a.G + a.H + (a_proj != nullptr ? a.H : 1);
    for (int u = blockIdx.y * nwarps + warp; u < units; u += nwarps * gridDim.y) {
        if (u < 2 * a.G) {                                // a q head, then the k heads
            float ss = 0.f;
            if constexpr (VEC) {
                if (a.D <= 128) {                         // a lane keeps its four in registers
                    float y[4] = {0.f, 0.f, 0.f, 0.f};
                    const int d = lane * 4;
                    if (d < a.D) delta_conv_silu4(row, slot, cw, u * a.D + d, channels, local, a, y);
                    ss = warp_sum(fmaf(y[0], y[0], y[1] * y[1]) + fmaf(y[2], y[2], y[3] * y[3]));
                    const float inv = rsqrtf(ss + a.unit_eps) * (u < a.G ? q_scale : 1.f);
                    float* dst = (u < a.G ? a.q : a.k) + (size_t)t * qk + (size_t)(u < a.G ? u : u - a.G) * a.D;
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[e] *= inv;
                    if (d < a.D) store4(dst + d, y);
                    continue;
                }
            }
            for (int d = lane; d < a.D; d += 32) {
                const float y = delta_conv_silu(row, slot, cw, u * a.D + d, channels, local, a);
                mine[d] = y;
                ss = fmaf(y, y, ss);
            }
            ss = warp_sum(ss);
            const bool is_q = u < a.G;
            const float inv = rsqrtf(ss + a.unit_eps) * (is_q ? q_scale : 1.f);
            float* dst = (is_q ? a.q : a.k) + (size_t)t * qk + (size_t)(is_q ? u : u - a.G) * a.D;
            __syncwarp();
            for (int d = lane; d < a.D; d += 32) dst[d] = mine[d] * inv;
            __syncwarp();
        } else if (u < 2 * a.G + a.H) {                   // the values of a head
            const int h = u - 2 * a.G;
            if constexpr (VEC) {
                for (int d = lane * 4; d < a.VD; d += 128) {
                    float y[4];
                    delta_conv_silu4(row, slot, cw, 2 * qk + h * a.VD + d, channels, local, a, y);
                    store4(a.v + (size_t)t * vv + (size_t)h * a.VD + d, y);
                }
            } else {
                for (int d = lane; d < a.VD; d += 32)
                    a.v[(size_t)t * vv + (size_t)h * a.VD + d] =
                        delta_conv_silu(row, slot, cw, 2 * qk + h * a.VD + d, channels, local, a);
            }
        } else if (a_proj == nullptr) {                   // the decays and write strengths of all heads
            for (int h = lane; h < a.H; h += 32) {
                const float step = gd_softplus(row[channels + a.H + h] + a.dt_bias[h]);
                a.decay[(size_t)t * a.H + h] = expf(-a.a_exp[h] * step);
                a.beta[(size_t)t * a.H + h] = 1.f / (1.f + expf(-row[channels + h]));
            }
        } else {                                          // the decays of a head, its write strength
            const int h = u - 2 * a.G - a.H;
            const float rate = a.a_exp[h];
            for (int d = lane; d < a.D; d += 32) {
                const size_t i = (size_t)h * a.D + d;
                const float step = gd_softplus(a_proj[(size_t)t * a.H * a.D + i] + a.dt_bias[i]);
                a.decay[(size_t)t * a.H * a.D + i] = expf(-rate * step);
            }
            if (lane == 0) a.beta[(size_t)t * a.H + h] = 1.f / (1.f + expf(-row[channels + h]));
        }
    }
}

// Prompts, with four taps and heads of 128: a warp takes a unit of DP_RUN tokens in a row, so that a
// projected row is read once instead of four times and the taps' weights once instead of DP_RUN times.  The
// arithmetic of a token is that of the kernel above.  Bound by instructions (the exponentials' and the IEEE
// quotients'): 2,048 tokens, 16 heads of 128 with a decay a key channel: 45 us, 55 above; 3 x 600 with one a head: 18, 21.
#define DP_RUN 8
template <typename W>
__global__ void __launch_bounds__(256) delta_prepare_run_kernel(DeltaPrepArgs a, int tokens) {
    const int qk = a.G * a.D, vv = a.H * a.VD, channels = 2 * qk + vv;
    const W* cw = reinterpret_cast<const W*>(a.conv_w);
    const int lane = threadIdx.x & 31, u = blockIdx.y * 8 + (threadIdx.x >> 5);
    const unsigned long long waited = pdl_wait();
    const float* proj = pdl_after(a.proj, waited);
    const float* a_proj = a.a_proj == nullptr ? nullptr : pdl_after(a.a_proj, waited);
    const float* state = pdl_after(a.state, waited);
    const int t0 = blockIdx.x * DP_RUN, many = min(DP_RUN, tokens - t0);
    if (u < 2 * a.G + a.H) {                              // a q head, then the k heads, then the values of a head
        const bool is_v = u >= 2 * a.G, is_q = u < a.G;
        const int width = is_v ? a.VD : a.D, d = lane * 4;
        const int c = (is_v ? 2 * qk + (u - 2 * a.G) * a.VD : u * a.D) + d;
        const bool in = d < width;
        const float scale = is_q ? rsqrtf((float)a.D) : 1.f;
        float* dst = is_v ? a.v + (size_t)t0 * vv + (c - 2 * qk)
                          : (is_q ? a.q + (size_t)t0 * qk + c : a.k + (size_t)t0 * qk + (c - qk));
        const size_t step = is_v ? vv : qk;
        float w[4][4], row[DP_RUN][4], past[3][4];        // w[channel][tap]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i][0] = w[i][1] = w[i][2] = w[i][3] = 0.f;
            if (in) load4(cw + (size_t)(c + i) * 4, w[i]);
        }
        const float* src = proj + (size_t)t0 * a.row_stride + c;
#pragma unroll
        for (int r = 0; r < DP_RUN; ++r) {
            row[r][0] = row[r][1] = row[r][2] = row[r][3] = 0.f;
            if (in && r < many) load4(src + (size_t)r * a.row_stride, row[r]);
        }
        int entry = -1;
#pragma unroll
        for (int r = 0; r < DP_RUN; ++r) {
            if (r >= many) break;
            const int e = a.token_req[t0 + r];
            if (e != entry) {                             // the inputs before the first token, or before an entry's
                entry = e;
                const int local = t0 + r - a.qo_indptr[e];
                const float* slot = state + (size_t)a.slots[e] * a.state_stride;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int back = 3 - j;
                    past[j][0] = past[j][1] = past[j][2] = past[j][3] = 0.f;
                    if (in)
                        load4(back <= local ? src + (ptrdiff_t)(r - back) * a.row_stride
                                            : slot + (size_t)(3 + local - back) * channels + c, past[j]);
                }
            }
            float y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                y[i] = fmaf(w[i][0], past[0][i], 0.f);
                y[i] = fmaf(w[i][1], past[1][i], y[i]);
                y[i] = fmaf(w[i][2], past[2][i], y[i]);
                y[i] = fmaf(w[i][3], row[r][i], y[i]);
                y[i] = y[i] / (1.f + expf(-y[i]));
                past[0][i] = past[1][i], past[1][i] = past[2][i], past[2][i] = row[r][i];
            }
            if (!is_v) {
                const float ss = warp_sum(fmaf(y[0], y[0], y[1] * y[1]) + fmaf(y[2], y[2], y[3] * y[3]));
                const float inv = rsqrtf(ss + a.unit_eps) * scale;
#pragma unroll
                for (int i = 0; i < 4; ++i) y[i] *= inv;
            }
            if (in) store4(dst + (size_t)r * step, y);
        }
    } else if (a_proj == nullptr) {                       // the decays and write strengths of all heads
        if (u == 2 * a.G + a.H)
            for (int i = lane; i < many * a.H; i += 32) {
                const int t = t0 + i / a.H, h = i % a.H;
                const float* row = proj + (size_t)t * a.row_stride + channels;
                const float step = gd_softplus(row[a.H + h] + a.dt_bias[h]);
                a.decay[(size_t)t * a.H + h] = expf(-a.a_exp[h] * step);
                a.beta[(size_t)t * a.H + h] = 1.f / (1.f + expf(-row[h]));
            }
    } else if (u < 2 * a.G + 2 * a.H) {                   // the decays of a head, its write strength
        const int h = u - 2 * a.G - a.H, d = lane * 4;
        const float rate = a.a_exp[h];
        const size_t at = (size_t)t0 * a.H * a.D + (size_t)h * a.D + d;
        if (d < a.D) {
            float bias[4], z[DP_RUN][4];
            load4(a.dt_bias + h * a.D + d, bias);
#pragma unroll
            for (int r = 0; r < DP_RUN; ++r)
                if (r < many) load4(a_proj + at + (size_t)r * a.H * a.D, z[r]);
#pragma unroll
            for (int r = 0; r < DP_RUN; ++r) {
                if (r >= many) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) z[r][i] = expf(-rate * gd_softplus(z[r][i] + bias[i]));
                store4(a.decay + at + (size_t)r * a.H * a.D, z[r]);
            }
        }
        if (lane < many)
            a.beta[(size_t)(t0 + lane) * a.H + h] = 1.f / (1.f + expf(-proj[(size_t)(t0 + lane) * a.row_stride + channels + h]));
    }
}

MSTAR_API int mstar_delta_prepare(const float* proj, int row_stride, const void* conv_w,
                                  int weight_dtype, const float* a_proj, const float* dt_bias,
                                  const float* a_exp, const int* token_req, const int* qo_indptr,
                                  const int* slots, const float* state, long long state_stride,
                                  float* q, float* k, float* v, float* beta, float* decay,
                                  int tokens, int H, int G, int D, int VD, int taps, float unit_eps,
                                  void* stream) {
    if (tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || VD <= 0 || taps < 1) return -1;
    const int channels = 2 * G * D + H * VD;
    const bool head_decay = a_proj == nullptr;
    if (row_stride < channels + (head_decay ? 2 : 1) * H) return -1;
    if (taps > 1 && (!slots || !state)) return -1;
    const int threads = 256, warps = threads / 32;
    const size_t smem = sizeof(float) * (size_t)warps * D;
    if (smem > 160 * 1024) return -1;
    DeltaPrepArgs a{proj, row_stride, conv_w, a_proj, dt_bias, a_exp, token_req, qo_indptr, slots,
                    state, state_stride, q, k, v, beta, decay, H, G, D, VD, taps, unit_eps};
    cudaStream_t s = (cudaStream_t)stream;
    // with fewer blocks than SMs a token's units go to several blocks
    const int units = 2 * G + H + (head_decay ? 1 : H);
    int parts = 1;
    if (tokens < device_sm_count()) {
        parts = (units + warps - 1) / warps;
        const int room = (2 * device_sm_count() + tokens - 1) / tokens;
        if (parts > room) parts = room;
        if (parts < 1) parts = 1;
    }
    dim3 grid(tokens, parts);
    // 16-byte accesses: whole pieces per head, aligned rows, buffers and state
    bool vec = D % 4 == 0 && VD % 4 == 0 && row_stride % 4 == 0 && state_stride % 4 == 0;
    const void* ptrs[] = {proj, conv_w, state, q, k, v};
    for (const void* p : ptrs) vec = vec && (uintptr_t)p % 16 == 0;
    // Runs of tokens (the same bits) where a head keeps all lanes of a warp busy (heads of 64: 98 us against 68, 32 heads,
    // 2,000 tokens) and there are enough of them, since a run is a chain: with a decay a key channel 7.4 against 11.1 us
    // for 12,800 (200 tokens of 64 units), 43 against 55 for 128,000, but 6.3 against 4.5 for 3,840; with one a head 6.8
    // against 10.4 for 13,000, 11.1 against 12.7 for 30,600, but 6.1 against 5.5 for 8,500 and 52.7 against 48.1 for
    // 130,000.
    const long long all = (long long)tokens * units;
    if (vec && taps == 4 && D == 128 && VD == 128 && (head_decay ? all >= 9000 && all <= 64000 : all >= 12000) &&
        (head_decay || (((uintptr_t)a_proj | (uintptr_t)dt_bias | (uintptr_t)decay) % 16 == 0))) {
        const dim3 runs((tokens + DP_RUN - 1) / DP_RUN, (units + 7) / 8);
        mstar_launch(weight_dtype == MSTAR_F32 ? delta_prepare_run_kernel<float> : delta_prepare_run_kernel<bf16>, runs,
                     dim3(256), 0, s, a, tokens);
        return launch_status();
    }
#define GO1(W, VV)                                                                                \
    do {                                                                                          \
        static size_t configured = 0;                                                             \
        if (smem > 48 * 1024 && smem > configured) {                                              \
            cudaFuncSetAttribute(delta_prepare_kernel<W, VV>,                                     \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
            configured = smem;                                                                    \
        }                                                                                         \
        mstar_launch((delta_prepare_kernel<W, VV>), grid, dim3(threads), smem, s, a);             \
    } while (0)
    if (weight_dtype == MSTAR_F32) {
        if (vec) GO1(float, true); else GO1(float, false);
    } else {
        if (vec) GO1(bf16, true); else GO1(bf16, false);
    }
#undef GO1
    return launch_status();
}

// ------------------------------------------------------------------ scan
#define GD_THREADS 256
#define GD_ROWS 16          // most rows of a column that one lane keeps
#define GD_CHUNK 16         // tokens staged at a time

// The convolutions' rows in a slot move on with the scan: the last taps - 1 rows of the sequence's
// projected channels (a portion shorter than that keeps the newer part of what the slot held).
struct ConvAdvance {
    const float* raw;           // null: not here; else the projected rows of the batch's tokens
    int raw_ld, channels, taps;
};

// Oldest row first: row s is read from s + n, which is written later or not at all.  Only a head's first
// block does this (for its share of the channels), so that the others end without that latency.
__device__ __forceinline__ void gd_advance_conv(const ConvAdvance& c, unsigned long long waited, float* slot,
                                                int start, int n, int h, int H) {
    if (c.raw == nullptr || blockIdx.z != 0) return;
    const float* raw = pdl_after(c.raw, waited);
    const int keep = c.taps - 1, share = (c.channels + H - 1) / H, end = min(c.channels, (h + 1) * share);
    for (int ch = h * share + threadIdx.x; ch < end; ch += blockDim.x)
        for (int s = 0; s < keep; ++s) {
            const int src = n - keep + s;
            slot[(size_t)s * c.channels + ch] = src >= 0 ? raw[(size_t)(start + src) * c.raw_ld + ch]
                                                         : slot[(size_t)(s + n) * c.channels + ch];
        }
}

struct DeltaScanArgs {
    const float* q;
    const float* k;
    const float* v;
    const float* beta;
    const float* decay;
    const int* qo_indptr;
    const int* slots;
    float* state;               // the slot's S^T part starts at state_offset
    long long state_stride;
    long long state_offset;
    float* out;                 // [tokens][H*VD]
    int H, G, D, VD, chunk;
    ConvAdvance conv;
};

__device__ __forceinline__ void gd_copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void gd_copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}

// A block owns GD_THREADS / L value columns of one head of one batch entry; the D rows of a
// column lie on L lanes, lane l keeping rows l, l + L, ...  What the block's columns share of
// a token (its q, k and decay rows, its write strength) and their values are staged in shared
// memory, `chunk` tokens at a time, the next chunk on its way (cp.async) while this one is
// walked.  Along the chain a token costs the decay, four short sums, the shuffles over the L
// lanes and the write; q . k does not depend on the state and runs beside it.
// A warp that waits for its own shuffles has nothing else to issue, so a token's time is the
// length of its instruction chain: the lanes of a column are as many as leave four rows a lane
// (a whole warp a column from 128 rows on), R is the compiled number of rows a lane.
// VEC: rows are whole 16-byte pieces (D a multiple of 4).  HD: one decay a head (`decay` is
// [tokens][H] and travels with the write strength).
template <int L, int R, bool VEC, bool HD>
__global__ void __launch_bounds__(GD_THREADS) delta_scan_kernel(DeltaScanArgs a) {
    extern __shared__ __align__(16) float stage[];     // [2][chunk][NR D + COLS + 4]
    constexpr int COLS = GD_THREADS / L;
    constexpr int NR = HD ? 2 : 3;                     // rows of a token: q, k (, decay)
    const int e = blockIdx.x, h = blockIdx.y;
    const int g = h / (a.H / a.G);
    const int lane = threadIdx.x % L;
    const int mycol = threadIdx.x / L;
    const int col0 = blockIdx.z * COLS;
    const int col = col0 + mycol;
    const bool live = col < a.VD;
    const int D = a.D;
    constexpr int DP = L * R;                          // rows as the lanes see them, zeros past D
    const int per_tok = NR * DP + COLS + 4;            // rows, values, beta, a head's decay (+ padding)
    const unsigned long long waited = pdl_wait();
    const float* q = pdl_after(a.q, waited);
    const float* k = pdl_after(a.k, waited);
    const float* v = pdl_after(a.v, waited);
    const float* beta = pdl_after(a.beta, waited);
    const float* decay = pdl_after(a.decay, waited);
    float* state = pdl_after(a.state, waited);
    const int start = a.qo_indptr[e], n = a.qo_indptr[e + 1] - start;
    if (n <= 0) return;
    const int qk = a.G * D, hd = a.H * D, vv = a.H * a.VD;
    const int ncols = min(COLS, a.VD - col0);

    auto fetch = [&](int buf, int base) {
        const int here = min(a.chunk, n - base);
        float* dst0 = stage + (size_t)buf * a.chunk * per_tok;
        // copy i of the chunk is piece r of token j; both move on by fixed steps from copy to
        // copy, so the loop divides nothing
        const int unit = VEC ? 4 : 1;
        const int per = NR * (D / unit);                // copies a token
        const int dj = GD_THREADS / per, dr = GD_THREADS % per;
        int j = threadIdx.x / per, r = threadIdx.x % per;
        for (; j < here; j += dj, r += dr) {
            if (r >= per) { r -= per; ++j; if (j >= here) break; }
            const int which = r / (D / unit), d = (r - which * (D / unit)) * unit;
            const size_t tok = (size_t)(start + base + j);
            const float* src = which == 0 ? q + tok * qk + (size_t)g * D + d
                             : which == 1 ? k + tok * qk + (size_t)g * D + d
                                          : decay + tok * hd + (size_t)h * D + d;
            float* dst = dst0 + (size_t)j * per_tok + which * DP + d;
            if constexpr (VEC) gd_copy16(dst, src); else gd_copy4(dst, src);
        }
        constexpr int NS = HD ? 2 : 1;                  // numbers of a token: beta (, decay)
        for (int i = threadIdx.x; i < here * (ncols + NS); i += GD_THREADS) {
            const int j = i / (ncols + NS), c = i - j * (ncols + NS);
            const size_t tok = (size_t)(start + base + j);
            float* dst = dst0 + (size_t)j * per_tok + NR * DP;
            if (c < ncols) gd_copy4(dst + c, v + tok * vv + (size_t)h * a.VD + col0 + c);
            else if (c == ncols) gd_copy4(dst + COLS, beta + tok * a.H + h);
            else gd_copy4(dst + COLS + 1, decay + tok * a.H + h);
        }
    };

    // rows past D read as zeros (q, k) whatever the chunk: no copy ever writes there
    if (DP > D) {
        for (int i = threadIdx.x; i < 2 * a.chunk * NR * (DP - D); i += GD_THREADS) {
            const int j = i / (NR * (DP - D)), r = i - j * NR * (DP - D);
            stage[(size_t)j * per_tok + (r / (DP - D)) * DP + D + r % (DP - D)] = 0.f;
        }
    }
    fetch(0, 0);
    cp_async_commit();
    float* s_col = state + (size_t)a.slots[e] * a.state_stride + a.state_offset +
                   ((size_t)h * a.VD + (live ? col : 0)) * D;
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = lane + L * i;
        s[i] = (live && r < D) ? s_col[r] : 0.f;
    }
    int buf = 0;
    float o_prev = 0.f;                        // the last token's read-out, not yet summed
    int prev_tok = -1;
    for (int base = 0; base < n; base += a.chunk, buf ^= 1) {
        if (base + a.chunk < n) fetch(buf ^ 1, base + a.chunk);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const int here = min(a.chunk, n - base);
        const float* tokp = stage + (size_t)buf * a.chunk * per_tok;
        // the rows of the token after this one are read from shared memory while this one's
        // sums go round the lanes
        float qn[R], kn[R], gn[HD ? 1 : R], vn, bn;
        auto next_rows = [&]() {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                qn[i] = tokp[lane + L * i];
                kn[i] = tokp[DP + lane + L * i];
                if constexpr (!HD) gn[i] = tokp[2 * DP + lane + L * i];
            }
            if constexpr (HD) gn[0] = tokp[NR * DP + COLS + 1];
            vn = tokp[NR * DP + mycol];
            bn = tokp[NR * DP + COLS];
        };
        next_rows();
        for (int j = 0; j < here; ++j) {
            float qr[R], kr[R], gr[HD ? 1 : R];
#pragma unroll
            for (int i = 0; i < R; ++i) { qr[i] = qn[i]; kr[i] = kn[i]; }
#pragma unroll
            for (int i = 0; i < (HD ? 1 : R); ++i) gr[i] = gn[i];
            const float vt = vn, bt = bn;
            tokp += per_tok;
            if (j + 1 < here) next_rows();
            float r4[4] = {0.f, 0.f, 0.f, 0.f}, p4[4] = {0.f, 0.f, 0.f, 0.f}, qkdot = 0.f;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                s[i] *= gr[HD ? 0 : i];
                r4[i & 3] = fmaf(kr[i], s[i], r4[i & 3]);
                p4[i & 3] = fmaf(qr[i], s[i], p4[i & 3]);
                qkdot = fmaf(qr[i], kr[i], qkdot);
            }
            // a warp issues in order, so a round of shuffles costs its latency wherever it
            // stands: the read-out of the token before goes round together with this token's r
            float r = (r4[0] + r4[1]) + (r4[2] + r4[3]);
            float o_red = o_prev;
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) {
                r += __shfl_xor_sync(0xffffffffu, r, o);
                o_red += __shfl_xor_sync(0xffffffffu, o_red, o);
            }
            if (prev_tok >= 0 && live && lane == 0)
                a.out[(size_t)prev_tok * vv + (size_t)h * a.VD + col] = o_red;
            const float u = bt * (vt - r);
#pragma unroll
            for (int i = 0; i < R; ++i) s[i] = fmaf(kr[i], u, s[i]);
            o_prev = fmaf(qkdot, u, (p4[0] + p4[1]) + (p4[2] + p4[3]));
            prev_tok = start + base + j;
        }
        __syncthreads();                       // the buffer is free for the chunk after next
    }
    cp_async_wait<0>();
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) o_prev += __shfl_xor_sync(0xffffffffu, o_prev, o);
    if (live && lane == 0) a.out[(size_t)prev_tok * vv + (size_t)h * a.VD + col] = o_prev;
    if (live) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = lane + L * i;
            if (r < D) s_col[r] = s[i];
        }
    }
    gd_advance_conv(a.conv, waited, state + (size_t)a.slots[e] * a.state_stride, start, n, h, a.H);
}

MSTAR_API int mstar_delta_scan(const float* q, const float* k, const float* v, const float* beta,
                               const float* decay, const int* qo_indptr, const int* slots,
                               float* state, long long state_stride, long long state_offset,
                               float* out, int entries, int max_q_len, int H, int G, int D, int VD,
                               int head_decay, const float* conv_raw, int conv_ld, int channels,
                               int taps, void* stream) {
    if (entries <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || VD <= 0 || D > 32 * GD_ROWS) return -1;
    if (H > 65535) return -1;
    // lanes a column: four rows a lane where that fills at most a warp (MSTAR_DELTA_LANES=8
    // or 16: that many from 128 rows on, for measurements)
    int L = 4;
    while (L < 32 && L * 4 < D) L *= 2;
    static int forced = -1;
    if (forced < 0) {
        const char* e = getenv("MSTAR_DELTA_LANES");
        forced = e != nullptr ? atoi(e) : 0;
    }
    if (L == 32 && (forced == 8 || forced == 16) && D <= forced * 16) L = forced;
    const int R = D <= L * 4 ? 4 : (D <= L * 8 ? 8 : 16);
    const int cols = GD_THREADS / L;
    // (the staged rows are padded to L * R)
    // tokens staged at a time: 16, fewer where a token's rows are wide or the entries short
    int chunk = GD_CHUNK;
    const size_t per_tok = (size_t)(head_decay ? 2 : 3) * L * R + cols + 4;
    while (chunk > 1 && (chunk / 2 >= max_q_len || 2 * chunk * per_tok * sizeof(float) > 64 * 1024))
        chunk /= 2;
    const size_t smem = 2 * chunk * per_tok * sizeof(float);
    DeltaScanArgs a{q, k, v, beta, decay, qo_indptr, slots, state, state_stride, state_offset, out,
                    H, G, D, VD, chunk, {taps > 1 ? conv_raw : nullptr, conv_ld, channels, taps}};
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(entries, H, (VD + cols - 1) / cols);
    if (grid.z > 65535) return -1;
    // 16-byte copies want whole pieces and aligned rows (the buffers are allocations of their own)
    const bool vec = D % 4 == 0 && (state_offset % 4) == 0 &&
                     ((uintptr_t)q % 16 == 0) && ((uintptr_t)k % 16 == 0) &&
                     (head_decay || (uintptr_t)decay % 16 == 0);
#define GO1(LL, RR, VV, HH)                                                                           \
    do {                                                                                          \
        static size_t configured = 0;                                                             \
        if (smem > 48 * 1024 && smem > configured) {                                              \
            cudaFuncSetAttribute(delta_scan_kernel<LL, RR, VV, HH>,                               \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
            configured = smem;                                                                    \
        }                                                                                         \
        mstar_launch((delta_scan_kernel<LL, RR, VV, HH>), grid, dim3(GD_THREADS), smem, s, a);    \
    } while (0)
#define GO2(LL, RR, VV)                                                                           \
    do {                                                                                          \
        if (head_decay) GO1(LL, RR, VV, true); else GO1(LL, RR, VV, false);                       \
    } while (0)
#define GO(LL, RR)                                                                                \
    do {                                                                                          \
        if (vec) GO2(LL, RR, true); else GO2(LL, RR, false);                                      \
    } while (0)
    if (L == 4) GO(4, 4);
    else if (L == 8 && R == 4) GO(8, 4);
    else if (L == 8 && R == 8) GO(8, 8);
    else if (L == 8) GO(8, 16);
    else if (L == 16 && R == 4) GO(16, 4);
    else if (L == 16 && R == 8) GO(16, 8);
    else if (L == 16) GO(16, 16);
    else if (R == 4) GO(32, 4);
    else if (R == 8) GO(32, 8);
    else GO(32, 16);
#undef GO
#undef GO2
#undef GO1
    return launch_status();
}

// ------------------------------------------------------------------ scans in pieces of 16 tokens
// With one decay g_t a head the decayed rows are the rows times a number, and everything inside a
// piece of C tokens that does not depend on the state is a C x C matrix.  With P_t = g_1 .. g_t
// (from the piece's first token), dec(t, j) = g_{j+1} .. g_t, the state S0 at the piece's start and
//   L_tj = beta_t (k_t . k_j) dec(t, j)  (j < t),    B_tj = (q_t . k_j) dec(t, j)  (j <= t),
// the delta rule of the piece is the triangular system (I + L) u = beta c, c_t = v_t - P_t k_t . S0:
//   T = (I + L)^-1 diag(beta),   u = T c,   o_t = P_t q_t . S0 + (B T c)_t,
//   S_C = P_C S0 + sum_j dec(C, j) k_j u_j.
// A first kernel makes T, B T, P and dec(C, .) for all pieces and heads side by side (products of
// decays only, never a quotient; the products of keys and queries among themselves are shared by
// the heads of a group) and lays them, and the piece's k and q rows, down as the scan wants them in
// its shared memory, so that a piece is two bulk copies.  The scan has no chain from token to token
// inside a piece.  All float.
//
// With a decay per key channel, P_t, dec(t, j) and P_C are vectors over the key channels: the products
// k_t . k_j become sums of k_t k_j dec(t, j), and the piece's rows are decayed rows, P_t k_t, P_t q_t,
// dec(C, t) k_t and P_C (CHANNEL below; a first kernel of its own makes them, a block a head); the rest
// is the same, with P and dec of the matrices' rows at 1.
#define GC_TOKENS 16
#define GH_THREADS 128
#define GH_WAIT_CODE 18             // what the error word gets when a wait for a piece ran out
#define GH_LD (GC_TOKENS + 4)       // floats between the rows of a C x C matrix in shared memory
#define GH_MROW (2 * GC_TOKENS + 4) // a token's row of T, of B T, then P_t and dec(C, t)

struct DeltaHeadArgs {
    const float* q;
    const float* k;
    const float* v;
    const float* beta;
    const float* decay;         // [tokens][H], CHANNEL: [tokens][H][D]
    const int* qo_indptr;
    const int* slots;
    // [pieces][G][2 C][D + 4]: the k rows, then the q rows; zeros past the end.  CHANNEL: [pieces][H][
    // 3 C + 1][D + 4]: P_t k_t, P_t q_t, dec(C, t) k_t and P_C
    float* rows;
    float* mats;                // [pieces][H][C][GH_MROW]
    float* state;
    long long state_stride;
    long long state_offset;
    float* out;
    int H, G, D, VD, tokens;
    int* error_word;
    ConvAdvance conv;
};

// Pieces are numbered over the batch so that an entry's are consecutive: at most tokens / C + entries.
__device__ __forceinline__ size_t gh_first_piece(int start, int e) { return (size_t)(start / GC_TOKENS + e); }

// Column j of T and of B T by forward substitution with L and B in shared memory (rows of GH_LD floats);
// bj: the write strength of token j, m: the piece's matrices.
__device__ __forceinline__ void gh_solve(const float* L, const float* B, int j, float bj, float* m) {
    constexpr int C = GC_TOKENS;
    float col[C];                                 // column j of (I + L)^-1, zero above j
#pragma unroll
    for (int t = 0; t < C; ++t) {
        float s = t == j ? 1.f : 0.f;
#pragma unroll
        for (int x = 0; x < t; x += 4) {
            float l[4];
            load4(L + t * GH_LD + x, l);
#pragma unroll
            for (int w = 0; w < 4; ++w)
                if (x + w < t) s = fmaf(-l[w], col[x + w], s);
        }
        col[t] = s;
    }
#pragma unroll
    for (int t = 0; t < C; ++t) {
        float s = 0.f;
#pragma unroll
        for (int x = 0; x <= t; x += 4) {
            float bt[4];
            load4(B + t * GH_LD + x, bt);
#pragma unroll
            for (int w = 0; w < 4; ++w)
                if (x + w <= t) s = fmaf(bt[w], col[x + w], s);
        }
        m[t * GH_MROW + j] = col[t] * bj;
        m[t * GH_MROW + C + j] = s * bj;
    }
}

// A block per (piece, entry, group of heads); thread (t, j) of 256 makes k_t . k_j and q_t . k_j,
// then a warp a head: lane j the column j of T and of B T by forward substitution.
__global__ void __launch_bounds__(256) delta_head_pieces_kernel(DeltaHeadArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int C = GC_TOKENS;
    const int D = a.D, LD = D + 4;
    float* ks = sm;                              // [C][LD]
    float* qs = ks + C * LD;                     // [C][LD]
    float* kk = qs + C * LD;                     // [C][GH_LD] k_t . k_j
    float* qk = kk + C * GH_LD;                  // [C][GH_LD] q_t . k_j
    float* per_warp = qk + C * GH_LD;            // [min(8, heads of the group)]{L, B [C][GH_LD], g, beta [C]}
    const int piece = blockIdx.x, e = blockIdx.y, grp = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long waited = pdl_wait();
    const float* q = pdl_after(a.q, waited);
    const float* k = pdl_after(a.k, waited);
    const float* beta = pdl_after(a.beta, waited);
    const float* decay = pdl_after(a.decay, waited);
    const int start = a.qo_indptr[e], n = a.qo_indptr[e + 1] - start;
    const int base = piece * C;
    if (base >= n) return;
    const int here = min(C, n - base);
    const int qkw = a.G * D;
    for (int i = tid; i < C * (D / 4); i += 256) {
        const int t = i / (D / 4), d = (i - t * (D / 4)) * 4;
        float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), qv = kv;
        if (t < here) {
            const size_t o = (size_t)(start + base + t) * qkw + (size_t)grp * D + d;
            kv = *reinterpret_cast<const float4*>(k + o);
            qv = *reinterpret_cast<const float4*>(q + o);
        }
        *reinterpret_cast<float4*>(ks + t * LD + d) = kv;
        *reinterpret_cast<float4*>(qs + t * LD + d) = qv;
        float* dst = a.rows + (((gh_first_piece(start, e) + piece) * a.G + grp) * 2 * C + t) * LD + d;
        *reinterpret_cast<float4*>(dst) = kv;
        *reinterpret_cast<float4*>(dst + C * LD) = qv;
    }
    __syncthreads();
    {
        const int t = tid >> 4, j = tid & 15;
        float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
        for (int d = 0; d < D; d += 4) {
            const float4 kt = *reinterpret_cast<const float4*>(ks + t * LD + d);
            const float4 qt = *reinterpret_cast<const float4*>(qs + t * LD + d);
            const float4 kj = *reinterpret_cast<const float4*>(ks + j * LD + d);
            a0 = fmaf(kt.x, kj.x, a0); a1 = fmaf(kt.y, kj.y, a1);
            b0 = fmaf(qt.x, kj.x, b0); b1 = fmaf(qt.y, kj.y, b1);
            a0 = fmaf(kt.z, kj.z, a0); a1 = fmaf(kt.w, kj.w, a1);
            b0 = fmaf(qt.z, kj.z, b0); b1 = fmaf(qt.w, kj.w, b1);
        }
        kk[t * GH_LD + j] = a0 + a1;
        qk[t * GH_LD + j] = b0 + b1;
    }
    __syncthreads();
    const int per = a.H / a.G;
    float* L = per_warp + (size_t)warp * (2 * C * GH_LD + 2 * C);
    float* B = L + C * GH_LD;
    float* gs = B + C * GH_LD;
    float* bs = gs + C;
    for (int i = warp; i < per && warp < 8; i += 8) {
        const int h = grp * per + i;
        if (lane < C) {
            const size_t o = (size_t)(start + base + lane) * a.H + h;
            gs[lane] = lane < here ? decay[o] : 1.f;
            bs[lane] = lane < here ? beta[o] : 0.f;
        }
        __syncwarp();
        // lane (j, half): column j of L and B, dec(t, j) growing as t walks on; the lower half
        // of the lanes writes L, the upper B
        const int j = lane & 15;
        float dec = 1.f;
        for (int t = j; t < C; ++t) {
            if (t > j) dec *= gs[t];
            if (lane < C) { if (t > j) L[t * GH_LD + j] = bs[t] * kk[t * GH_LD + j] * dec; }
            else B[t * GH_LD + j] = qk[t * GH_LD + j] * dec;
        }
        float P = 1.f;
        for (int t = 0; t <= j; ++t) P *= gs[t];
        __syncwarp();
        if (lane < C) {
            float* m = a.mats + ((gh_first_piece(start, e) + piece) * a.H + h) * C * GH_MROW;
            m[j * GH_MROW + 2 * C] = P;
            m[j * GH_MROW + 2 * C + 1] = dec;            // dec(C, j): a short piece's g are 1 past its end
            gh_solve(L, B, j, bs[j], m);
        }
        __syncwarp();
    }
}

// The pieces of a decay per key channel: a block per (piece, entry, head).
//
// The piece's sums A_tj = sum_d k_t k_j dec(t, j) (and B_tj with q_t) take products of decays only, so
// dec(t, j) cannot be cut into a factor of t and one of j by a quotient.  It is cut at the start m of
// token t's four: for j before m it is (g_m .. g_t) (g_{j+1} .. g_{m-1}), which makes the sum a plain product
// of rows X_t = k_t g_m .. g_t and Y_j = k_j g_{j+1} .. g_{m-1} (24 rows for the three later fours), and within a
// four the six rows W_tj = k_j g_{j+1} .. g_t are made as they are.  A thread a pair (t, j <= t) then takes its
// two products by 16-byte loads; the rows are made a thread a channel.  Bound by shared loads and by how few
// blocks an SM holds: 46 us for 2,048 tokens and 16 heads of 128 (56 with two blocks an SM and a thread
// for the other pairs too; 78 for a warp a token j that walked on over t with two warp sums each).
#define GK_ROWS(C) (3 * (C) + 1)            // decayed keys, decayed queries, keys on their way to the end, P_C
__global__ void __launch_bounds__(256, 3) delta_channel_pieces_kernel(DeltaHeadArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int C = GC_TOKENS;
    const int D = a.D, LD = D + 4;
    float* ks = sm;                              // [C][LD]
    float* qs = ks + C * LD;                     // [C][LD]
    float* gs = qs + C * LD;                     // [C][LD]
    float* Xk = gs + C * LD;                     // [C][LD]
    float* Xq = Xk + C * LD;                     // [C][LD]
    float* Y = Xq + C * LD;                      // [24][LD]: of fours 1, 2, 3 (4, 8, 12 rows)
    float* W = Y + 24 * LD;                      // [24][LD]: six of each four, (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
    float* L = W + 24 * LD;                      // [C][GH_LD]
    float* B = L + C * GH_LD;                    // [C][GH_LD]
    const int piece = blockIdx.x, e = blockIdx.y, h = blockIdx.z, g_head = h / (a.H / a.G);
    const int tid = threadIdx.x;
    const unsigned long long waited = pdl_wait();
    const float* q = pdl_after(a.q, waited);
    const float* k = pdl_after(a.k, waited);
    const float* beta = pdl_after(a.beta, waited);
    const float* decay = pdl_after(a.decay, waited);
    const int start = a.qo_indptr[e], n = a.qo_indptr[e + 1] - start;
    const int base = piece * C;
    if (base >= n) return;
    const int here = min(C, n - base);
    for (int i = tid; i < C * (D / 4); i += 256) {
        const int t = i / (D / 4), d = (i - t * (D / 4)) * 4;
        float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), qv = kv, gv = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < here) {
            const size_t tok = (size_t)(start + base + t);
            kv = *reinterpret_cast<const float4*>(k + tok * a.G * D + (size_t)g_head * D + d);
            qv = *reinterpret_cast<const float4*>(q + tok * a.G * D + (size_t)g_head * D + d);
            gv = *reinterpret_cast<const float4*>(decay + tok * a.H * D + (size_t)h * D + d);
        }
        *reinterpret_cast<float4*>(ks + t * LD + d) = kv;
        *reinterpret_cast<float4*>(qs + t * LD + d) = qv;
        *reinterpret_cast<float4*>(gs + t * LD + d) = gv;
    }
    __syncthreads();
    const size_t at = (gh_first_piece(start, e) + piece) * a.H + h;
    // a thread a channel: half of the threads the rows for the scan, half those for the sums here
    for (int i = tid; i < 2 * D; i += 256) {
        const int d = i % D;
        float kd[C], gd[C];
#pragma unroll
        for (int t = 0; t < C; ++t) {
            kd[t] = ks[t * LD + d];
            gd[t] = gs[t * LD + d];
        }
        if (i < D) {
            float* dst = a.rows + at * GK_ROWS(C) * LD + d;
            float P = 1.f, S = 1.f;
#pragma unroll
            for (int t = 0; t < C; ++t) {
                P *= gd[t];
                dst[t * LD] = kd[t] * P;
                dst[(C + t) * LD] = qs[t * LD + d] * P;
            }
            dst[3 * C * LD] = P;
#pragma unroll
            for (int t = C - 1; t >= 0; --t) {
                dst[(2 * C + t) * LD] = kd[t] * S;
                S *= gd[t];
            }
        } else {
            float y[C - 4];                      // Y of the four that comes next
#pragma unroll
            for (int f = 0; f < C / 4; ++f) {
                float P = 1.f;
#pragma unroll
                for (int t = 4 * f; t < 4 * f + 4; ++t) {
                    P *= gd[t];
                    Xk[t * LD + d] = kd[t] * P;
                    Xq[t * LD + d] = qs[t * LD + d] * P;
#pragma unroll
                    for (int j = 4 * f; j < t; ++j) {
                        float w = kd[j];
#pragma unroll
                        for (int x = j + 1; x <= t; ++x) w *= gd[x];
                        const int tt = t - 4 * f, jj = j - 4 * f;
                        W[(6 * f + tt * (tt - 1) / 2 + jj) * LD + d] = w;
                    }
                }
                if (f == C / 4 - 1) break;
#pragma unroll
                for (int j = 0; j < 4 * f; ++j) y[j] *= P;
                float S = 1.f;
#pragma unroll
                for (int j = 4 * f + 3; j >= 4 * f; --j) {
                    y[j] = kd[j] * S;
                    S *= gd[j];
                }
#pragma unroll
                for (int j = 0; j < 4 * f + 4; ++j) Y[(2 * f * (f + 1) + j) * LD + d] = y[j];
            }
        }
    }
    __syncthreads();
    if (tid < C * (C + 1) / 2) {
        // pair tid of (0, 0), (1, 0), (1, 1), (2, 0), ..: the largest t with t (t + 1) / 2 <= tid
        int t = 0;
#pragma unroll
        for (int x = 1; x < C; ++x) t += tid >= x * (x + 1) / 2;
        const int j = tid - t * (t + 1) / 2, f = t >> 2;
        const bool near = (j >> 2) == f;         // in token t's own four
        const float* right = j == t ? ks + t * LD
                             : near ? W + (6 * f + (t & 3) * ((t & 3) - 1) / 2 + (j & 3)) * LD
                                    : Y + (2 * (f - 1) * f + j) * LD;
        const float* left_k = (near ? ks : Xk) + t * LD;
        const float* left_q = (near ? qs : Xq) + t * LD;
        float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
        for (int d = 0; d < D; d += 4) {
            const float4 kt = *reinterpret_cast<const float4*>(left_k + d);
            const float4 qt = *reinterpret_cast<const float4*>(left_q + d);
            const float4 kj = *reinterpret_cast<const float4*>(right + d);
            a0 = fmaf(kt.x, kj.x, a0); a1 = fmaf(kt.y, kj.y, a1);
            b0 = fmaf(qt.x, kj.x, b0); b1 = fmaf(qt.y, kj.y, b1);
            a0 = fmaf(kt.z, kj.z, a0); a1 = fmaf(kt.w, kj.w, a1);
            b0 = fmaf(qt.z, kj.z, b0); b1 = fmaf(qt.w, kj.w, b1);
        }
        const float bt = t < here ? beta[(size_t)(start + base + t) * a.H + h] : 0.f;
        if (j < t) L[t * GH_LD + j] = bt * (a0 + a1);
        B[t * GH_LD + j] = b0 + b1;
    }
    __syncthreads();
    if (tid < C) {
        float* m = a.mats + at * C * GH_MROW;
        m[tid * GH_MROW + 2 * C] = 1.f;          // (the rows carry P and dec)
        m[tid * GH_MROW + 2 * C + 1] = 1.f;
        gh_solve(L, B, tid, tid < here ? beta[(size_t)(start + base + tid) * a.H + h] : 0.f, m);
    }
}

// A block owns COLS (8 or 16) value columns of one head of one entry.  Per piece, all as small matrix
// products in registers: [r; p] = [k; q] S0 (32 rows x COLS columns, each warp over a quarter of D, a
// thread 4 rows x COLS / 4 columns), the warps' shares met in shared memory; c, then u = T c and o by
// thread (t, COLS / 8 columns); S = P_C S0 + (dec k)^T u by a thread that keeps its part of S in registers and
// leaves a copy, a column a row, in shared memory for the next piece's products.
__device__ __forceinline__ void gh_load(const float* p, float (&v)[1]) { v[0] = p[0]; }
__device__ __forceinline__ void gh_load(const float* p, float (&v)[2]) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    v[0] = a.x; v[1] = a.y;
}
__device__ __forceinline__ void gh_load(const float* p, float (&v)[4]) { load4(p, v); }
__device__ __forceinline__ void gh_store(float* p, const float (&v)[1]) { p[0] = v[0]; }
__device__ __forceinline__ void gh_store(float* p, const float (&v)[2]) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
__device__ __forceinline__ void gh_bulk(float* dst, const float* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc_smem(dst)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

//
// CHANNEL: the rows hold the decays (P and dec are 1 in the matrices), the new state takes rows of its own,
// and P_C is a row.  2,048 tokens, 16 heads of 128 x 128: 173 us (a scan that gave a warp a column and a lane a
// token's dot products, every warp reading all of the piece's rows, took 430 us: shared loads, which bound
// this one too: with eight warps and half the columns of S a thread, 195 us).
template <int D, int COLS, bool CHANNEL>
__global__ void __launch_bounds__(GH_THREADS, 2) delta_head_scan_kernel(DeltaHeadArgs a) {
    extern __shared__ __align__(16) float sm[];
    constexpr int C = GC_TOKENS, LD = D + 4, WARPS = GH_THREADS / 32;
    constexpr int ROWS = CHANNEL ? GK_ROWS(C) : 2 * C;
    constexpr int per_buf = ROWS * LD + C * GH_MROW;
    constexpr int PJ = COLS / 4;                             // columns a thread takes of [r; p]
    constexpr int CT = D >= 96 ? PJ : (D == 64 || PJ < 4 ? PJ / 2 : 1);      // and keeps of S
    constexpr int TN = COLS / 8;                             // and makes of u and o
    constexpr int DT = D > 128 ? D / 128 : 1;                // groups of 4 rows it keeps
    constexpr int DG = D / 4 / DT;                           // row groups that lie on threads
    constexpr int PLD = COLS + 4;
    float* cols = sm + 2 * per_buf;              // [COLS][LD] S0, a column a row
    float* part = cols + COLS * LD;              // [WARPS][2 C][PLD] shares of r and p
    float* cs = part + WARPS * 2 * C * PLD;      // [C][COLS]
    float* us = cs + C * COLS;                   // [C][COLS] dec(C, t) u_t
    __shared__ __align__(8) unsigned long long full[2];
    const int e = blockIdx.x, h = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = blockIdx.z * COLS;
    const unsigned long long waited = pdl_wait();
    const float* v = pdl_after(a.v, waited);
    const float* rows = pdl_after((const float*)a.rows, waited);
    const float* mats = pdl_after((const float*)a.mats, waited);
    float* state = pdl_after(a.state, waited);
    const int start = a.qo_indptr[e], n = a.qo_indptr[e + 1] - start;
    if (n <= 0) return;
    const int vv = a.H * a.VD, grp = h / (a.H / a.G);
    const size_t first = gh_first_piece(start, e);

    auto fetch = [&](int buf, int piece) {       // one thread; both copies complete on the buffer's barrier
        const uint32_t bar = tc_smem(full + buf);
        float* dst = sm + buf * per_buf;
        mbar_expect_tx(bar, (uint32_t)(per_buf * sizeof(float)));
        gh_bulk(dst, rows + (CHANNEL ? (first + piece) * a.H + h : (first + piece) * a.G + grp) * ROWS * LD,
                ROWS * LD * sizeof(float), bar);
        gh_bulk(dst + ROWS * LD, mats + ((first + piece) * a.H + h) * C * GH_MROW, C * GH_MROW * sizeof(float), bar);
    };

    const int pieces = (n + C - 1) / C;
    if (tid == 0) {
        mbar_init(tc_smem(full), 1);
        mbar_init(tc_smem(full + 1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fetch(0, 0);
    }
    __syncthreads();
    // the thread's part of S: rows 4 (dg + DG x) .. + 3, columns CT cg .. (lanes: 8 row groups x 4
    // column groups)
    const int cg = (tid / 8) % (COLS / CT), dg = tid % 8 + (tid / 8 / (COLS / CT)) * 8;
    const bool keeps = dg < DG;
    float* s_head = state + (size_t)a.slots[e] * a.state_stride + a.state_offset +
                    ((size_t)h * a.VD + col0) * D;
    float s[DT][CT][4];
#pragma unroll
    for (int x = 0; x < DT; ++x)
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            s[x][c][0] = s[x][c][1] = s[x][c][2] = s[x][c][3] = 0.f;
            if (keeps) {
                const int col = cg * CT + c, d = (dg + DG * x) * 4;
                if (col0 + col < a.VD) load4(s_head + (size_t)col * D + d, s[x][c]);
                store4(cols + col * LD + d, s[x][c]);
            }
        }
    // thread (token t, columns tc .. tc + TN - 1) between the products
    const int t = tid / 8, tc = tid % 8 * TN;
    float v_next[TN];
#pragma unroll
    for (int x = 0; x < TN; ++x) v_next[x] = 0.f;
    auto ahead = [&](int piece) {                // the values the thread itself needs of a piece
        const int at = piece * C + t;
        if (at < n) {
            const float* src = v + (size_t)(start + at) * vv + (size_t)h * a.VD + col0 + tc;
#pragma unroll
            for (int x = 0; x < TN; ++x)
                if (col0 + tc + x < a.VD) v_next[x] = src[x];
        }
    };
    ahead(0);
    const int tg = lane & 7, pg = lane >> 3;     // rows tg + 8 i of [k; q], columns pg + 4 j
    for (int piece = 0; piece < pieces; ++piece) {
        const int buf = piece & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(tc_smem(full + buf), (piece >> 1) & 1))) {
            if (lane == 0) atomicExch(a.error_word, GH_WAIT_CODE);
            mbar_wait(tc_smem(full + buf), (piece >> 1) & 1);    // no copy in flight outlives the block
            return;
        }
        __syncthreads();                         // the piece and S0 are here, the other buffer is free
        float vt[TN];
#pragma unroll
        for (int x = 0; x < TN; ++x) vt[x] = v_next[x];
        if (piece + 1 < pieces) {
            if (tid == 0) fetch(buf ^ 1, piece + 1);
            ahead(piece + 1);
        }
        const int here = min(C, n - piece * C);
        const float* ks = sm + buf * per_buf;    // (the q rows follow the k rows)
        const float* ms = ks + ROWS * LD;
        const float P = ms[t * GH_MROW + 2 * C], dec = ms[t * GH_MROW + 2 * C + 1];
        {
            float acc[4][PJ];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < PJ; ++j) acc[i][j] = 0.f;
            const float* rowp = ks + tg * LD + warp * (D / WARPS);
            const float* colp = cols + pg * LD + warp * (D / WARPS);
#pragma unroll
            for (int d = 0; d < D / WARPS; d += 4) {
                float rv[4][4], cv[PJ][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) load4(rowp + 8 * i * LD + d, rv[i]);
#pragma unroll
                for (int j = 0; j < PJ; ++j) load4(colp + 4 * j * LD + d, cv[j]);
#pragma unroll
                for (int w = 0; w < 4; ++w)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < PJ; ++j) acc[i][j] = fmaf(rv[i][w], cv[j][w], acc[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < PJ; ++j)
                    part[(warp * 2 * C + tg + 8 * i) * PLD + pg + 4 * j] = acc[i][j];
        }
        __syncthreads();
        float r[TN], p[TN];
#pragma unroll
        for (int x = 0; x < TN; ++x) r[x] = p[x] = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            float rs[TN], ps[TN];
            gh_load(part + (w * 2 * C + t) * PLD + tc, rs);
            gh_load(part + (w * 2 * C + C + t) * PLD + tc, ps);
#pragma unroll
            for (int x = 0; x < TN; ++x) {
                r[x] += rs[x];
                p[x] += ps[x];
            }
        }
        // (a token past the piece has c = 0: its row and column of T and B T are not used)
        float ct[TN];
#pragma unroll
        for (int x = 0; x < TN; ++x) ct[x] = t < here ? fmaf(-P, r[x], vt[x]) : 0.f;
        gh_store(cs + t * COLS + tc, ct);
        __syncthreads();
        {
            float u[TN], o[TN];
#pragma unroll
            for (int x = 0; x < TN; ++x) {
                u[x] = 0.f;
                o[x] = P * p[x];
            }
            const float* trow = ms + t * GH_MROW;
            const float* brow = trow + C;
#pragma unroll
            for (int i = 0; i < C; i += 4) {
                // up to t only, not with the zeros behind: a later token's value that is not finite stays out
                // (0 times it would be no 0; skipping the later fours took 3 % more time than these selects)
                float t4[4], b4[4];
                load4(trow + i, t4);
                load4(brow + i, b4);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    float c[TN];
                    gh_load(cs + (i + w) * COLS + tc, c);
                    const bool seen = i + w <= t;
                    if (!seen) t4[w] = b4[w] = 0.f;
#pragma unroll
                    for (int x = 0; x < TN; ++x) {
                        if (!seen) c[x] = 0.f;
                        u[x] = fmaf(t4[w], c[x], u[x]);
                        o[x] = fmaf(b4[w], c[x], o[x]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < TN; ++x) u[x] = t < here ? dec * u[x] : 0.f;
            gh_store(us + t * COLS + tc, u);
            if (t < here) {
                float* dst = a.out + (size_t)(start + piece * C + t) * vv + (size_t)h * a.VD + col0 + tc;
#pragma unroll
                for (int x = 0; x < TN; ++x)
                    if (col0 + tc + x < a.VD) dst[x] = o[x];
            }
        }
        __syncthreads();
        if (keeps) {
            const float* news = CHANNEL ? ks + 2 * C * LD : ks;  // the rows that enter the state
#pragma unroll
            for (int x = 0; x < DT; ++x) {
                float pc[4];
                if (CHANNEL) {
                    load4(ks + 3 * C * LD + (dg + DG * x) * 4, pc);
                } else {
                    pc[0] = pc[1] = pc[2] = pc[3] = ms[(here - 1) * GH_MROW + 2 * C];
                }
#pragma unroll
                for (int c = 0; c < CT; ++c)
#pragma unroll
                    for (int w = 0; w < 4; ++w) s[x][c][w] *= pc[w];
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                float u[CT];
                gh_load(us + j * COLS + cg * CT, u);
#pragma unroll
                for (int x = 0; x < DT; ++x) {
                    float kv[4];
                    load4(news + j * LD + (dg + DG * x) * 4, kv);
#pragma unroll
                    for (int c = 0; c < CT; ++c)
#pragma unroll
                        for (int w = 0; w < 4; ++w) s[x][c][w] = fmaf(kv[w], u[c], s[x][c][w]);
                }
            }
#pragma unroll
            for (int x = 0; x < DT; ++x)
#pragma unroll
                for (int c = 0; c < CT; ++c) store4(cols + (cg * CT + c) * LD + (dg + DG * x) * 4, s[x][c]);
        }
    }
    if (keeps) {
#pragma unroll
        for (int x = 0; x < DT; ++x)
#pragma unroll
            for (int c = 0; c < CT; ++c)
                if (col0 + cg * CT + c < a.VD)
                    store4(s_head + (size_t)(cg * CT + c) * D + (dg + DG * x) * 4, s[x][c]);
    }
    gd_advance_conv(a.conv, waited, state + (size_t)a.slots[e] * a.state_stride, start, n, h, a.H);
}

template <int D, int COLS, bool CHANNEL>
static int launch_head_scan(const DeltaHeadArgs& a, int entries, cudaStream_t s) {
    constexpr int rows = CHANNEL ? GK_ROWS(GC_TOKENS) : 2 * GC_TOKENS;
    constexpr size_t smem = ((size_t)2 * (rows * (D + 4) + GC_TOKENS * GH_MROW) + COLS * (D + 4) +
                             (GH_THREADS / 32) * 2 * GC_TOKENS * (COLS + 4) + 2 * GC_TOKENS * COLS) * sizeof(float);
    static bool configured = false;
    if (smem > 48 * 1024 && !configured) {
        const cudaError_t e = cudaFuncSetAttribute(delta_head_scan_kernel<D, COLS, CHANNEL>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const dim3 grid(entries, a.H, (a.VD + COLS - 1) / COLS);
    if (grid.z > 65535) return -1;
    mstar_launch((delta_head_scan_kernel<D, COLS, CHANNEL>), grid, dim3(GH_THREADS), smem, s, a);
    return launch_status();
}
template <int D, bool CHANNEL>
static int launch_head_scan_cols(const DeltaHeadArgs& a, int entries, cudaStream_t s) {
    // 16 columns a block where that gives most SMs a block, else 8
    return (long long)entries * a.H * ((a.VD + 15) / 16) * 4 >= 3LL * device_sm_count()
               ? launch_head_scan<D, 16, CHANNEL>(a, entries, s)
               : launch_head_scan<D, 8, CHANNEL>(a, entries, s);
}
template <int D> static int launch_head_scan_kind(const DeltaHeadArgs& a, int entries, bool channel, cudaStream_t s) {
    return channel ? launch_head_scan_cols<D, true>(a, entries, s) : launch_head_scan_cols<D, false>(a, entries, s);
}

// The scan in pieces, for key sizes of 32, 64, 128 or 256, with one decay a head 96 as well.  head_decay: `decay` is [tokens][H] and `work`
// holds (tokens / 16 + entries) * (G * 32 * (D + 4) + H * 16 * 36) floats; else `decay` is [tokens][H][D]
// and `work` holds (tokens / 16 + entries) * H * (49 * (D + 4) + 16 * 36).  Returns 0, a CUDA error code,
// or -1 when the shape is refused.
MSTAR_API int mstar_delta_scan_pieces(const float* q, const float* k, const float* v,
                                      const float* beta, const float* decay,
                                      const int* qo_indptr, const int* slots, float* state,
                                      long long state_stride, long long state_offset, float* out,
                                      float* work, int tokens, int entries, int max_q_len, int H,
                                      int G, int D, int VD, int head_decay, int* error_word,
                                      const float* conv_raw, int conv_ld, int channels, int taps,
                                      void* stream) {
    if (entries <= 0 || tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || VD <= 0) return -1;
    if (D != 32 && D != 64 && D != 128 && D != 256 && !(D == 96 && head_decay)) return -1;
    if (H > 65535 || entries > 65535 || (state_offset % 4) != 0 || (state_stride % 4) != 0) return -1;
    if ((uintptr_t)q % 16 || (uintptr_t)k % 16 || (uintptr_t)work % 16 || (uintptr_t)state % 16 || !error_word ||
        (!head_decay && (uintptr_t)decay % 16))
        return -1;
    const int max_pieces = (max_q_len + GC_TOKENS - 1) / GC_TOKENS;
    const size_t most = (size_t)(tokens / GC_TOKENS + entries);
    const size_t row_floats = head_decay ? most * G * 2 * GC_TOKENS * (D + 4) : most * H * GK_ROWS(GC_TOKENS) * (D + 4);
    DeltaHeadArgs a{q, k, v, beta, decay, qo_indptr, slots, work, work + row_floats, state, state_stride, state_offset, out,
                    H, G, D, VD, tokens, error_word, {taps > 1 ? conv_raw : nullptr, conv_ld, channels, taps}};
    cudaStream_t s = (cudaStream_t)stream;
    if (head_decay) {
        // a warp a head in the second half of the first kernel: eight at most, as many as a group has
        const int per = H / G, warps = per < 8 ? per : 8;
        const size_t smem1 = (2 * (size_t)GC_TOKENS * (D + 4) + 2 * GC_TOKENS * GH_LD +
                              warps * (2 * GC_TOKENS * GH_LD + 2 * GC_TOKENS)) * sizeof(float);
        static size_t configured = 0;
        if (smem1 > 48 * 1024 && smem1 > configured) {
            cudaFuncSetAttribute(delta_head_pieces_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
            configured = smem1;
        }
        mstar_launch(delta_head_pieces_kernel, dim3(max_pieces, entries, G), dim3(256), smem1, s, a);
    } else {
        const size_t smem1 = ((size_t)128 * (D + 4) + 2 * GC_TOKENS * GH_LD) * sizeof(float);
        static size_t configured = 0;
        if (smem1 > 48 * 1024 && smem1 > configured) {
            cudaFuncSetAttribute(delta_channel_pieces_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
            configured = smem1;
        }
        mstar_launch(delta_channel_pieces_kernel, dim3(max_pieces, entries, H), dim3(256), smem1, s, a);
    }
    const int code = launch_status();
    if (code != 0) return code;
    if (D == 32) return launch_head_scan_kind<32>(a, entries, !head_decay, s);
    if (D == 64) return launch_head_scan_kind<64>(a, entries, !head_decay, s);
    if (D == 96) return launch_head_scan_cols<96, false>(a, entries, s);
    if (D == 128) return launch_head_scan_kind<128>(a, entries, !head_decay, s);
    return launch_head_scan_kind<256>(a, entries, !head_decay, s);
}

// ------------------------------------------------------------------ finish
// out[t, h, :] = o[t, h, :] / rms(o[t, h, :]) * weight[:] * act(gate[t, h, :]) * scale, act the
// sigmoid or the SiLU; a warp per (token, head).  V: elements an access; a lane keeps up to four
// accesses' worth of its head in registers.  Results that are rounded to bfloat16 take the quotient of
// 2 ulp, as the other gates do: 12.0 us for 2,048 tokens of 16 heads of 128, 13.8 with the IEEE division.
template <typename A> __device__ __forceinline__ float gd_over_one_plus(float x, float e) {
    if constexpr (sizeof(A) == 2) return over_one_plus_bf16(x, e);
    else return x / (1.f + e);
}
template <typename A, typename T, int V>
__global__ void delta_finish_kernel(const float* o, const T* gate, int gate_stride,
                                    const float* __restrict__ weight, A* __restrict__ out,
                                    int pairs, int heads, int vdim, float eps, float scale, int silu) {
    const unsigned long long waited = pdl_wait();
    o = pdl_after(o, waited);
    gate = pdl_after(gate, waited);
    const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (pair >= pairs) return;
    const int t = pair / heads, h = pair - t * heads;
    const float* row = o + (size_t)pair * vdim;
    const T* g = gate + (size_t)t * gate_stride + (size_t)h * vdim;
    A* dst = out + (size_t)pair * vdim;
    float ss = 0.f;
    if (vdim <= 128 * V) {
        float v[4][4], z[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = (i * 32 + lane) * V;
            if (j < vdim) {
                load_v<V>(row + j, v[i]);
                load_v<V>(g + j, z[i]);
#pragma unroll
                for (int e = 0; e < V; ++e) ss = fmaf(v[i][e], v[i][e], ss);
            }
        }
        const float inv = rsqrtf(warp_sum(ss) / (float)vdim + eps) * scale;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = (i * 32 + lane) * V;
            if (j < vdim) {
                float w[4];
                load_v<V>(weight + j, w);
#pragma unroll
                for (int e = 0; e < V; ++e)
                    v[i][e] = gd_over_one_plus<A>(v[i][e] * inv * w[e], expf(-z[i][e])) * (silu ? z[i][e] : 1.f);
                store_v<V>(dst + j, v[i]);
            }
        }
        return;
    }
    for (int j = lane; j < vdim; j += 32) ss = fmaf(row[j], row[j], ss);
    const float inv = rsqrtf(warp_sum(ss) / (float)vdim + eps) * scale;
    for (int j = lane; j < vdim; j += 32) {
        const float z = to_float(g[j]);
        dst[j] = from_float<A>(gd_over_one_plus<A>(row[j] * inv * weight[j], expf(-z)) * (silu ? z : 1.f));
    }
}

// gate_dtype: that of the activations, or float.
MSTAR_API int mstar_delta_finish(const float* o, const void* gate, int gate_stride,
                                 const float* weight, void* out, int act_dtype, int tokens,
                                 int heads, int vdim, float eps, float scale, int gate_dtype, int silu,
                                 void* stream) {
    if (tokens <= 0) return 0;
    if (gate_dtype != MSTAR_F32 && gate_dtype != act_dtype) return -1;
    const int pairs = tokens * heads, warps = 4;
    dim3 grid((pairs + warps - 1) / warps);
    cudaStream_t s = (cudaStream_t)stream;
    const bool vec = vdim % 4 == 0 && gate_stride % 4 == 0 && (uintptr_t)o % 16 == 0 &&
                     (uintptr_t)gate % 16 == 0 && (uintptr_t)weight % 16 == 0 && (uintptr_t)out % 16 == 0;
#define GO(A, T)                                                                                  \
    do {                                                                                          \
        if (vec)                                                                                  \
            mstar_launch((delta_finish_kernel<A, T, 4>), grid, dim3(32 * warps), 0, s, o,         \
                         (const T*)gate, gate_stride, weight, (A*)out, pairs, heads, vdim, eps,   \
                         scale, silu);                                                            \
        else                                                                                      \
            mstar_launch((delta_finish_kernel<A, T, 1>), grid, dim3(32 * warps), 0, s, o,         \
                         (const T*)gate, gate_stride, weight, (A*)out, pairs, heads, vdim, eps,   \
                         scale, silu);                                                            \
    } while (0)
    if (act_dtype == MSTAR_F32) GO(float, float);
    else if (gate_dtype == MSTAR_F32) GO(bf16, float);
    else GO(bf16, bf16);
#undef GO
    return launch_status();
}
