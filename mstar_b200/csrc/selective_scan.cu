// Selective scan (the Mamba mixer): a short causal convolution per channel with SiLU, and a
// diagonal linear recurrence per channel whose step size and input/output maps depend on the
// token.  Per-request state in a slot: the convolution's last taps-1 inputs [taps-1][inner],
// then S [inner][state], all float.
//
//   conv   xc[t, c] = silu(b_c + sum_k w[c, k] x[t - (taps-1) + k, c]), inputs before the
//          portion's start from the slot, zeros before the sequence's start (a fresh slot).
//   scan   dt = softplus(W_dt dt_in + b_dt);  S[c, n] = exp(dt_c A[c, n]) S[c, n] + dt_c xc_c B_n;
//          y_c = sum_n S[c, n] C_n + D_c xc_c;  out = y * silu(z).
//
// Step sizes, decays, their exponentials, the state and its sums are float for both
// activation types.  A channel's arithmetic depends on its own portion and on whether the batch holds a
// long portion (which has the step sizes' product made ahead and portions cut into pieces), on nothing
// else of the batch: how a portion is cut follows from its own length.
#include <type_traits>

#include "common.cuh"
#include "gemm_f32.h"
#include "mma_util.cuh"

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// ------------------------------------------------------------------ convolution + SiLU
// xz: [tokens] rows of ld elements, x in columns [0, inner).  One thread per (token, channel):
// a block row of the grid is a token, so neighbours in a warp are neighbouring channels.
template <typename A, typename W>
__global__ void conv_silu_kernel(const A* __restrict__ xz, int ld, const W* __restrict__ w,
                                 const W* __restrict__ bias, const int* __restrict__ token_req,
                                 const int* __restrict__ qo_indptr, const int* __restrict__ slots,
                                 const float* __restrict__ state, long long state_stride,
                                 A* __restrict__ out, int t_first, int inner, int taps) {
    xz = pdl_after(xz, pdl_wait());
    const int t = t_first + blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= inner) return;
    const size_t idx = (size_t)t * inner + c;
    const int e = token_req[t];
    const int start = qo_indptr[e], local = t - start;
    const float* past = state + (size_t)slots[e] * state_stride;   // [taps-1][inner]
    float acc = to_float(bias[c]);
    for (int k = 0; k < taps; ++k) {
        const int src = local - (taps - 1) + k;
        const float v = src >= 0 ? to_float(xz[(size_t)(start + src) * ld + c])
                                 : past[(size_t)(taps - 1 + src) * inner + c];
        acc = fmaf(to_float(w[(size_t)c * taps + k]), v, acc);
    }
    out[idx] = from_float<A>(silu_f(acc));
}

template <typename A> __device__ __forceinline__ float conv_silu_of(float v);
template <> __device__ __forceinline__ float conv_silu_of<float>(float v) { return silu_f(v); }
template <> __device__ __forceinline__ float conv_silu_of<bf16>(float v) { return silu_bf16(v); }

// The same for 8 channels a thread with 16-byte accesses: weights transposed to float
// [taps][inner], bias float; inner and ld multiples of 8.
template <typename A>
__global__ void conv_silu_vec_kernel(const A* __restrict__ xz, int ld, const float* __restrict__ wt,
                                     const float* __restrict__ bias, const int* __restrict__ token_req,
                                     const int* __restrict__ qo_indptr, const int* __restrict__ slots,
                                     const float* __restrict__ state, long long state_stride,
                                     A* __restrict__ out, int t_first, int inner, int taps) {
    xz = pdl_after(xz, pdl_wait());
    const int t = t_first + blockIdx.y, c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= inner) return;
    const int e = token_req[t];
    const int start = qo_indptr[e], local = t - start;
    const float* past = state + (size_t)slots[e] * state_stride;
    float acc[8];
    load8(bias + c, acc);
    for (int k = 0; k < taps; ++k) {
        const int src = local - (taps - 1) + k;
        float v[8], w[8];
        if (src >= 0) load8(xz + (size_t)(start + src) * ld + c, v);
        else load8(past + (size_t)(taps - 1 + src) * inner + c, v);
        load8(wt + (size_t)k * inner + c, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(w[i], v[i], acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = conv_silu_of<A>(acc[i]);
    store8(out + (size_t)t * inner + c, acc);
}

// For prompts, four taps: CS_RUN tokens a thread, so that the weights (twice the bytes of the rows) and
// rows are read once for all of them.  Where these are of several entries each is done as above.
// What counts is instructions: 2 x 1,024 tokens of 4,096 channels take 12.5 us, a token a thread with the
// quotient in IEEE division 19.
#define CS_RUN 4
template <typename A>
__global__ void __launch_bounds__(128)
conv_silu_run_kernel(const A* __restrict__ xz, int ld, const float* __restrict__ wt, const float* __restrict__ bias,
                     const int* __restrict__ token_req, const int* __restrict__ qo_indptr,
                     const int* __restrict__ slots, const float* __restrict__ state, long long state_stride,
                     A* __restrict__ out, int t_first, int t_end, int inner) {
    xz = pdl_after(xz, pdl_wait());
    const int first = t_first + blockIdx.y * CS_RUN, many = min(CS_RUN, t_end - first);
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= inner) return;
    float w[4][8], b[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) load8(wt + (size_t)k * inner + c, w[k]);
    load8(bias + c, b);
    const int e0 = token_req[first];
    const int step = token_req[first + many - 1] == e0 ? many : 1;
    for (int t0 = first; t0 < first + many; t0 += step) {
        const int e = token_req[t0], local = t0 - qo_indptr[e];
        const float* past = state + (size_t)slots[e] * state_stride;       // [3][inner]
        const A* row = xz + (size_t)t0 * ld + c;
        float v[4][8];                           // the rows of the taps, row i of the portion at i % 4
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (local >= 3 - i) load8(row - (ptrdiff_t)(3 - i) * ld, v[i]);
            else load8(past + (size_t)(local + i) * inner + c, v[i]);
        }
#pragma unroll
        for (int t = 0; t < CS_RUN; ++t) {
            if (t >= step) break;
            load8(row + (size_t)t * ld, v[(t + 3) % 4]);
            float acc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i] = b[i];
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[i] = fmaf(w[k][i], v[(t + k) % 4][i], acc[i]);
                acc[i] = conv_silu_of<A>(acc[i]);
            }
            store8(out + (size_t)(t0 + t) * inner + c, acc);
        }
    }
}

MSTAR_API int mstar_conv_silu_vec(const void* xz, int ld, const float* wt, const float* bias,
                                  const int* token_req, const int* qo_indptr, const int* slots,
                                  const float* state, long long state_stride, void* out,
                                  int act_dtype, int tokens, int inner, int taps, void* stream) {
    if (tokens <= 0) return 0;
    if (inner <= 0 || taps <= 0 || inner % 8 || ld % 8 || state_stride % 4) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    const int lanes = inner / 8;
    const int threads = lanes >= 128 ? 128 : 32;
    // several tokens a thread where that still gives every SM two blocks (4,096 channels: 512 tokens 12.3 us
    // against 14.4, 128 tokens 10.2 against 10.3, 64 tokens 10.3 against 8.3)
    const int columns = (lanes + threads - 1) / threads;
    if (taps == 4 && (long long)((tokens + CS_RUN - 1) / CS_RUN) * columns >= 2LL * device_sm_count()) {
        for (int t0 = 0; t0 < tokens; t0 += 65535 * CS_RUN) {
            const int end = tokens - t0 < 65535 * CS_RUN ? tokens : t0 + 65535 * CS_RUN;
            const dim3 blocks(columns, (end - t0 + CS_RUN - 1) / CS_RUN);
            if (act_dtype == MSTAR_F32)
                mstar_launch((conv_silu_run_kernel<float>), blocks, dim3(threads), 0, s, (const float*)xz, ld, wt,
                             bias, token_req, qo_indptr, slots, state, state_stride, (float*)out, t0, end, inner);
            else
                mstar_launch((conv_silu_run_kernel<bf16>), blocks, dim3(threads), 0, s, (const bf16*)xz, ld, wt,
                             bias, token_req, qo_indptr, slots, state, state_stride, (bf16*)out, t0, end, inner);
        }
        return launch_status();
    }
    for (int t0 = 0; t0 < tokens; t0 += 65535) {
        const dim3 blocks(columns, tokens - t0 < 65535 ? tokens - t0 : 65535);
        if (act_dtype == MSTAR_F32)
            mstar_launch((conv_silu_vec_kernel<float>), blocks, dim3(threads), 0, s, (const float*)xz,
                         ld, wt, bias, token_req, qo_indptr, slots, state, state_stride, (float*)out,
                         t0, inner, taps);
        else
            mstar_launch((conv_silu_vec_kernel<bf16>), blocks, dim3(threads), 0, s, (const bf16*)xz,
                         ld, wt, bias, token_req, qo_indptr, slots, state, state_stride, (bf16*)out,
                         t0, inner, taps);
    }
    return launch_status();
}

MSTAR_API int mstar_conv_silu(const void* xz, int ld, const void* w, const void* bias,
                              int weight_dtype, const int* token_req, const int* qo_indptr,
                              const int* slots, const float* state, long long state_stride,
                              void* out, int act_dtype, int tokens, int inner, int taps,
                              void* stream) {
    if (tokens <= 0) return 0;
    if (inner <= 0 || taps <= 0) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    const int threads = inner >= 256 ? 256 : 64;
#define GO(A, W)                                                                                  \
    mstar_launch((conv_silu_kernel<A, W>), blocks, dim3(threads), 0, s, (const A*)xz, ld,         \
                 (const W*)w, (const W*)bias, token_req, qo_indptr, slots, state, state_stride,   \
                 (A*)out, t0, inner, taps)
    // (a grid's second dimension ends at 65,535: longer batches go in slices)
    for (int t0 = 0; t0 < tokens; t0 += 65535) {
        const dim3 blocks((inner + threads - 1) / threads, tokens - t0 < 65535 ? tokens - t0 : 65535);
        if (act_dtype == MSTAR_F32) {
            if (weight_dtype == MSTAR_F32) { GO(float, float); } else { GO(float, bf16); }
        } else {
            if (weight_dtype == MSTAR_F32) { GO(bf16, float); } else { GO(bf16, bf16); }
        }
    }
#undef GO
    return launch_status();
}

// ------------------------------------------------------------------ the recurrence
#define SS_THREADS 64     // threads of a block: SS_THREADS / LANES channels
#define SS_TC 16          // tokens staged at a time

// 4 bytes global -> shared, asynchronously (rows of floats have no wider alignment)
__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_all_done() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Tokens of a piece where the kernel for 16 states cuts a portion of n tokens: some 16 pieces, by the
// portion's own length alone, so that its sums do not depend on the batch (600 tokens of 2,048 channels:
// 44 us in pieces of 64, 52 of 128; 2,048 of 4,096: 217 of 128, 223 and 226 of 64 and 256; 8,192: 809 of
// 256, 832 of 128).
// Shorter portions stay whole: one of 130 tokens of 4,096 channels took 32 us either way, one of 100 28 us
// against 30 in two pieces, one of 333 58 against 46; with several of them the SMs are full and whole is
// faster (three of 333: 85 against 97).  At the line, 191 tokens whole and 192 in three pieces: 37 and 31 us of 4,096 channels,
// 35 and 25 of 2,048, 31 and 21 of 1,024, 57 and 55 of 8,192.  The whole ones pay some 4 of that for an exponential that
// is nearer (error of the outputs against 64 bits, one portion of 60 tokens: 7.7e-8, with 2^x 1.3e-7).
#define SCAN_CUT_FROM 192
__host__ __device__ __forceinline__ int scan_piece(int n) {
    if (n < SCAN_CUT_FROM) return SCAN_CUT_FROM;
    const int p = n / 16 / 64 * 64;
    return p < 64 ? 64 : p > 256 ? 256 : p;
}

struct ScanArgs {
    int inner, n_state, rank, taps, ld_xz, entries;
    long long state_stride;
    // a long portion is cut into pieces of `piece` tokens (0: not cut; below 0, in the kernel for 16 states:
    // scan_piece of its own length) that run side by side:
    // pass 1 walks every piece but the last from a zero state and leaves its end state and the
    // sum of its step sizes in scratch (the recurrence is linear: the state after a piece is
    // exp(A sum dt) times the state before it, plus that end state); pass 2 starts every piece
    // from the state so joined and writes the outputs
    int piece, pass, max_pieces;
    float* piece_state;   // [entries][max_pieces][inner][n_state]; piece < 0: [tokens / 64 + entries][..]
    float* piece_dt;      // [entries][max_pieces][inner]; likewise
    // W_dt dt_in of every token and channel, made by a product of its own [tokens][inner], or nullptr: the kernel makes it from the staged rows.  Pass 1 of the kernel for
    // 16 states leaves the step sizes made of it in its place.
    float* dt_pre;
};

// A block takes one batch entry and SS_THREADS / LANES channels; LANES lanes share a channel:
// lane s holds states s, s + LANES, ... (NPER of them).  Tokens come in chunks of SS_TC: the
// chunk's [dt_in | B | C] rows, conv outputs and gates stand in shared memory, and the next
// chunk's are on their way (the rows by asynchronous copies into the other buffer, x and z
// in registers) while this one is walked.  The step sizes of a chunk
// are made for all its tokens at once (W_dt read once a chunk), then the chain runs token by
// token: one multiply-add per state on the chain, the decays' exponentials beside it.  At the
// end the state goes back to the slot and the convolution's window moves on.
template <typename A, int LANES, int NPER>
__global__ void __launch_bounds__(SS_THREADS, 8)
selective_scan_kernel(const A* __restrict__ xc, const A* __restrict__ xz,
                      const float* __restrict__ proj, const float* __restrict__ w_dt,
                      const float* __restrict__ dt_bias, const float* __restrict__ a_neg,
                      const float* __restrict__ d_skip, const int* __restrict__ qo_indptr,
                      const int* __restrict__ slots, float* __restrict__ state,
                      A* __restrict__ out, ScanArgs a) {
    constexpr int CH = SS_THREADS / LANES;
    extern __shared__ float sm[];
    const int row = a.rank + 2 * a.n_state;
    const int buf_floats = SS_TC * row + 3 * SS_TC * CH;   // rows, then x, z, and W_dt dt_in
    const int e = blockIdx.x;
    const int tid = threadIdx.x, sub = tid % LANES, ch = tid / LANES;
    const int c = blockIdx.y * CH + ch;
    const bool live = c < a.inner;
    const int cc = live ? c : a.inner - 1;
    const unsigned long long waited = pdl_wait();
    xc = pdl_after(xc, waited);
    xz = pdl_after(xz, waited);
    proj = pdl_after(proj, waited);
    const int e_start = qo_indptr[e], e_tok = qo_indptr[e + 1] - e_start;
    // this block's piece of the entry's tokens
    const int piece = blockIdx.z;
    const int pieces = a.piece > 0 ? max(1, (e_tok + a.piece - 1) / a.piece) : 1;
    if (piece >= pieces || (a.pass == 1 && piece == pieces - 1)) return;
    const int start = e_start + piece * (a.piece > 0 ? a.piece : 0);
    const int n_tok = a.piece > 0 ? min(a.piece, e_tok - piece * a.piece) : e_tok;
    const bool last_piece = piece == pieces - 1;
    float* slot = state + (size_t)slots[e] * a.state_stride;
    float* s_slot = slot + (size_t)(a.taps - 1) * a.inner + (size_t)cc * a.n_state;

    float S[NPER], An[NPER];
#pragma unroll
    for (int i = 0; i < NPER; ++i) {
        const int n = sub + LANES * i;
        S[i] = 0.f;
        // A in units of log2(e): the decays are then 2^(dt A), one exponential instruction
        An[i] = n < a.n_state ? a_neg[(size_t)cc * a.n_state + n] * 1.4426950408889634f : 0.f;
    }
    // The state the portion starts from.  Cut into pieces, the last piece puts the new state
    // into the slot while others may not have started: so pass 1 leaves a copy of the old one
    // in the scratch entry of the last piece (which pass 1 does not walk), and pass 2 reads that.
    float* kept_start = a.piece_state + (((size_t)e * a.max_pieces + pieces - 1) * a.inner + cc) * a.n_state;
    const float* s_from = (a.pass == 2 && pieces > 1) ? kept_start : s_slot;
    if (a.pass == 1 && piece == 0 && live) {
#pragma unroll
        for (int i = 0; i < NPER; ++i) {
            const int n = sub + LANES * i;
            if (n < a.n_state) kept_start[n] = s_slot[n];
        }
    }
    if (a.pass != 1) {
#pragma unroll
        for (int i = 0; i < NPER; ++i) {
            const int n = sub + LANES * i;
            if (n < a.n_state) S[i] = s_from[n];
        }
    }
    if (a.pass == 2) {
        // the state before this piece: the slot's, carried over the pieces before it
        for (int j = 0; j < piece; ++j) {
            const size_t at = (size_t)e * a.max_pieces + j;
            const float sdt = a.piece_dt[at * a.inner + cc];
            const float* E = a.piece_state + (at * a.inner + cc) * a.n_state;
#pragma unroll
            for (int i = 0; i < NPER; ++i) {
                const int n = sub + LANES * i;
                if (n < a.n_state) S[i] = fmaf(exp2f(sdt * An[i]), S[i], E[n]);
            }
        }
    }
    float dt_sum = 0.f;
    const float bias = dt_bias[cc], dsk = d_skip[cc];
    const float* wrow = w_dt + (size_t)cc * a.rank;

    // what a thread fetches of a chunk: its share of the rows, and of the x and z values
    const int row_items = SS_TC * row, xz_items = SS_TC * CH;
    float pf_x[(SS_TC * CH + SS_THREADS - 1) / SS_THREADS],
        pf_z[(SS_TC * CH + SS_THREADS - 1) / SS_THREADS],
        pf_d[(SS_TC * CH + SS_THREADS - 1) / SS_THREADS];
    const float* dt_pre = pdl_after((const float*)a.dt_pre, waited);
    auto fetch = [&](float* buf, int t0, int nt) {
        const float* src = proj + (size_t)(start + t0) * row;
        for (int i = tid; i < nt * row; i += SS_THREADS) cp_async_4(buf + i, src + i);
#pragma unroll
        for (int k = 0; k < (xz_items + SS_THREADS - 1) / SS_THREADS; ++k) {
            const int i = tid + k * SS_THREADS;
            const int tk = i / CH, j = i - tk * CH;
            const int col = min(blockIdx.y * CH + j, a.inner - 1);
            const bool ok = i < xz_items && tk < nt;
            pf_x[k] = ok ? to_float(xc[(size_t)(start + t0 + tk) * a.inner + col]) : 0.f;
            pf_z[k] = ok ? to_float(xz[(size_t)(start + t0 + tk) * a.ld_xz + a.inner + col]) : 0.f;
            pf_d[k] = (ok && a.dt_pre != nullptr) ? dt_pre[(size_t)(start + t0 + tk) * a.inner + col] : 0.f;
        }
    };
    auto stash = [&](float* buf) {
        cp_async_all_done();
#pragma unroll
        for (int k = 0; k < (xz_items + SS_THREADS - 1) / SS_THREADS; ++k) {
            const int i = tid + k * SS_THREADS;
            if (i < xz_items) {
                buf[row_items + i] = pf_x[k];
                buf[row_items + xz_items + i] = pf_z[k];
                buf[row_items + 2 * xz_items + i] = pf_d[k];
            }
        }
    };

    if (n_tok > 0) {
        fetch(sm, 0, min(SS_TC, n_tok));
        stash(sm);
    }
    __syncthreads();
    int which = 0;
    for (int t0 = 0; t0 < n_tok; t0 += SS_TC, which ^= 1) {
        const int nt = min(SS_TC, n_tok - t0);
        const bool more = t0 + SS_TC < n_tok;
        if (more) fetch(sm + (which ^ 1) * buf_floats, t0 + SS_TC, min(SS_TC, n_tok - t0 - SS_TC));
        const float* rows = sm + which * buf_floats;
        const float* xs = rows + row_items;
        const float* zs = xs + xz_items;
        const float* ds = zs + xz_items;
        if (nt < SS_TC) {
            // a short portion, or a portion's tail: token by token
            for (int k = 0; k < nt; ++k) {
                float d = 0.f;
                if (a.dt_pre != nullptr) {
                    d = ds[k * CH + ch];
                } else {
                    for (int r = sub; r < a.rank; r += LANES) d = fmaf(wrow[r], rows[k * row + r], d);
#pragma unroll
                    for (int o = LANES / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                }
                d = softplus_f(d + bias);
                dt_sum += d;
                const float x = xs[k * CH + ch];
                const float dx = d * x;
                const float* B = rows + k * row + a.rank;
                const float* C = B + a.n_state;
                float y = 0.f;
#pragma unroll
                for (int i = 0; i < NPER; ++i) {
                    const int n = sub + LANES * i;
                    if (n < a.n_state) {
                        S[i] = fmaf(exp2f(d * An[i]), S[i], dx * B[n]);
                        y = fmaf(S[i], C[n], y);
                    }
                }
#pragma unroll
                for (int o = LANES / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                if (sub == 0 && live && a.pass != 1)
                    out[(size_t)(start + t0 + k) * a.inner + c] =
                        from_float<A>(fmaf(dsk, x, y) * silu_f(zs[k * CH + ch]));
            }
        } else {
            // step sizes of the chunk
            float dt[SS_TC];
            if (a.dt_pre != nullptr) {
                // the softplus of a channel's 16 step sizes is dealt out among its lanes (in
                // place in the staged values), not made by each of them
                float* dsw = sm + which * buf_floats + row_items + 2 * xz_items;
#pragma unroll
                for (int j = 0; j < SS_TC / LANES; ++j) {
                    const int k = sub + LANES * j;
                    dsw[k * CH + ch] = softplus_f(dsw[k * CH + ch] + bias);
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < SS_TC; ++k) {
                    dt[k] = ds[k * CH + ch];
                    dt_sum += dt[k];
                }
            } else {
#pragma unroll
                for (int k = 0; k < SS_TC; ++k) dt[k] = 0.f;
                for (int r = sub; r < a.rank; r += LANES) {
                    const float w = wrow[r];
#pragma unroll
                    for (int k = 0; k < SS_TC; ++k) dt[k] = fmaf(w, rows[k * row + r], dt[k]);
                }
#pragma unroll
                for (int k = 0; k < SS_TC; ++k) {
#pragma unroll
                    for (int o = LANES / 2; o > 0; o >>= 1)
                        dt[k] += __shfl_xor_sync(0xffffffffu, dt[k], o);
                }
#pragma unroll
                for (int k = 0; k < SS_TC; ++k) {
                    dt[k] = softplus_f(dt[k] + bias);
                    dt_sum += dt[k];
                }
            }
            // the chain, SUB tokens at a time: first everything that does not depend on the
            // state (decays exp(dt A), inputs dt x B), then one multiply-add per state and token
            // on the chain with the output sums beside it, then the sums of the lanes and the
            // gated outputs, the tokens dealt out among the lanes of a channel
            constexpr int SUB = NPER <= 1 ? SS_TC : (NPER <= 4 ? 8 : 2);
#pragma unroll
            for (int k0 = 0; k0 < SS_TC; k0 += SUB) {
                float da[SUB][NPER], db[SUB][NPER], yk[SUB];
#pragma unroll
                for (int kk = 0; kk < SUB; ++kk) {
                    const int k = k0 + kk;
                    const float dx = dt[k] * xs[k * CH + ch];
                    const float* B = rows + k * row + a.rank;
#pragma unroll
                    for (int i = 0; i < NPER; ++i) {
                        const int n = sub + LANES * i;
                        const bool use = n < a.n_state;
                        da[kk][i] = use ? exp2f(dt[k] * An[i]) : 1.f;
                        db[kk][i] = use ? dx * B[use ? n : 0] : 0.f;
                    }
                }
#pragma unroll
                for (int kk = 0; kk < SUB; ++kk) {
                    const float* C = rows + (k0 + kk) * row + a.rank + a.n_state;
                    float y = 0.f;
#pragma unroll
                    for (int i = 0; i < NPER; ++i) {
                        const int n = sub + LANES * i;
                        S[i] = fmaf(da[kk][i], S[i], db[kk][i]);
                        y = fmaf(S[i], n < a.n_state ? C[n] : 0.f, y);
                    }
                    yk[kk] = y;
                }
                if (a.pass != 1) {
#pragma unroll
                    for (int kk = 0; kk < SUB; ++kk) {
#pragma unroll
                        for (int o = LANES / 2; o > 0; o >>= 1)
                            yk[kk] += __shfl_xor_sync(0xffffffffu, yk[kk], o);
                    }
#pragma unroll
                    for (int kk = 0; kk < SUB; ++kk) {
                        const int k = k0 + kk;
                        if (kk % LANES == sub && live) {
                            const float y = fmaf(dsk, xs[k * CH + ch], yk[kk]);
                            out[(size_t)(start + t0 + k) * a.inner + c] =
                                from_float<A>(y * silu_f(zs[k * CH + ch]));
                        }
                    }
                }
            }
        }
        if (more) stash(sm + (which ^ 1) * buf_floats);
        __syncthreads();
    }
    if (!live) return;
    if (a.pass == 1) {                         // this piece alone, for the pieces after it
        const size_t at = (size_t)e * a.max_pieces + piece;
        float* E = a.piece_state + (at * a.inner + c) * a.n_state;
#pragma unroll
        for (int i = 0; i < NPER; ++i) {
            const int n = sub + LANES * i;
            if (n < a.n_state) E[n] = S[i];
        }
        if (sub == 0) a.piece_dt[at * a.inner + c] = dt_sum;
        return;
    }
    if (!last_piece) return;
#pragma unroll
    for (int i = 0; i < NPER; ++i) {
        const int n = sub + LANES * i;
        if (n < a.n_state) s_slot[n] = S[i];
    }
    if (sub == 0 && e_tok > 0) {
        // the window of the convolution: the last taps-1 inputs of [old window | this portion]
        for (int j = 0; j < a.taps - 1; ++j) {
            const int at = e_tok + j;                  // index into the joined sequence
            slot[(size_t)j * a.inner + c] =
                at < a.taps - 1 ? slot[(size_t)at * a.inner + c]
                                : to_float(xz[(size_t)(e_start + at - (a.taps - 1)) * a.ld_xz + c]);
        }
    }
}

// The same for 16 states a channel and step sizes' products made by the caller (long portions). Lane s of a
// channel's four holds states 4 s .. 4 s + 3 as two pairs, so that B and C come as one 16-byte
// load each and multiplications run two to an instruction (f32x2); a chunk's [B | C], x, z and
// step sizes come by 16-byte asynchronous copies, STAGES - 1 chunks ahead, the rest of the projection
// rows stays where it is.  Tokens past the portion's end get a step size of 0 and leave the
// state as it is.  The output sums of four tokens meet in one exchange among the lanes, each of which
// then finishes one token.  Bound by the exponential (one ex2 per state and token: 30 us for 2,048 tokens x
// 4,096 channels at 16 a cycle and SM) and by one warp a scheduler where channels are few.
// 2 x 1,024 tokens, 4,096 channels, pieces of 64: 49 + 69 us for the two passes one at a time with cold caches (64
// + 94 with the step sizes made in both, the copies' addresses made anew for every chunk and every token asked
// for its place in it: instructions took 82 % of the issue slots); the kernel above takes 203 us each (a 4-byte copy for every
// number of the rows, two 4-byte loads of B and C a state, exp2f).
#define SX_STAGES 3

__device__ __forceinline__ unsigned long long sx_pack(float lo, float hi) {
    return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float sx_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float sx_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ unsigned long long sx_mul(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long sx_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// 2^x for x <= 0 (what underflows is 0)
__device__ __forceinline__ float sx_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The decays of two states, of dt A (exact) or of dt A log2(e): portions that are not cut keep the exponential of the
// kernel for any state, whose error the few roundings of a short portion do not hide.
template <bool EXACT> __device__ __forceinline__ unsigned long long sx_decays(unsigned long long z) {
    return EXACT ? sx_pack(expf(sx_lo(z)), expf(sx_hi(z))) : sx_pack(sx_ex2(sx_lo(z)), sx_ex2(sx_hi(z)));
}
__device__ __forceinline__ float sx_silu(float v, bf16) { return silu_bf16(v); }
__device__ __forceinline__ float sx_silu(float v, float) { return silu_f(v); }

template <typename A> struct ScanStage {
    float bc[SS_TC][32];            // B then C
    float d[SS_TC][32];             // W_dt dt_in, then the step size
    A x[SS_TC][32], z[SS_TC][32];
};

// PASS as in the kernel above: 0 whole portions, 1 a piece from zero state, 2 a piece from the state
// that the pieces before it leave.
template <typename A, int PASS>
__global__ void __launch_bounds__(128)
selective_scan16_kernel(const A* __restrict__ xc, const A* __restrict__ xz, const float* __restrict__ proj,
                        const float* __restrict__ dt_bias, const float* __restrict__ a_neg,
                        const float* __restrict__ d_skip, const int* __restrict__ qo_indptr,
                        const int* __restrict__ slots, float* __restrict__ state, A* __restrict__ out, ScanArgs a) {
    __shared__ __align__(16) ScanStage<A> stage[SX_STAGES];
    const int e = blockIdx.x, piece = blockIdx.z;
    const int tid = threadIdx.x, sub = tid & 3, ch = tid >> 2;
    const int c0 = blockIdx.y * 32, c = c0 + ch;
    const unsigned long long waited = pdl_wait();
    xc = pdl_after(xc, waited);
    xz = pdl_after(xz, waited);
    proj = pdl_after(proj, waited);
    const float* dt_pre = pdl_after((const float*)a.dt_pre, waited);
    float* dt_made = pdl_after(a.dt_pre, waited);
    const int e_start = qo_indptr[e], e_tok = qo_indptr[e + 1] - e_start;
    const int len = a.piece > 0 ? a.piece : scan_piece(e_tok);
    // the scratch of the entry's first piece: entries take max_pieces each, or, cut by their own lengths, one
    // for every started 64 tokens
    const size_t at0 = a.piece > 0 ? (size_t)e * a.max_pieces : (size_t)(e_start / 64 + e);
    const int pieces = PASS != 0 ? max(1, (e_tok + len - 1) / len) : 1;
    if (piece >= pieces || (PASS == 1 && piece == pieces - 1)) return;
    const int start = e_start + (PASS != 0 ? piece * len : 0);
    const int n_tok = PASS != 0 ? min(len, e_tok - piece * len) : e_tok;
    float* slot = state + (size_t)slots[e] * a.state_stride;
    float* s_slot = slot + (size_t)(a.taps - 1) * a.inner + (size_t)c * 16 + 4 * sub;
    const int row = a.rank + 32;

    // A thread copies the same places of every chunk: 16-byte piece i = tid, tid + 128, .. of the chunk's
    // tokens (8 pieces of [B | C], 8 of step sizes, XQ of x, XQ of z each); what moves on is the source.
    constexpr int XQ = 32 * (int)sizeof(A) / 16, PER = 16 + 2 * XQ, ITEMS = SS_TC * PER / 128;
    const char* from[ITEMS];
    uint32_t step[ITEMS], to[ITEMS];
#pragma unroll
    for (int m = 0; m < ITEMS; ++m) {
        const int i = tid + 128 * m, k = i / PER, q = i - k * PER;
        const size_t t = (size_t)(start + k);
        const ScanStage<A>* st = stage;
        if (q < 8) {
            from[m] = reinterpret_cast<const char*>(proj + t * row + a.rank + 4 * q);
            step[m] = (uint32_t)row * SS_TC * sizeof(float);
            to[m] = smem_u32(&st->bc[k][4 * q]);
        } else if (q < 16) {
            from[m] = reinterpret_cast<const char*>(dt_pre + t * a.inner + c0 + 4 * (q - 8));
            step[m] = (uint32_t)a.inner * SS_TC * sizeof(float);
            to[m] = smem_u32(&st->d[k][4 * (q - 8)]);
        } else {
            const bool is_x = q < 16 + XQ;
            const int part = q - (is_x ? 16 : 16 + XQ);
            from[m] = reinterpret_cast<const char*>(is_x ? xc + t * a.inner + c0 : xz + t * a.ld_xz + a.inner + c0) + 16 * part;
            step[m] = (uint32_t)(is_x ? a.inner : a.ld_xz) * SS_TC * sizeof(A);
            to[m] = smem_u32(is_x ? st->x[k] : st->z[k]) + 16 * part;
        }
    }
    auto fetch = [&](int t0) {                    // chunks in order
        const uint32_t at = (uint32_t)((t0 / SS_TC) % SX_STAGES * sizeof(ScanStage<A>));
#pragma unroll
        for (int m = 0; m < ITEMS; ++m) {
            if (t0 + (tid + 128 * m) / PER < n_tok) cp_async_16(to[m] + at, from[m], 16);
            from[m] += step[m];
        }
    };
#pragma unroll
    for (int s = 0; s < SX_STAGES - 1; ++s) {
        if (s * SS_TC < n_tok) fetch(s * SS_TC);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    // A in units of log2(e): the decays are then 2^(dt A); exact: A as it is
    const bool exact = PASS != 1 && pieces == 1 && e_tok < SCAN_CUT_FROM;
    unsigned long long S[2], An[2];
    {
        const float4 an = *reinterpret_cast<const float4*>(a_neg + (size_t)c * 16 + 4 * sub);
        const float L = exact ? 1.f : 1.4426950408889634f;
        An[0] = sx_pack(an.x * L, an.y * L);
        An[1] = sx_pack(an.z * L, an.w * L);
    }
    // (the last piece puts the new state into the slot while others may not have started: pass 1
    // leaves a copy of the old one in the scratch entry of the last piece, which pass 2 reads)
    float* kept = PASS != 0 ? a.piece_state + ((at0 + pieces - 1) * a.inner + c) * 16 + 4 * sub : nullptr;
    if (PASS == 1 && piece == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) kept[i] = s_slot[i];
    }
    if (PASS == 1) {
        S[0] = S[1] = 0ull;
    } else {
        const float* from = PASS == 2 && pieces > 1 ? kept : s_slot;
        S[0] = sx_pack(from[0], from[1]);
        S[1] = sx_pack(from[2], from[3]);
    }
    if (PASS == 2) {
        for (int j = 0; j < piece; ++j) {
            const size_t at = at0 + j;
            const float sdt = a.piece_dt[at * a.inner + c];
            const float4 E = *reinterpret_cast<const float4*>(a.piece_state + (at * a.inner + c) * 16 + 4 * sub);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                S[i] = sx_fma(sx_pack(sx_ex2(sdt * sx_lo(An[i])), sx_ex2(sdt * sx_hi(An[i]))), S[i],
                              i == 0 ? sx_pack(E.x, E.y) : sx_pack(E.z, E.w));
        }
    }
    float dt_sum = 0.f;
    const float bias = dt_bias[c], dsk = d_skip[c];

    // The step sizes that pass 1 made lie where it found their products.
    const bool made = PASS == 2 && piece < pieces - 1;

    auto walk = [&](auto whole, auto exactly, ScanStage<A>& st, int t0, int nt) {
        constexpr bool WHOLE = decltype(whole)::value, EXACT = decltype(exactly)::value;
        if (!made || !WHOLE) {
            // the softplus of a channel's step sizes is dealt out among its lanes
#pragma unroll
            for (int j = 0; j < SS_TC / 4; ++j) {
                const int k = sub + 4 * j;
                float dt = 0.f;
                if (WHOLE || k < nt) {
                    dt = st.d[k][ch];
                    if (!made) dt = softplus_f(dt + bias);
                    if (PASS == 1) dt_made[(size_t)(start + t0 + k) * a.inner + c] = dt;
                }
                st.d[k][ch] = dt;
            }
            __syncwarp();
        }
#pragma unroll
        for (int k0 = 0; k0 < SS_TC; k0 += 4) {
            unsigned long long da[4][2], db[4][2];
            float y[4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const int k = k0 + kk;
                const bool here = WHOLE || k < nt;
                const float dt = st.d[k][ch], dx = here ? dt * to_float(st.x[k][ch]) : 0.f;
                if (PASS == 1) dt_sum += dt;
                const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(&st.bc[k][4 * sub]);
                const unsigned long long dt2 = sx_pack(dt, dt), dx2 = sx_pack(dx, dx);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const unsigned long long z = sx_mul(dt2, An[i]);
                    da[kk][i] = sx_decays<EXACT>(z);
                    db[kk][i] = here ? sx_mul(dx2, i == 0 ? B.x : B.y) : 0ull;
                }
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                S[0] = sx_fma(da[kk][0], S[0], db[kk][0]);
                S[1] = sx_fma(da[kk][1], S[1], db[kk][1]);
                if (PASS != 1) {
                    const ulonglong2 C = *reinterpret_cast<const ulonglong2*>(&st.bc[k0 + kk][16 + 4 * sub]);
                    const unsigned long long y2 = sx_fma(S[1], C.y, sx_mul(S[0], C.x));
                    y[kk] = sx_lo(y2) + sx_hi(y2);
                }
            }
            if (PASS != 1) {
                // lane s ends up with the sum of token k0 + s over the four lanes
                const bool odd = sub & 1, high = sub & 2;
                const float r0 = (odd ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, odd ? y[0] : y[1], 1);
                const float r1 = (odd ? y[3] : y[2]) + __shfl_xor_sync(0xffffffffu, odd ? y[2] : y[3], 1);
                const float sum = (high ? r1 : r0) + __shfl_xor_sync(0xffffffffu, high ? r0 : r1, 2);
                const int k = k0 + sub;
                if (WHOLE || k < nt)
                    out[(size_t)(start + t0 + k) * a.inner + c] = from_float<A>(
                        fmaf(dsk, to_float(st.x[k][ch]), sum) * sx_silu(to_float(st.z[k][ch]), A()));
            }
        }
    };

    for (int t0 = 0; t0 < n_tok; t0 += SS_TC) {
        asm volatile("cp.async.wait_group %0;" ::"n"(SX_STAGES - 2) : "memory");
        __syncthreads();            // the chunk is there, and the one before it is done with
        if (t0 + (SX_STAGES - 1) * SS_TC < n_tok) fetch(t0 + (SX_STAGES - 1) * SS_TC);
        asm volatile("cp.async.commit_group;" ::: "memory");
        ScanStage<A>& st = stage[(t0 / SS_TC) % SX_STAGES];
        const int nt = min(SS_TC, n_tok - t0);
        // whole chunks ask for no token's place in them
        auto one = [&](auto exactly) {
            if (nt == SS_TC) walk(std::true_type(), exactly, st, t0, nt);
            else walk(std::false_type(), exactly, st, t0, nt);
        };
        if (PASS != 1 && exact) one(std::true_type());
        else one(std::false_type());
    }
    if (PASS == 1) {                           // this piece alone, for the pieces after it
        const size_t at = at0 + piece;
        *reinterpret_cast<float4*>(a.piece_state + (at * a.inner + c) * 16 + 4 * sub) =
            make_float4(sx_lo(S[0]), sx_hi(S[0]), sx_lo(S[1]), sx_hi(S[1]));
        if (sub == 0) a.piece_dt[at * a.inner + c] = dt_sum;
        return;
    }
    if (piece != pieces - 1) return;
    s_slot[0] = sx_lo(S[0]);
    s_slot[1] = sx_hi(S[0]);
    s_slot[2] = sx_lo(S[1]);
    s_slot[3] = sx_hi(S[1]);
    if (sub == 0 && e_tok > 0) {
        // the window of the convolution: the last taps-1 inputs of [old window | this portion]
        for (int j = 0; j < a.taps - 1; ++j) {
            const int at = e_tok + j;
            slot[(size_t)j * a.inner + c] =
                at < a.taps - 1 ? slot[(size_t)at * a.inner + c]
                                : to_float(xz[(size_t)(e_start + at - (a.taps - 1)) * a.ld_xz + c]);
        }
    }
}

// Portions of a few tokens (decode steps): nothing is staged, a lane reads its tokens' numbers itself, two tokens
// at a time, all loads in flight at once; the arithmetic is the kernel's above, number by number.  MAKE: the
// block makes its own step sizes' products, the rows of W_dt of its channels in shared memory, a lane a
// token, summed in the order of the product for many tokens (gemm_f32.cu: even and odd places apart), so that a
// token's bits do not depend on which of the two made them.  Every entry reads W_dt again then, which
// costs less than a launch up to some 32 tokens.  Bound by the stream of the states and by two dependent
// rounds of loads: 20 entries of one token, 4,096 channels and rank 128: 12.9 us (24.8 in the kernel for any state, whose
// lanes read W_dt from global memory), 64: 20.8 (68); 1,024 channels and rank 64: 4.5 (7.9) and 8.6 (16.3).
#define SCAN_FEW 8
#define SCAN_FEW_RANK 256           // rows of W_dt that a block can hold
template <typename A, bool MAKE>
__global__ void __launch_bounds__(128)
selective_scan16_few_kernel(const A* __restrict__ xc, const A* __restrict__ xz, const float* __restrict__ proj,
                            const float* __restrict__ w_dt, const float* __restrict__ dt_bias, const float* __restrict__ a_neg,
                            const float* __restrict__ d_skip, const int* __restrict__ qo_indptr,
                            const int* __restrict__ slots, float* __restrict__ state, A* __restrict__ out, ScanArgs a) {
    constexpr int FEW = 2;
    extern __shared__ __align__(16) float sf_smem[];             // MAKE: [32][rank + 4] of W_dt, [SCAN_FEW][rank]
    const int e = blockIdx.x, sub = threadIdx.x & 3, ch = threadIdx.x >> 2, c = blockIdx.y * 32 + ch;
    const int ld = a.rank + 4, quads = a.rank / 4;
    if (MAKE) {                                                  // (no kernel writes W_dt)
        for (int i = threadIdx.x; i < 32 * quads; i += 128)
            cp_async_16(smem_u32(sf_smem + i / quads * ld + i % quads * 4),
                        w_dt + (size_t)(blockIdx.y * 32 + i / quads) * a.rank + i % quads * 4, 16);
    }
    const unsigned long long waited = pdl_wait();
    xc = pdl_after(xc, waited);
    xz = pdl_after(xz, waited);
    proj = pdl_after(proj, waited);
    const float* dt_pre = pdl_after((const float*)a.dt_pre, waited);
    const int start = qo_indptr[e], n_tok = qo_indptr[e + 1] - start;
    const int row = a.rank + 32;
    float* dt_in = sf_smem + 32 * ld;
    if (MAKE) {
        for (int i = threadIdx.x; i < n_tok * quads; i += 128)
            cp_async_16(smem_u32(dt_in + i * 4), proj + (size_t)(start + i / quads) * row + i % quads * 4, 16);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    if (n_tok <= 0) return;
    float made[SCAN_FEW / 4];                                    // of tokens sub and sub + 4
    if (MAKE) {
#pragma unroll
        for (int m = 0; m < SCAN_FEW / 4; ++m) {
            unsigned long long acc = 0ull;
            if (sub + 4 * m < n_tok) {
                const float* w = sf_smem + ch * ld;
                const float* d = dt_in + (sub + 4 * m) * a.rank;
#pragma unroll 8
                for (int k = 0; k < a.rank; k += 4) {
                    const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(d + k), w2 = *reinterpret_cast<const ulonglong2*>(w + k);
                    acc = sx_fma(x2.x, w2.x, acc);
                    acc = sx_fma(x2.y, w2.y, acc);
                }
            }
            made[m] = sx_lo(acc) + sx_hi(acc);
        }
    }
    float* slot = state + (size_t)slots[e] * a.state_stride;
    float* s_slot = slot + (size_t)(a.taps - 1) * a.inner + (size_t)c * 16 + 4 * sub;
    const float4 an = *reinterpret_cast<const float4*>(a_neg + (size_t)c * 16 + 4 * sub);
    const unsigned long long An[2] = {sx_pack(an.x, an.y), sx_pack(an.z, an.w)};
    const float bias = dt_bias[c], dsk = d_skip[c];
    const bool wide = (reinterpret_cast<uintptr_t>(s_slot) & 15) == 0;
    unsigned long long S[2];
    if (wide) {
        const float4 s4 = *reinterpret_cast<const float4*>(s_slot);
        S[0] = sx_pack(s4.x, s4.y);
        S[1] = sx_pack(s4.z, s4.w);
    } else {
        S[0] = sx_pack(s_slot[0], s_slot[1]);
        S[1] = sx_pack(s_slot[2], s_slot[3]);
    }
    // the window of the convolution: the last taps - 1 inputs of [old window | this portion]
    if (a.taps <= 5) {
        float w = 0.f;
        const int at = n_tok + sub;
        if (sub < a.taps - 1)
            w = at < a.taps - 1 ? slot[(size_t)at * a.inner + c]
                                : to_float(xz[(size_t)(start + at - (a.taps - 1)) * a.ld_xz + c]);
        __syncwarp();
        if (sub < a.taps - 1) slot[(size_t)sub * a.inner + c] = w;
    } else if (sub == 0) {
        for (int j = 0; j < a.taps - 1; ++j) {
            const int at = n_tok + j;
            slot[(size_t)j * a.inner + c] =
                at < a.taps - 1 ? slot[(size_t)at * a.inner + c]
                                : to_float(xz[(size_t)(start + at - (a.taps - 1)) * a.ld_xz + c]);
        }
    }
    for (int t0 = 0; t0 < n_tok; t0 += FEW) {
        float dt[FEW], x[FEW], z[FEW];
        ulonglong2 B[FEW], C[FEW];
#pragma unroll
        for (int k = 0; k < FEW; ++k) {
            const size_t t = (size_t)(start + min(t0 + k, n_tok - 1));
            const float* bc = proj + t * row + a.rank + 4 * sub;
            B[k] = *reinterpret_cast<const ulonglong2*>(bc);
            C[k] = *reinterpret_cast<const ulonglong2*>(bc + 16);
            if (MAKE) {
                const int j = min(t0 + k, n_tok - 1);
                dt[k] = __shfl_sync(0xffffffffu, j < 4 ? made[0] : made[1], j & 3, 4);
            } else {
                dt[k] = dt_pre[t * a.inner + c];
            }
            x[k] = to_float(xc[t * a.inner + c]);
            z[k] = to_float(xz[t * a.ld_xz + a.inner + c]);
        }
#pragma unroll
        for (int k = 0; k < FEW; ++k) {
            if (t0 + k >= n_tok) break;
            const float d = softplus_f(dt[k] + bias), dx = d * x[k];
            const unsigned long long d2 = sx_pack(d, d), dx2 = sx_pack(dx, dx);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned long long p = sx_mul(d2, An[i]);
                S[i] = sx_fma(sx_decays<true>(p), S[i], sx_mul(dx2, i == 0 ? B[k].x : B[k].y));
            }
            const unsigned long long y2 = sx_fma(S[1], C[k].y, sx_mul(S[0], C[k].x));
            float y = sx_lo(y2) + sx_hi(y2);
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            y += __shfl_xor_sync(0xffffffffu, y, 2);
            if (sub == 0)
                out[(size_t)(start + t0 + k) * a.inner + c] = from_float<A>(fmaf(dsk, x[k], y) * sx_silu(z[k], A()));
        }
    }
    if (wide) {
        *reinterpret_cast<float4*>(s_slot) = make_float4(sx_lo(S[0]), sx_hi(S[0]), sx_lo(S[1]), sx_hi(S[1]));
    } else {
        s_slot[0] = sx_lo(S[0]);
        s_slot[1] = sx_hi(S[0]);
        s_slot[2] = sx_lo(S[1]);
        s_slot[3] = sx_hi(S[1]);
    }
}

template <typename A>
static int launch_scan16(const void* xc, const void* xz, const float* proj, const float* w_dt, const float* dt_bias, const float* a_neg,
                          const float* d_skip, const int* qo_indptr, const int* slots, float* state, void* out,
                          ScanArgs a, bool few, cudaStream_t s) {
    const dim3 grid(a.entries, a.inner / 32, a.max_pieces);
    if (few) {
        const bool make = a.dt_pre == nullptr;
        const size_t smem = make ? sizeof(float) * (32 * (a.rank + 4) + SCAN_FEW * a.rank) : 0;
        mstar_launch(make ? selective_scan16_few_kernel<A, true> : selective_scan16_few_kernel<A, false>, grid, dim3(128),
                     smem, s, (const A*)xc, (const A*)xz, proj, w_dt, dt_bias, a_neg, d_skip, qo_indptr, slots, state,
                     (A*)out, a);
        return launch_status();
    }
#define GO(PASS)                                                                                  \
    a.pass = PASS;                                                                                \
    mstar_launch((selective_scan16_kernel<A, PASS>), grid, dim3(128), 0, s, (const A*)xc, (const A*)xz, proj, \
                 dt_bias, a_neg, d_skip, qo_indptr, slots, state, (A*)out, a)
    if (a.piece != 0) {
        GO(1);
        GO(2);
    } else {
        GO(0);
    }
#undef GO
    return launch_status();
}

// xc: [tokens, inner] conv outputs; xz: [tokens] rows of ld_xz elements, x then z; proj: float
// [tokens, rank + 2 n_state]; w_dt float [inner, rank]; a_neg float [inner, n_state] = -exp(A_log);
// out [tokens, inner].  piece > 0: portions are cut into pieces of that many tokens (a multiple
// of the token chunk) that run side by side in two passes; max_pieces bounds the pieces of any
// entry, piece_state is float scratch [entries, max_pieces, inner, n_state], piece_dt
// [entries, max_pieces, inner].  dt_pre: nullptr, or float scratch [dt_tokens, inner], all tokens', for a
// product dt_in W_dt^T of its own (with pieces it may hold step sizes afterwards).  piece < 0, where the kernel for 16 states
// takes the sizes: pieces of scan_piece tokens, max_pieces as with piece > 0, scratch for tokens / 64 +
// entries pieces.  max_tokens: no entry has more (0: not known).  Returns 0, a CUDA error code, or -1 when the shape is refused.
MSTAR_API int mstar_selective_scan(const void* xc, const void* xz, int ld_xz, const float* proj,
                                   const float* w_dt, const float* dt_bias, const float* a_neg,
                                   const float* d_skip, const int* qo_indptr, const int* slots,
                                   float* state, long long state_stride, void* out, int act_dtype,
                                   int entries, int inner, int n_state, int rank, int taps,
                                   int piece, int max_pieces, float* piece_state, float* piece_dt,
                                   float* dt_pre, int dt_tokens, int max_tokens, int* error, void* stream) {
    if (entries <= 0) return 0;
    if (inner <= 0 || n_state <= 0 || rank <= 0 || taps <= 0 || n_state > 256) return -1;
    if (piece != 0 && (max_pieces < 1 || piece_state == nullptr || piece_dt == nullptr)) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    ScanArgs a{inner, n_state, rank, taps, ld_xz, entries, state_stride, piece, 0,
               piece != 0 ? max_pieces : 1, piece_state, piece_dt, dt_pre};
    if (dt_pre != nullptr) {
        const int code = mstar_sgemm_nt(proj, w_dt, dt_pre, dt_tokens, inner, rank, rank + 2 * n_state, rank, inner,
                                        error, stream);
        if (code != 0) return code;
    }
    const int piece16 = act_dtype == MSTAR_F32 ? 4 : 8;          // elements of 16 bytes
    // (without a product of its own the kernel for a few tokens makes it; the row of W_dt must fit)
    const bool few = piece == 0 && max_tokens > 0 && max_tokens <= SCAN_FEW &&
                     (dt_pre != nullptr || (rank <= SCAN_FEW_RANK && ((uintptr_t)w_dt & 15) == 0));
    if ((dt_pre != nullptr || few) && n_state == 16 && inner % 32 == 0 && rank % 4 == 0 && ld_xz % piece16 == 0 &&
        (((uintptr_t)xc | (uintptr_t)xz | (uintptr_t)proj | (uintptr_t)dt_pre | (uintptr_t)a_neg | (uintptr_t)piece_state) & 15) == 0) {
        return act_dtype == MSTAR_F32 ? launch_scan16<float>(xc, xz, proj, w_dt, dt_bias, a_neg, d_skip, qo_indptr, slots,
                                                             state, out, a, few, s)
                                      : launch_scan16<bf16>(xc, xz, proj, w_dt, dt_bias, a_neg, d_skip, qo_indptr, slots,
                                                            state, out, a, few, s);
    }
    if (piece < 0) return -1;
#define GO(A, LANES, NPER)                                                                        \
    {                                                                                             \
        constexpr int CH = SS_THREADS / LANES;                                                    \
        const size_t smem = sizeof(float) * 2 * ((size_t)SS_TC * (rank + 2 * n_state) + 3 * SS_TC * CH); \
        if (smem > 200 * 1024) return -1;                                                         \
        static size_t configured = 0;                                                             \
        if (smem > 48 * 1024 && smem > configured) {                                              \
            cudaFuncSetAttribute(selective_scan_kernel<A, LANES, NPER>,                           \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
            configured = smem;                                                                    \
        }                                                                                         \
        dim3 grid(entries, (inner + CH - 1) / CH, a.max_pieces);                                  \
        for (int pass = (piece > 0 ? 1 : 0); pass <= (piece > 0 ? 2 : 0); ++pass) {               \
            a.pass = pass;                                                                        \
            mstar_launch((selective_scan_kernel<A, LANES, NPER>), grid, dim3(SS_THREADS), smem, s, \
                         (const A*)xc, (const A*)xz, proj, w_dt, dt_bias, a_neg, d_skip,          \
                         qo_indptr, slots, state, (A*)out, a);                                    \
        }                                                                                         \
    }
#define PICK(A)                                                                                   \
    if (n_state <= 4) GO(A, 4, 1)                                                                 \
    else if (n_state <= 16) GO(A, 4, 4)                                                           \
    else if (n_state <= 64) GO(A, 4, 16)                                                          \
    else GO(A, 16, 16)
    if (act_dtype == MSTAR_F32) { PICK(float) } else { PICK(bf16) }
#undef PICK
#undef GO
    return launch_status();
}
