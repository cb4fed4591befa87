// A selective state-space mixer with scalar decay per head, between its input and output projections:
//
//   pb_causal_conv_silu     u = silu(conv(xBC) + bias) per channel over the last `taps` tokens; what lies before the
//                           step's first token comes from the sequence's carried inputs
//   pb_conv_state_update    the last taps - 1 inputs of every sequence, carried to its next step
//   pb_ssm_scan             dt = softplus(dt + bias); S <- exp(-exp(A_log) dt) S + dt B x^T; y = S^T C + D x, token by
//                           token, the state [heads, state, head_dim] float32 per sequence, read at the start and written
//                           at the end of the step
//   pb_decay_scan           the same recurrence with a constant decay per head and no step size: linear attention with a
//                           decaying state, S <- decay S + k v^T; o = S^T q, q, k, v the SiLU of the projection's columns
//   pb_gated_group_rmsnorm  y * silu(z), brought to unit root mean square in equal parts, times a scale; or, with the gate
//                           after the norm, y brought to unit root mean square in equal parts, times a scale, times silu(z)
//
// Decay, step size, softplus, exponentials, the state and the sums over it are float32 whatever the run's type;
// the projections and the convolution's output are of the run's type.  A scan here visits a sequence's tokens in order,
// one after the other, by the same threads.  In 32-bit all results are therefore the same however a prompt was cut into steps and
// whatever else is in the batch.  In bfloat16 the state-space recurrence is not, in the last bits: a prompt step runs it by chunks
// (ssm_chunk.cu), but for sequences of one token, which pb_ssm_step visits; and the gated norm's order of sums follows the number of
// rows.  All kernels find a step's sequences through device arrays (cumulative lengths, state slots): a row whose length is not positive
// is skipped, so the launches have the same shape whatever the step holds and can be recorded.
#include "sequences.cuh"

#include <math.h>

#include <type_traits>

namespace {

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ bool pb_aligned_dev(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
// 16 bytes of a row as floats: 4 of float32, 8 of bfloat16
__device__ __forceinline__ void pb_unpack_vec(const uint4& raw, float (&out)[4]) {
    out[0] = __uint_as_float(raw.x); out[1] = __uint_as_float(raw.y); out[2] = __uint_as_float(raw.z); out[3] = __uint_as_float(raw.w);
}
__device__ __forceinline__ void pb_unpack_vec(const uint4& raw, float (&out)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); out[2 * i] = f.x; out[2 * i + 1] = f.y; }
}
// 8 bytes of a bfloat16 row as floats
__device__ __forceinline__ void pb_unpack_vec(const uint2& raw, float (&out)[4]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 2; ++i) { const float2 f = __bfloat1622float2(h[i]); out[2 * i] = f.x; out[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void pb_st_vec(__nv_bfloat16* p, const float (&v)[4]) {
    uint2 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 2; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint2*>(p) = raw;
}
template <typename T, int VN> __device__ __forceinline__ void pb_ld_vec(const T* p, float (&out)[VN]) { pb_unpack_vec(*reinterpret_cast<const uint4*>(p), out); }
__device__ __forceinline__ void pb_st_vec(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void pb_st_vec(__nv_bfloat16* p, const float (&v)[8]) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}
// ---------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void causal_conv_silu_kernel(const T* in, long long ld_in, const float* w,
                                        const float* bias, const T* carried, T* out,
                                        const int32_t* token_seq, const int32_t* positions,
                                        const int32_t* q_start, const int32_t* slots, int n_tokens,
                                        int channels, int taps, T* advance) {
    pb_grid_dep_launch();
    pb_grid_dep_wait();
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t = blockIdx.x;
    if (c >= channels) return;
    const int seq = token_seq[t];
    if (seq < 0) return;                                   // a padding row
    const int i = positions[t] - q_start[seq];             // the token's index among its sequence's tokens of this step
    const T* old = carried + (size_t)slots[seq] * (taps - 1) * channels;
    float acc = bias ? bias[c] : 0.f;
    for (int j = 0; j < taps; ++j) {
        const int idx = i - (taps - 1 - j);                // in-step index of the input under tap j
        const float x = idx >= 0 ? pb_ld(in + (size_t)(t - (taps - 1 - j)) * ld_in + c)
                                 : pb_ld(old + (size_t)(taps - 1 + idx) * channels + c);
        acc = fmaf(w[(size_t)c * taps + j], x, acc);
    }
    pb_st(out + (size_t)t * channels + c, pb_silu_for<T>(acc));
    if (advance != nullptr) {                              // the sequence's only token: the inputs move on by one
        T* st = advance + (size_t)slots[seq] * (taps - 1) * channels + c;
        for (int j = 0; j + 2 < taps; ++j) st[(size_t)j * channels] = st[(size_t)(j + 1) * channels];
        if (taps > 1) st[(size_t)(taps - 2) * channels] = in[(size_t)t * ld_in + c];
    }
}

// The same, 16 bytes of channels per thread and RUN consecutive tokens (channels, row stride and pointers in multiples of 16
// bytes; TAPS known at compile time; a long step: CONV_RUN tokens a thread, a step of few tokens: one).  A run inside one
// sequence asks for all its rows and the TAPS - 1 before it at once, so a thread waits for memory once; the rows that two
// runs share come from the caches.  (One token after the other with the window kept in registers waited once a token: 2,048
// tokens of 10,240 channels 87 us, 48 in runs, 43 with the one-instruction reciprocal, now 33, with twice the warps and half the registers.)
#define CONV_RUN 8
template <typename T, int TAPS, int RUN>
__global__ void __launch_bounds__(128) causal_conv_silu_vec_kernel(const T* in, long long ld_in, const float* w, const float* bias, const T* carried,
                                                                   T* out, const int32_t* token_seq, const int32_t* positions, const int32_t* q_start,
                                                                   const int32_t* slots, int n_tokens, int channels, T* advance) {
    // a run's thread has 4 channels whatever the type: with 8 it takes 161 registers, and 12 warps a multiprocessor wait for memory
    constexpr int VN = RUN > 1 ? 4 : 16 / sizeof(T);
    using Raw = std::conditional_t<VN * sizeof(T) == 16, uint4, uint2>;
    pb_grid_dep_launch();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * VN;
    if (c >= channels) return;
    float wt[VN][TAPS], bs[VN];
#pragma unroll
    for (int e = 0; e < VN; ++e) {
        bs[e] = bias ? bias[c + e] : 0.f;
        if constexpr (TAPS == 4) {
            const float4 v = *reinterpret_cast<const float4*>(w + (size_t)(c + e) * 4);
            wt[e][0] = v.x; wt[e][1] = v.y; wt[e][2] = v.z; wt[e][3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < TAPS; ++j) wt[e][j] = w[(size_t)(c + e) * TAPS + j];
        }
    }
    pb_grid_dep_wait();
    const int t0 = blockIdx.x * RUN, t_end = min(n_tokens, t0 + RUN);
    // row `idx` (below 0: before the step) of the sequence whose token `t` has in-step index `i`
    auto row = [&](int t, int i, const T* old, int idx) {
        return idx >= 0 ? in + (size_t)(t - i + idx) * ld_in + c : old + (size_t)(TAPS - 1 + idx) * channels + c;
    };
    auto token = [&](int t, const Raw* win) {            // win[j]: the input under tap j
        float acc[VN];
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[e] = bs[e];
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            float x[VN];
            pb_unpack_vec(win[j], x);
#pragma unroll
            for (int e = 0; e < VN; ++e) acc[e] = fmaf(wt[e][j], x[e], acc[e]);
        }
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[e] = pb_silu_for<T>(acc[e]);
        pb_st_vec(out + (size_t)t * channels + c, acc);
    };
    const int seq0 = token_seq[t0];
    if (RUN > 1 && t0 + RUN <= n_tokens && seq0 >= 0 && token_seq[t0 + RUN - 1] == seq0) {
        const int i = positions[t0] - q_start[seq0];
        const T* old = carried + (size_t)slots[seq0] * (TAPS - 1) * channels;
        Raw rows[RUN + TAPS - 1];
#pragma unroll
        for (int j = 0; j < RUN + TAPS - 1; ++j) rows[j] = *reinterpret_cast<const Raw*>(row(t0, i, old, i - (TAPS - 1) + j));
#pragma unroll
        for (int k = 0; k < RUN; ++k) token(t0 + k, rows + k);
        return;
    }
    for (int t = t0; t < t_end; ++t) {                     // a run over the end of a sequence, and a step of few tokens
        const int seq = token_seq[t];
        if (seq < 0) continue;                             // a padding row
        const int i = positions[t] - q_start[seq];
        const T* old = carried + (size_t)slots[seq] * (TAPS - 1) * channels;
        Raw win[TAPS];
#pragma unroll
        for (int j = 0; j < TAPS; ++j) win[j] = *reinterpret_cast<const Raw*>(row(t, i, old, i - (TAPS - 1) + j));
        token(t, win);
        if (RUN == 1 && advance != nullptr) {              // the sequence's only token: the inputs move on by one
#pragma unroll
            for (int j = 1; j < TAPS; ++j) *reinterpret_cast<Raw*>(advance + ((size_t)slots[seq] * (TAPS - 1) + j - 1) * channels + c) = win[j];
        }
    }
}

// Row s of a sequence's carried inputs holds the input at in-step index s - (taps - 1) of its NEXT step.  One thread
// owns a (sequence, channel): it reads rows above the one it writes, in ascending order, so nothing is lost.
template <typename T>
__global__ void conv_state_update_kernel(const T* in, long long ld_in, T* carried,
                                         const int32_t* cu_q, const int32_t* slots, int channels, int taps) {
    pb_grid_dep_launch();
    pb_grid_dep_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (c >= channels) return;
    const int first = cu_q[r], n = cu_q[r + 1] - first;
    if (n <= 0) return;
    T* st = carried + (size_t)slots[r] * (taps - 1) * channels;
    for (int s = 0; s < taps - 1; ++s) {
        const int idx = n - (taps - 1) + s;
        st[(size_t)s * channels + c] = idx >= 0 ? in[(size_t)(first + idx) * ld_in + c] : st[(size_t)(taps - 1 + idx) * channels + c];
    }
}

// ---------------------------------------------------------------------------------------------------------
// The scan.  A block is eight warps on one head's state, 16 columns p of it.  Warps 0-3 compute: 16 columns x 8 lanes
// over the state rows n, a lane keeping NPL rows in registers (rows 4 (8 i + j) .. + 3 for i = 0 .. NPL / 4 - 1, so
// that the lanes of a column read consecutive 16-byte pieces of B and C).  Warps 4-7 load: while the others work on
// one chunk of tokens they put the next chunk's x, B, C (as float32), step size dt = softplus(dt + bias) and decay
// exp(-exp(A_log) dt) into the other half of shared memory, so the recurrence, which visits tokens one after the
// other, never waits for global memory.  Per token: S[n][p] = decay S[n][p] + (dt x[p]) B[n],
// y[p] = sum_n S[n][p] C[n] (own rows in ascending order, then the 8 lanes by three exchanges) + D x[p].
#define SCAN_COLS 16
#define SCAN_LANES 8
#ifndef SCAN_UNROLL
#define SCAN_UNROLL 4
#endif

//
// FIXED: the same recurrence with a decay per head that is a constant of the model and no step size (linear attention
// with a decaying state: S <- decay_h S + k v^T, o = S^T q).  x, B, C are then v, k, q read straight from the
// projection's columns (rows `ld_u` apart) and passed through SiLU by the loaders, in float32; dt is 1, D is 0, and
// `a_log` holds the decays themselves.  With `activate` 0 the columns hold SiLU's values already.
template <typename T, int NPL, bool FIXED>
__global__ void __launch_bounds__(256)
ssm_scan_kernel(const T* u, long long ld_u, const T* dt_in, long long ld_dt, const float* dt_bias,
                const float* a_log, const float* d_skip, float* state,
                float* y, const int32_t* cu_q, const int32_t* slots, int heads, int P,
                int N, int groups, int activate) {
    constexpr int NPAD = NPL * SCAN_LANES;                     // state rows with padding: a power of two
    constexpr int CHUNK = NPL == 32 ? 8 : 16;                  // tokens per chunk
    constexpr int BUF = CHUNK * (2 * NPAD + SCAN_COLS + 2);    // floats per half: B, C, x, dt, decay
    __shared__ __align__(16) float sm[2 * BUF];
    pb_grid_dep_launch();
    const int col_blocks = (P + SCAN_COLS - 1) / SCAN_COLS;
    const int h = blockIdx.x / col_blocks, p_first = (blockIdx.x % col_blocks) * SCAN_COLS;
    const int r = blockIdx.y;
    const int tid = threadIdx.x;
    const bool computes = tid < SCAN_COLS * SCAN_LANES;
    // written by no kernel: before the wait
    const float neg_a = FIXED ? a_log[h] : -expf(a_log[h]), bias = FIXED ? 0.f : dt_bias[h], skip = FIXED ? 0.f : d_skip[h];
    pb_grid_dep_wait();
    const int first = cu_q[r], n_tok = cu_q[r + 1] - first;
    if (n_tok <= 0) return;
    const int inner = heads * P, channels = inner + 2 * groups * N;
    const int g = h / (heads / groups);
    const int n_chunks = (n_tok + CHUNK - 1) / CHUNK;

    // compute threads
    const int colp = tid / SCAN_LANES, j = tid % SCAN_LANES;
    const int p = p_first + colp;
    const bool live = computes && p < P;
    const int pp = p < P ? p : P - 1;                                             // idle columns follow along and store nothing
    float* S = state + (((size_t)slots[r] * heads + h) * N) * P + pp;
    float s[NPL];
    if (computes) {
#pragma unroll
        for (int i = 0; i < NPL; ++i) { const int n = ((i >> 2) * SCAN_LANES + j) * 4 + (i & 3); s[i] = n < N ? S[(size_t)n * P] : 0.f; }
    }
    // load threads
    const int lt = tid - SCAN_COLS * SCAN_LANES;
    constexpr int VN = 16 / sizeof(T);                                            // elements of a 16-byte load
    const bool vec = N % VN == 0 && channels % VN == 0 && inner % VN == 0 && ld_u % VN == 0 && pb_aligned_dev(u, 16);
    // every block of a head's columns activates the head's keys and queries anew; a long step has them activated once,
    // in place, by a kernel ahead of this one (`activate` 0)
    auto act = [activate](float v) { return (FIXED && activate) ? silu_f(v) : v; };
    if (N < NPAD) {                                                               // rows past N are read as zeros by the lanes
        if (!computes)
            for (int idx = lt; idx < 2 * BUF; idx += 128) sm[idx] = 0.f;
        __syncthreads();
    }
    auto load_chunk = [&](int k) {
        float* buf = sm + (k & 1) * BUF;
        const int t0 = k * CHUNK, cnt = min(CHUNK, n_tok - t0);
        const T* rows = u + (size_t)(first + t0) * ld_u;
        // everything a thread fetches for the chunk is asked for before anything is stored: one wait per chunk
        float xv[(CHUNK * SCAN_COLS + 127) / 128];
#pragma unroll
        for (int it = 0; it < (CHUNK * SCAN_COLS + 127) / 128; ++it) {
            const int idx = lt + it * 128;
            const int tt = idx / SCAN_COLS, cc = idx % SCAN_COLS;
            xv[it] = (idx < cnt * SCAN_COLS && p_first + cc < P) ? act(pb_ld(rows + (size_t)tt * ld_u + h * P + p_first + cc)) : 0.f;
        }
        const float dt_raw = (!FIXED && lt < cnt) ? pb_ld(dt_in + (size_t)(first + t0 + lt) * ld_dt + h) : 0.f;
        if (vec) {
            // B and C of a token: 2 N / VN pieces of 16 bytes; four of a thread's loads in flight at a time
            const int per_tok = 2 * (N / VN), total = cnt * per_tok;
            for (int base = lt; base < total; base += 4 * 128) {
                float v[4][VN];
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int idx = base + it * 128;
                    if (idx < total) {
                        const int tt = idx / per_tok, rem = idx - tt * per_tok;
                        pb_ld_vec(rows + (size_t)tt * ld_u + inner + g * N + (rem >= N / VN ? (groups - 1) * N : 0) + rem * VN, v[it]);
                    }
                }
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int idx = base + it * 128;
                    if (idx < total) {
                        const int tt = idx / per_tok, rem = idx - tt * per_tok;
                        const bool is_c = rem >= N / VN;
                        float* dst = buf + (is_c ? CHUNK * NPAD : 0) + tt * NPAD + (is_c ? rem - N / VN : rem) * VN;
#pragma unroll
                        for (int e = 0; e < VN; e += 4)
                            *reinterpret_cast<float4*>(dst + e) = make_float4(act(v[it][e]), act(v[it][e + 1]), act(v[it][e + 2]), act(v[it][e + 3]));
                    }
                }
            }
        } else {
            for (int base = lt; base < cnt * N; base += 4 * 128) {
                float vb[4], vc[4];
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int idx = base + it * 128;
                    if (idx < cnt * N) {
                        const int tt = idx / N, n = idx - tt * N;
                        const T* row = rows + (size_t)tt * ld_u + inner + g * N;
                        vb[it] = act(pb_ld(row + n));
                        vc[it] = act(pb_ld(row + groups * N + n));
                    }
                }
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int idx = base + it * 128;
                    if (idx < cnt * N) {
                        const int tt = idx / N, n = idx - tt * N;
                        buf[tt * NPAD + n] = vb[it];
                        buf[CHUNK * NPAD + tt * NPAD + n] = vc[it];
                    }
                }
            }
        }
#pragma unroll
        for (int it = 0; it < (CHUNK * SCAN_COLS + 127) / 128; ++it) {
            const int idx = lt + it * 128;
            if (idx < cnt * SCAN_COLS) buf[2 * CHUNK * NPAD + idx] = xv[it];
        }
        if (!FIXED && lt < cnt) {
            const float dt = pb_softplus(dt_raw + bias);
            buf[2 * CHUNK * NPAD + CHUNK * SCAN_COLS + lt] = dt;
            buf[2 * CHUNK * NPAD + CHUNK * SCAN_COLS + CHUNK + lt] = expf(neg_a * dt);
        }
    };
    if (!computes) load_chunk(0);
    __syncthreads();
    for (int k = 0; k < n_chunks; ++k) {
        if (!computes) {
            if (k + 1 < n_chunks) load_chunk(k + 1);
        } else {
            const float* buf = sm + (k & 1) * BUF;
            const int t0 = k * CHUNK, cnt = min(CHUNK, n_tok - t0);
            auto token = [&](int tt) {
                const float x = buf[2 * CHUNK * NPAD + tt * SCAN_COLS + colp];
                const float dt = FIXED ? 1.0f : buf[2 * CHUNK * NPAD + CHUNK * SCAN_COLS + tt];
                const float decay = FIXED ? neg_a : buf[2 * CHUNK * NPAD + CHUNK * SCAN_COLS + CHUNK + tt];
                const float dx = FIXED ? x : dt * x;
                const float4* b4 = reinterpret_cast<const float4*>(buf + tt * NPAD) + j;
                const float4* c4 = reinterpret_cast<const float4*>(buf + CHUNK * NPAD + tt * NPAD) + j;
                float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;                   // four sums side by side, added up in a fixed order
#pragma unroll
                for (int i = 0; i < NPL / 4; ++i) {
                    const float4 b = b4[i * SCAN_LANES], c = c4[i * SCAN_LANES];
                    s[4 * i + 0] = fmaf(decay, s[4 * i + 0], dx * b.x); a0 = fmaf(s[4 * i + 0], c.x, a0);
                    s[4 * i + 1] = fmaf(decay, s[4 * i + 1], dx * b.y); a1 = fmaf(s[4 * i + 1], c.y, a1);
                    s[4 * i + 2] = fmaf(decay, s[4 * i + 2], dx * b.z); a2 = fmaf(s[4 * i + 2], c.z, a2);
                    s[4 * i + 3] = fmaf(decay, s[4 * i + 3], dx * b.w); a3 = fmaf(s[4 * i + 3], c.w, a3);
                }
                float acc = (a0 + a1) + (a2 + a3);
                acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                if (live && j == 0) y[(size_t)(first + t0 + tt) * inner + h * P + p] = FIXED ? acc : fmaf(skip, x, acc);
            };
            // a whole chunk is unrolled so that a token's loads from shared memory are under way while the token before
            // it is still being summed over its lanes; the arithmetic and its order are the same either way
            constexpr int UNROLL = SCAN_UNROLL;
            if (cnt == CHUNK) {
#pragma unroll UNROLL
                for (int tt = 0; tt < CHUNK; ++tt) token(tt);
            } else {
                for (int tt = 0; tt < cnt; ++tt) token(tt);
            }
        }
        __syncthreads();
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < NPL; ++i) { const int n = ((i >> 2) * SCAN_LANES + j) * 4 + (i & 3); if (n < N) S[(size_t)n * P] = s[i]; }
    }
}

// One token per sequence (a decode step, or those sequences of any step: `which`) in bfloat16: a block owns a head's state, a thread four columns and every 16th (or so) row of
// it, eight rows' pieces under way at a time; the rows' shares of the output meet in shared memory in their order.  What bounds it is
// the state, read and written once.  (The scan above reads it 16 bytes of a row at a time, and makes ready for a chunk of
// sixteen tokens: 2 sequences, 128 heads of 128 x 64, 16.3 us, here 6.7.)  Beside a prompt portion it takes the sequences of one token:
// 60 of them and a portion of 64, 64 heads of 128 x 64, 68 us against 211 by chunks and 193 token by token.
#define SSM_STEP_THREADS 256
#define SSM_STEP_ROWS 8
// RECORDED as in delta_rule.cu.
template <bool RECORDED>
__global__ void __launch_bounds__(SSM_STEP_THREADS)
ssm_step_kernel(const __nv_bfloat16* u, const __nv_bfloat16* dt_in, long long ld_dt, const float* dt_bias, const float* a_log, const float* d_skip,
                float* state, float* y, const int32_t* cu_q, const int32_t* slots, PbSequences which, int heads, int P, int N, int groups) {
    __shared__ __align__(16) float part[SSM_STEP_THREADS * 4];
    pb_grid_dep_launch();
    const int h = blockIdx.x, tid = threadIdx.x;
    const float neg_a = -expf(a_log[h]), bias = dt_bias[h], skip = d_skip[h];     // written by no kernel: before the wait
    const int cg = P >> 2, rg = SSM_STEP_THREADS / cg, c = tid % cg, row0 = tid / cg;
    pb_grid_dep_wait();
    auto work = [&](int r, int) {
        const int t = cu_q[r];
        const int inner = heads * P, g = h / (heads / groups);
        const __nv_bfloat16* row = u + (size_t)t * (inner + 2 * groups * N);
        float4* S = reinterpret_cast<float4*>(state + ((size_t)slots[r] * heads + h) * N * (size_t)P) + c;
        const bool works = row0 < rg;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (works) {
            const uint2 xr = *reinterpret_cast<const uint2*>(row + h * P + 4 * c);
            const float dt = pb_softplus(pb_ld(dt_in + (size_t)t * ld_dt + h) + bias), decay = expf(neg_a * dt);
            const float2 x0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xr.x)), x1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xr.y));
            const float4 dx = make_float4(dt * x0.x, dt * x0.y, dt * x1.x, dt * x1.y);
            const __nv_bfloat16* B = row + inner + g * N;
            const __nv_bfloat16* C = B + groups * N;
            for (int n0 = row0; n0 < N; n0 += rg * SSM_STEP_ROWS) {
                float4 s[SSM_STEP_ROWS];
                float b[SSM_STEP_ROWS], cc[SSM_STEP_ROWS];
#pragma unroll
                for (int i = 0; i < SSM_STEP_ROWS; ++i) {
                    const int n = min(n0 + i * rg, N - 1);
                    s[i] = S[(size_t)n * cg];
                    b[i] = pb_ld(B + n);
                    cc[i] = pb_ld(C + n);
                }
#pragma unroll
                for (int i = 0; i < SSM_STEP_ROWS; ++i) {
                    const int n = n0 + i * rg;
                    if (n < N) {
                        s[i] = make_float4(fmaf(decay, s[i].x, dx.x * b[i]), fmaf(decay, s[i].y, dx.y * b[i]), fmaf(decay, s[i].z, dx.z * b[i]), fmaf(decay, s[i].w, dx.w * b[i]));
                        S[(size_t)n * cg] = s[i];
                        acc.x = fmaf(s[i].x, cc[i], acc.x); acc.y = fmaf(s[i].y, cc[i], acc.y);
                        acc.z = fmaf(s[i].z, cc[i], acc.z); acc.w = fmaf(s[i].w, cc[i], acc.w);
                    }
                }
            }
            if (row0 == 0) {
                acc.x = fmaf(skip, x0.x, acc.x); acc.y = fmaf(skip, x0.y, acc.y); acc.z = fmaf(skip, x1.x, acc.z); acc.w = fmaf(skip, x1.y, acc.w);
            }
            *reinterpret_cast<float4*>(part + tid * 4) = acc;
        }
        __syncthreads();
        if (tid < P) {
            float v = part[tid];
            for (int k = 1; k < rg; ++k) v += part[k * P + tid];
            y[(size_t)t * inner + h * P + tid] = v;
        }
    };
    if constexpr (RECORDED) {
        pb_for_sequences<true>(cu_q, which, work);
    } else {
        const int n_tok = cu_q[blockIdx.y + 1] - cu_q[blockIdx.y];
        if (n_tok > 0 && n_tok < which.below) work(blockIdx.y, 0);
    }
}

// ---------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void gated_group_rmsnorm_kernel(const float* y, const T* z, long long ld_z,
                                           const float* w, T* out, int inner, int parts, float eps,
                                           int gate_after, int sigmoid_gate) {
    pb_grid_dep_launch();
    pb_grid_dep_wait();
    __shared__ float red[32];
    const int t = blockIdx.x, part = blockIdx.y, width = inner / parts;
    const float* yr = y + (size_t)t * inner + (size_t)part * width;
    const T* zr = z + (size_t)t * ld_z + (size_t)part * width;
    float ss = 0.f;
    auto gate = [&](float z) { return sigmoid_gate ? pb_sigmoid_for<T>(z) : pb_silu_for<T>(z); };
    for (int i = threadIdx.x; i < width; i += blockDim.x) { const float v = gate_after ? yr[i] : yr[i] * gate(pb_ld(zr + i)); ss += v * v; }
    ss = pb_warp_sum(ss);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < nwarp; ++i) total += red[i];
    const float inv = 1.0f / sqrtf(total / (float)width + eps);
    T* o = out + (size_t)t * inner + (size_t)part * width;
    for (int i = threadIdx.x; i < width; i += blockDim.x)
        pb_st(o + i, yr[i] * gate(pb_ld(zr + i)) * inv * w[(size_t)part * width + i]);   // the same product either way
}

// The same for parts of up to 128 * ITERS * WARPS elements: WARPS warps per (token, part), four elements per access, the whole part asked
// for at once and kept in registers between the sum and the store; the scales, which all tokens share, come from the caches when they
// are needed.  width, ld_z in multiples of 4, operands aligned, fewer than 2^31 parts.  What bounds it is how much is under way: parts of
// 1,024, 2,048 x 8,192, 80 us on the kernel above, which reads a part twice, an element an access, 33 with a warp a part (80 registers), 29 with
// two.  (Four parts of 128 a warp: 32 us for 21.)
template <typename T, int ITERS, int WARPS>
__global__ void __launch_bounds__(256) gated_part_rmsnorm_kernel(const float* y, const T* z, long long ld_z, const float* w, T* out, int n_tokens,
                                                                 int inner, int parts, float eps, int gate_after, int sigmoid_gate) {
    pb_grid_dep_launch();
    __shared__ float red[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, width = inner / parts, side = warp % WARPS;
    const unsigned item = (blockIdx.x * (blockDim.x >> 5) + warp) / WARPS;
    const bool live = item < (unsigned)n_tokens * (unsigned)parts;
    const unsigned t = live ? item / (unsigned)parts : 0u, part = live ? item - t * (unsigned)parts : 0u;
    const float* yr = y + (size_t)t * inner + (size_t)part * width;
    const T* zr = z + (size_t)t * ld_z + (size_t)part * width;
    float4 yv[ITERS];
    uint2 zv[ITERS];
    float4 zf[sizeof(T) == 4 ? ITERS : 1];
    pb_grid_dep_wait();
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int c = (lane + 32 * (side + WARPS * i)) * 4;
        yv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        zv[i] = make_uint2(0, 0);
        if constexpr (sizeof(T) == 4) zf[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < width && live) {
            yv[i] = *reinterpret_cast<const float4*>(yr + c);
            if constexpr (sizeof(T) == 2) zv[i] = *reinterpret_cast<const uint2*>(zr + c);
            else zf[i] = *reinterpret_cast<const float4*>(zr + c);
        }
    }
    auto gate = [&](float v) { return sigmoid_gate ? pb_sigmoid_for<T>(v) : pb_silu_for<T>(v); };
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        float4 g;
        if constexpr (sizeof(T) == 2) {
            const __nv_bfloat162* hh = reinterpret_cast<const __nv_bfloat162*>(&zv[i]);
            const float2 a = __bfloat1622float2(hh[0]), b = __bfloat1622float2(hh[1]);
            g = make_float4(a.x, a.y, b.x, b.y);
        } else {
            g = zf[i];
        }
        const float4 v = make_float4(yv[i].x * gate(g.x), yv[i].y * gate(g.y), yv[i].z * gate(g.z), yv[i].w * gate(g.w));
        const float4 n = gate_after ? yv[i] : v;
        ss += n.x * n.x + n.y * n.y + n.z * n.z + n.w * n.w;
        yv[i] = v;                                             // the same product either way
    }
    ss = pb_warp_sum(ss);
    if constexpr (WARPS == 2) {
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        ss = red[warp & ~1] + red[warp | 1];
    }
    if (!live) return;
    const float inv = 1.0f / sqrtf(ss / (float)width + eps);
    T* o = out + (size_t)t * inner + (size_t)part * width;
    const float* wr = w + (size_t)part * width;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int c = (lane + 32 * (side + WARPS * i)) * 4;
        if (c < width) {
            const float4 wv = *reinterpret_cast<const float4*>(wr + c);
            const float r[4] = {yv[i].x * inv * wv.x, yv[i].y * inv * wv.y, yv[i].z * inv * wv.z, yv[i].w * inv * wv.w};
            pb_st_vec(o + c, r);
        }
    }
}

// The same for parts of up to 4,096 elements: a block per (token, part), a thread four elements, asked for once (2 tokens of 8 parts of
// 1,024: 3.4 us against 7.8 for the kernel that reads them twice, an element an access).
template <typename T>
__global__ void gated_block_rmsnorm_kernel(const float* y, const T* z, long long ld_z, const float* w, T* out, int inner, int parts, float eps,
                                           int gate_after, int sigmoid_gate) {
    pb_grid_dep_launch();
    __shared__ float red[32];
    const int t = blockIdx.x, part = blockIdx.y, width = inner / parts, c = threadIdx.x * 4;
    const bool live = c < width;
    float4 wv = make_float4(0.f, 0.f, 0.f, 0.f), yv = wv, gv = wv;
    if (live) wv = *reinterpret_cast<const float4*>(w + (size_t)part * width + c);       // written by no kernel: before the wait
    pb_grid_dep_wait();
    if (live) {
        yv = *reinterpret_cast<const float4*>(y + (size_t)t * inner + (size_t)part * width + c);
        const T* zr = z + (size_t)t * ld_z + (size_t)part * width + c;
        if constexpr (sizeof(T) == 2) {
            const uint2 raw = *reinterpret_cast<const uint2*>(zr);
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
            gv = make_float4(a.x, a.y, b.x, b.y);
        } else {
            gv = *reinterpret_cast<const float4*>(zr);
        }
    }
    auto gate = [&](float v) { return sigmoid_gate ? pb_sigmoid_for<T>(v) : pb_silu_for<T>(v); };
    const float4 v = make_float4(yv.x * gate(gv.x), yv.y * gate(gv.y), yv.z * gate(gv.z), yv.w * gate(gv.w));
    const float4 n = gate_after ? yv : v;
    const float ss = pb_warp_sum(n.x * n.x + n.y * n.y + n.z * n.z + n.w * n.w);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < nwarp; ++i) total += red[i];
    const float inv = 1.0f / sqrtf(total / (float)width + eps);
    if (live) {
        T* o = out + (size_t)t * inner + (size_t)part * width + c;
        pb_st(o, v.x * inv * wv.x);
        pb_st(o + 1, v.y * inv * wv.y);
        pb_st(o + 2, v.z * inv * wv.z);
        pb_st(o + 3, v.w * inv * wv.w);
    }
}

template <typename TI, typename TO>
__global__ void scaled_sum_kernel(const TI* a, float sa, const TI* b, float sb, TO* out, long long n) {
    pb_grid_dep_launch();
    pb_grid_dep_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pb_st(out + i, sa * pb_ld(a + i) + sb * pb_ld(b + i));
}

}  // namespace

// in: the step's [x | B | C] columns of the input projection, [n_tokens, channels] with row stride ld_in; w float32
// [channels, taps] (last column: the current token); carried [slots, taps - 1, channels]; out [n_tokens, channels] dense.
// `advance`: every sequence has one token in this step, and the carried inputs are moved on as pb_conv_state_update would (the
// thread that reads a sequence's inputs of a channel is then the only one that does: one launch less in a decode step).
PB_API int pb_causal_conv_silu(const void* in, long long ld_in, const float* w, const float* bias, void* carried, void* out, int advance,
                               int dtype, const int32_t* token_seq, const int32_t* positions, const int32_t* q_start,
                               const int32_t* slots, int n_tokens, int channels, int taps, cudaStream_t stream) {
    PB_REQUIRE(n_tokens >= 0 && channels > 0 && taps >= 1 && ld_in >= channels, "causal_conv_silu: bad sizes");
    PB_REQUIRE(in && w && out && token_seq && positions && q_start && slots && (taps == 1 || carried), "causal_conv_silu: null pointer");
    if (n_tokens == 0) return 0;
    PB_REQUIRE((channels + 127) / 128 < 65536, "causal_conv_silu: %d channels in one launch", channels);
    const int vn = dtype == PB_BF16 ? 8 : 4;
    if (taps >= 2 && taps <= 4 && channels % vn == 0 && ld_in % vn == 0 && pb_aligned(in, 16) && pb_aligned(out, 16) && pb_aligned(carried, 16) &&
        (taps != 4 || pb_aligned(w, 16))) {
        // up to 64 tokens a thread has one: a run's threads would leave most of the chip idle
        const int run = n_tokens <= 64 || advance ? 1 : CONV_RUN, threads = run == 1 ? 64 : 128;
        const dim3 grid((n_tokens + run - 1) / run, (channels / (run == 1 ? vn : 4) + threads - 1) / threads);
#define CONV_LAUNCH(TAPS, RUN)                                                                                                \
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(causal_conv_silu_vec_kernel<T, TAPS, RUN>, grid, dim3(threads), 0, stream, (const T*)in, ld_in, w, bias, \
                                           (const T*)carried, (T*)out, token_seq, positions, q_start, slots, n_tokens, channels, advance ? (T*)carried : (T*)nullptr)))
        if (taps == 2) { if (run == 1) CONV_LAUNCH(2, 1); else CONV_LAUNCH(2, CONV_RUN); }
        else if (taps == 3) { if (run == 1) CONV_LAUNCH(3, 1); else CONV_LAUNCH(3, CONV_RUN); }
        else { if (run == 1) CONV_LAUNCH(4, 1); else CONV_LAUNCH(4, CONV_RUN); }
#undef CONV_LAUNCH
        PB_CHECK_LAUNCH("causal_conv_silu");
        return 0;
    }
    PB_DISPATCH_DTYPE(dtype, T,
        (pb_launch(causal_conv_silu_kernel<T>, dim3(n_tokens, (channels + 127) / 128), dim3(128), 0, stream, (const T*)in, ld_in, w, bias,
                   (const T*)carried, (T*)out, token_seq, positions, q_start, slots, n_tokens, channels, taps, advance ? (T*)carried : (T*)nullptr)));
    PB_CHECK_LAUNCH("causal_conv_silu");
    return 0;
}

// cu_q [n_seqs + 1], slots [n_seqs]: a sequence whose length cu_q[r + 1] - cu_q[r] is not positive is skipped.
PB_API int pb_conv_state_update(const void* in, long long ld_in, void* carried, int dtype, const int32_t* cu_q, const int32_t* slots,
                                int n_seqs, int channels, int taps, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && channels > 0 && taps >= 1 && ld_in >= channels, "conv_state_update: bad sizes");
    if (n_seqs == 0 || taps == 1) return 0;
    PB_REQUIRE(in && carried && cu_q && slots, "conv_state_update: null pointer");
    PB_REQUIRE(n_seqs < 65536, "conv_state_update: %d sequences in one launch", n_seqs);
    PB_DISPATCH_DTYPE(dtype, T,
        (pb_launch(conv_state_update_kernel<T>, dim3((channels + 127) / 128, n_seqs), dim3(128), 0, stream, (const T*)in, ld_in,
                   (T*)carried, cu_q, slots, channels, taps)));
    PB_CHECK_LAUNCH("conv_state_update");
    return 0;
}

// u: the convolution's output [n_tokens, heads * P + 2 * groups * N] dense, laid out [x | B | C]; dt_in: the step-size
// columns of the input projection, row stride ld_dt; state float32 [slots, heads, N, P]; y float32 [n_tokens, heads * P].
PB_API int pb_ssm_scan(const void* u, const void* dt_in, long long ld_dt, int dtype, const float* dt_bias, const float* a_log,
                       const float* d_skip, float* state, float* y, const int32_t* cu_q, const int32_t* slots, int n_seqs,
                       int heads, int P, int N, int groups, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && heads > 0 && P > 0 && N > 0 && groups > 0 && heads % groups == 0, "ssm_scan: bad sizes");
    PB_REQUIRE(N <= 32 * SCAN_LANES, "ssm_scan: a state of %d rows (at most %d)", N, 32 * SCAN_LANES);
    PB_REQUIRE(u && dt_in && dt_bias && a_log && d_skip && state && y && cu_q && slots && ld_dt >= heads, "ssm_scan: null pointer");
    if (n_seqs == 0) return 0;
    PB_REQUIRE(n_seqs < 65536, "ssm_scan: %d sequences in one launch", n_seqs);
    const int col_blocks = (P + SCAN_COLS - 1) / SCAN_COLS;
    const dim3 grid(heads * col_blocks, n_seqs), block(2 * SCAN_COLS * SCAN_LANES);
    const int npl = (N + SCAN_LANES - 1) / SCAN_LANES;
#define SCAN_LAUNCH(NPL)                                                                                                    \
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(ssm_scan_kernel<T, NPL, false>, grid, block, 0, stream, (const T*)u,               \
                                           (long long)(heads * P + 2 * groups * N), (const T*)dt_in, ld_dt, dt_bias, a_log, d_skip,  \
                                           state, y, cu_q, slots, heads, P, N, groups, 0)))
    if (npl <= 4) SCAN_LAUNCH(4);
    else if (npl <= 8) SCAN_LAUNCH(8);
    else if (npl <= 16) SCAN_LAUNCH(16);
    else SCAN_LAUNCH(32);
#undef SCAN_LAUNCH
    PB_CHECK_LAUNCH("ssm_scan");
    return 0;
}

// The same for a step of one token per sequence, bfloat16: whether it takes the sizes, and the call.  `single`: a step of any lengths, of
// which only the sequences of one token are visited; n_short: how many there are (`counted`), or the most there can be, for a step that is
// being recorded (few, beside: sequences.cuh).
PB_API int pb_ssm_step_takes(const void* u, const float* state, int heads, int P, int N, int groups) {
    return heads > 0 && groups > 0 && heads % groups == 0 && P >= 4 && P % 4 == 0 && P <= SSM_STEP_THREADS && N > 0 && (heads * P + 2 * groups * N) % 4 == 0 &&
                   pb_aligned(u, 8) && pb_aligned(state, 16)
               ? 1
               : 0;
}
PB_API int pb_ssm_step(const void* u, const void* dt_in, long long ld_dt, const float* dt_bias, const float* a_log, const float* d_skip, float* state, float* y,
                       const int32_t* cu_q, const int32_t* slots, int n_seqs, int heads, int P, int N, int groups, int single, int few, int beside, int n_short, int counted,
                       cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && pb_ssm_step_takes(u, state, heads, P, N, groups), "ssm_step: %d heads of %d, state %d, %d groups", heads, P, N, groups);
    PB_REQUIRE(u && dt_in && dt_bias && a_log && d_skip && state && y && cu_q && slots && ld_dt >= heads, "ssm_step: null pointer");
    if (n_seqs == 0) return 0;
    PB_REQUIRE(n_seqs < 65536, "ssm_step: %d sequences in one launch", n_seqs);
    if (single && n_short <= 0) return 0;
    const int recorded = single && !counted;
    const PbSequences which{n_seqs, 1, single ? 2 : INT_MAX, few, beside, 0, recorded, 0, 0};
    const dim3 grid(heads, recorded ? pb_recorded_rows(n_short, heads, 8) : n_seqs);
#define STEP_LAUNCH(R)                                                                                                             \
    pb_launch(ssm_step_kernel<R>, grid, dim3(SSM_STEP_THREADS), 0, stream, (const __nv_bfloat16*)u, (const __nv_bfloat16*)dt_in, ld_dt, dt_bias, a_log, \
              d_skip, state, y, cu_q, slots, which, heads, P, N, groups)
    if (recorded) STEP_LAUNCH(true);
    else STEP_LAUNCH(false);
#undef STEP_LAUNCH
    PB_CHECK_LAUNCH("ssm_step");
    return 0;
}

// Linear attention with a decaying state: per head S <- decay_h S + k v^T, o = S^T q, with q, k, v the SiLU of the
// projection's columns.  u: the projection, rows ld_u apart, laid out [v: heads * P | k: heads * N | q: heads * N];
// decay float32 [heads]; state float32 [slots, heads, N, P]; y float32 [n_tokens, heads * P].  activated: the columns
// hold silu(v), silu(k), silu(q) already (pb_silu_cols), the scan takes them as they are.
PB_API int pb_decay_scan(const void* u, long long ld_u, int dtype, const float* decay, float* state, float* y, const int32_t* cu_q,
                         const int32_t* slots, int n_seqs, int heads, int P, int N, int activated, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && heads > 0 && P > 0 && N > 0 && ld_u >= (long long)heads * (P + 2 * N), "decay_scan: bad sizes");
    PB_REQUIRE(N <= 32 * SCAN_LANES, "decay_scan: keys of %d elements (at most %d)", N, 32 * SCAN_LANES);
    PB_REQUIRE(u && decay && state && y && cu_q && slots, "decay_scan: null pointer");
    if (n_seqs == 0) return 0;
    PB_REQUIRE(n_seqs < 65536, "decay_scan: %d sequences in one launch", n_seqs);
    const int col_blocks = (P + SCAN_COLS - 1) / SCAN_COLS;
    const dim3 grid(heads * col_blocks, n_seqs), block(2 * SCAN_COLS * SCAN_LANES);
    const int npl = (N + SCAN_LANES - 1) / SCAN_LANES;
#define SCAN_LAUNCH(NPL)                                                                                                    \
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(ssm_scan_kernel<T, NPL, true>, grid, block, 0, stream, (const T*)u, ld_u, (const T*)nullptr, \
                                           0ll, (const float*)nullptr, decay, (const float*)nullptr, state, y, cu_q, slots, heads, P, \
                                           N, heads, activated ? 0 : 1)))
    if (npl <= 4) SCAN_LAUNCH(4);
    else if (npl <= 8) SCAN_LAUNCH(8);
    else if (npl <= 16) SCAN_LAUNCH(16);
    else SCAN_LAUNCH(32);
#undef SCAN_LAUNCH
    PB_CHECK_LAUNCH("decay_scan");
    return 0;
}

// y float32 [n_tokens, inner]; z: the gate columns of the input projection, row stride ld_z; w float32 [inner];
// out [n_tokens, inner] dense.  gate_after 0: norm(y * gate(z)) * w; 1: norm(y) * w * gate(z); gate is SiLU, or the
// sigmoid with sigmoid_gate.
PB_API int pb_gated_group_rmsnorm(const float* y, const void* z, long long ld_z, const float* w, void* out, int dtype, int n_tokens,
                                  int inner, int parts, float eps, int gate_after, int sigmoid_gate, cudaStream_t stream) {
    PB_REQUIRE(n_tokens >= 0 && inner > 0 && parts > 0 && inner % parts == 0 && ld_z >= inner, "gated_group_rmsnorm: bad sizes");
    PB_REQUIRE(y && z && w && out, "gated_group_rmsnorm: null pointer");
    if (n_tokens == 0) return 0;
    PB_REQUIRE(parts < 65536, "gated_group_rmsnorm: %d parts", parts);
    const int width = inner / parts;
    const size_t esz = dtype == PB_BF16 ? 2 : 4;
    // parts of up to 1,024 in bfloat16 too where there are rows enough that a warp each fills the chip (2 x 8,192: 13 us against 11
    // for a block each); in 32-bit a row's sum keeps one order whatever the step holds
    // (its places are counted in 32 bits: 2^31 and more go to the kernels below)
    const long long items = (long long)n_tokens * parts, units = items * (width > 512 ? 2 : 1);
    if ((width <= 512 || (width <= 1024 && dtype == PB_BF16 && items >= 4096)) && units < (1ll << 31) && width % 4 == 0 && ld_z % 4 == 0 && pb_aligned(y, 16) && pb_aligned(w, 16) && pb_aligned(z, 4 * esz) && pb_aligned(out, 4 * esz)) {
        const int warps = items >= 4096 ? 8 : 1;
        const dim3 grid((unsigned)((units + warps - 1) / warps)), block(32 * warps);
#define PART_LAUNCH(IT, WARPS)                                                                                                \
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(gated_part_rmsnorm_kernel<T, IT, WARPS>, grid, block, 0, stream, y, (const T*)z, ld_z, w, (T*)out, n_tokens, inner, \
                                           parts, eps, gate_after, sigmoid_gate)))
        if (width <= 128) PART_LAUNCH(1, 1);
        else if (width <= 256) PART_LAUNCH(2, 1);
        else if (width <= 512) PART_LAUNCH(4, 1);
        else PART_LAUNCH(4, 2);
#undef PART_LAUNCH
        PB_CHECK_LAUNCH("gated_group_rmsnorm");
        return 0;
    }
    if (width <= 4096 && width % 4 == 0 && ld_z % 4 == 0 && pb_aligned(y, 16) && pb_aligned(w, 16) && pb_aligned(z, 4 * esz) && pb_aligned(out, 4 * esz)) {
        const int block = (width / 4 + 31) / 32 * 32;
        PB_DISPATCH_DTYPE(dtype, T, (pb_launch(gated_block_rmsnorm_kernel<T>, dim3(n_tokens, parts), dim3(block), 0, stream, y, (const T*)z, ld_z, w, (T*)out, inner,
                                               parts, eps, gate_after, sigmoid_gate)));
        PB_CHECK_LAUNCH("gated_group_rmsnorm");
        return 0;
    }
    int threads = 32;
    while (threads < 256 && threads < inner / parts) threads <<= 1;
    PB_DISPATCH_DTYPE(dtype, T,
        (pb_launch(gated_group_rmsnorm_kernel<T>, dim3(n_tokens, parts), dim3(threads), 0, stream, y, (const T*)z, ld_z, w, (T*)out, inner,
                   parts, eps, gate_after, sigmoid_gate)));
    PB_CHECK_LAUNCH("gated_group_rmsnorm");
    return 0;
}

// out = sa * a + sb * b, element by element in float32; a and b of type in_dtype, out of out_dtype.
PB_API int pb_scaled_sum(const void* a, float sa, const void* b, float sb, void* out, int in_dtype, int out_dtype, long long n,
                         cudaStream_t stream) {
    PB_REQUIRE(n >= 0 && a && b && out, "scaled_sum: bad arguments");
    if (n == 0) return 0;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (in_dtype == PB_F32 && out_dtype == PB_F32)
        pb_launch(scaled_sum_kernel<float, float>, dim3(blocks), dim3(256), 0, stream, (const float*)a, sa, (const float*)b, sb, (float*)out, n);
    else if (in_dtype == PB_F32 && out_dtype == PB_BF16)
        pb_launch(scaled_sum_kernel<float, __nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (const float*)a, sa, (const float*)b, sb,
                  (__nv_bfloat16*)out, n);
    else if (in_dtype == PB_BF16 && out_dtype == PB_BF16)
        pb_launch(scaled_sum_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (const __nv_bfloat16*)a, sa,
                  (const __nv_bfloat16*)b, sb, (__nv_bfloat16*)out, n);
    else
        return pb_fail("scaled_sum: unsupported types in=%d out=%d", in_dtype, out_dtype);
    PB_CHECK_LAUNCH("scaled_sum");
    return 0;
}
