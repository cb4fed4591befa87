// Linear attention with a matrix state per head and a decay per key channel that every token makes anew:
//
//   a = sigmoid(z)^(1/tau),  z = W2 x1 + b           x1 the narrow projection of the token, W2 [heads * N, rank]
//   S <- diag(a) S + k v^T ;  o = scale * S^T q      per head, S [N (key channel), P (value)] float32 per sequence
//
//   pb_channel_decay    the decays of a step's tokens, float32 [tokens, heads * N]
//   pb_gla_scan         the recurrence over a step's tokens, sequence by sequence; o float32 [tokens, heads * P]
//   pb_gla_step         one token per sequence (a decode step): decay, recurrence, norm per head and gate in one kernel
//
// Decays and their logarithms, the state and every sum over it are float32 whatever the run's type; q, k, v and x1
// (projections) are of the run's type.  A sequence's tokens are visited in order; a token's numbers do not depend here on how a
// prompt was cut into steps or on what else is in the batch.  Sequences are found through device arrays (cumulative
// lengths, state slots), one block row per sequence the arrays have room for: a row whose length is not positive is
// skipped, so the launches can be recorded.  (A prompt step in bfloat16 runs the recurrence by sixteen tokens,
// which changes the last bits: gla_chunk.cu.)
#include "common.cuh"

#include <math.h>

namespace {

typedef unsigned long long u64;

// two float32 in one register pair: one instruction for two multiply-adds
__device__ __forceinline__ u64 pk2(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 up2(u64 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// 16 bytes of a row as floats
__device__ __forceinline__ void gla_unpack(const uint4& raw, float (&o)[4]) {
    o[0] = __uint_as_float(raw.x); o[1] = __uint_as_float(raw.y); o[2] = __uint_as_float(raw.z); o[3] = __uint_as_float(raw.w);
}
__device__ __forceinline__ void gla_unpack(const uint4& raw, float (&o)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
}

// sigmoid(z)^(1/tau) = exp(-softplus(-z) / tau)
__device__ __forceinline__ float gla_decay(float z, float inv_tau) {
    const float softplus = fmaxf(-z, 0.f) + log1pf(expf(-fabsf(z)));
    return expf(-softplus * inv_tau);
}

// ---------------------------------------------------------------------------------------------------------
// For ranks in multiples of 8 up to 64 in bfloat16: a thread owns one channel, its row of the matrix in registers (two for a number: more of
// them do not fit), and walks the block's tokens eight at a time, two in one instruction; their narrow rows lie in shared memory turned, so
// that one access brings four tokens.  Sums over the rank in ascending order, as below, and the same bits.  (2,048 tokens of 4,096 channels:
// rank 32 56 us below, where a block has eight tokens and every block fetches the rows of the matrix for them alone, 31 here; rank 64 157
// and 59; rank 8 25 and 19.)
template <int RANK>
__global__ void __launch_bounds__(128) channel_decay_rows_kernel(const __nv_bfloat16* x1, long long ld_x1, const __nv_bfloat16* w2, const float* bias,
                                                                 float inv_tau, float* out, int n_tokens, int channels, int block_tokens) {
    extern __shared__ __align__(16) float xs[];                // [RANK][block_tokens + 4]
    pb_grid_dep_launch();
    const int c = blockIdx.y * blockDim.x + threadIdx.x, ld = block_tokens + 4;
    const int t0 = blockIdx.x * block_tokens, cnt = min(block_tokens, n_tokens - t0);
    const int cc = min(c, channels - 1);
    const float b = bias[cc];                                  // matrix and bias are written by no kernel: before the wait
    u64 w[RANK];
#pragma unroll
    for (int r = 0; r < RANK; r += 8) {
        float f[8];
        gla_unpack(*reinterpret_cast<const uint4*>(w2 + (size_t)cc * RANK + r), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[r + e] = pk2(f[e], f[e]);
    }
    pb_grid_dep_wait();
    for (int i = threadIdx.x; i < block_tokens * (RANK / 8); i += blockDim.x) {
        const int u = i / (RANK / 8), r = i % (RANK / 8) * 8;
        float f[8];
        gla_unpack(u < cnt ? *reinterpret_cast<const uint4*>(x1 + (size_t)(t0 + u) * ld_x1 + r) : make_uint4(0, 0, 0, 0), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) xs[(r + e) * ld + u] = f[e];
    }
    __syncthreads();
    if (c >= channels) return;
#pragma unroll 1
    for (int u0 = 0; u0 < cnt; u0 += 8) {
        u64 acc[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[p] = pk2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < RANK; ++r) {
            const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(xs + r * ld + u0), hi = *reinterpret_cast<const ulonglong2*>(xs + r * ld + u0 + 4);
            acc[0] = fma2(lo.x, w[r], acc[0]);
            acc[1] = fma2(lo.y, w[r], acc[1]);
            acc[2] = fma2(hi.x, w[r], acc[2]);
            acc[3] = fma2(hi.y, w[r], acc[3]);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float2 z = up2(acc[p]);
            float* o = out + (size_t)(t0 + u0 + 2 * p) * channels + c;
            const float d0 = gla_decay(z.x + b, inv_tau), d1 = gla_decay(z.y + b, inv_tau);
            if (u0 + 2 * p < cnt) o[0] = d0;
            if (u0 + 2 * p + 1 < cnt) o[channels] = d1;
        }
    }
}

// A thread owns one channel and DECAY_TOKENS tokens, whose narrow rows the block keeps in shared memory as float32; the sum
// over the rank runs in ascending order (as in gla_step_kernel).
#define DECAY_TOKENS 8
template <typename T>
__global__ void __launch_bounds__(128) channel_decay_kernel(const T* x1, long long ld_x1, const T* w2,
                                                            const float* bias, float inv_tau, float* out, int n_tokens,
                                                            int channels, int rank, int vec) {
    extern __shared__ __align__(16) float xs[];                // [DECAY_TOKENS][rank]
    pb_grid_dep_launch();
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t0 = blockIdx.x * DECAY_TOKENS, cnt = min(DECAY_TOKENS, n_tokens - t0);
    const float b = c < channels ? bias[c] : 0.f;
    pb_grid_dep_wait();
    for (int i = threadIdx.x; i < DECAY_TOKENS * rank; i += blockDim.x) {
        const int u = i / rank;
        xs[i] = u < cnt ? pb_ld(x1 + (size_t)(t0 + u) * ld_x1 + i % rank) : 0.f;
    }
    __syncthreads();
    if (c >= channels) return;
    const T* w = w2 + (size_t)c * rank;
    float acc[DECAY_TOKENS];
#pragma unroll
    for (int u = 0; u < DECAY_TOKENS; ++u) acc[u] = 0.f;
    constexpr int VN = 16 / sizeof(T);
    int r = 0;
    if (vec) {
        for (; r + VN <= rank; r += VN) {
            float wv[VN];
            gla_unpack(*reinterpret_cast<const uint4*>(w + r), wv);
#pragma unroll
            for (int u = 0; u < DECAY_TOKENS; ++u) {
#pragma unroll
                for (int e = 0; e < VN; e += 4) {
                    const float4 f = *reinterpret_cast<const float4*>(xs + u * rank + r + e);
                    acc[u] = fmaf(f.x, wv[e], acc[u]);
                    acc[u] = fmaf(f.y, wv[e + 1], acc[u]);
                    acc[u] = fmaf(f.z, wv[e + 2], acc[u]);
                    acc[u] = fmaf(f.w, wv[e + 3], acc[u]);
                }
            }
        }
    }
    for (; r < rank; ++r) {
        const float wv = pb_ld(w + r);
#pragma unroll
        for (int u = 0; u < DECAY_TOKENS; ++u)
            if (u < cnt) acc[u] = fmaf(xs[u * rank + r], wv, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < DECAY_TOKENS; ++u)
        if (u < cnt) out[(size_t)(t0 + u) * channels + c] = gla_decay(acc[u] + b, inv_tau);
}

// ---------------------------------------------------------------------------------------------------------
// The scan.  A block is eight warps on one head's state.  Warps 0-3 compute: a thread keeps R key channels x C value columns
// of the state in registers (channel pairs packed, so one instruction moves two of them on), RL lanes share a column group;
// nothing but the multiply-add by the decay lies between one token's state and the next one's.  The outputs of four tokens
// are summed over the RL lanes together: every exchange halves the values a lane still holds.  Warps 4-7 load: while the
// others work on one chunk of tokens they put the next chunk's k, q, decay and v into the other half of shared memory as
// float32 (channels past N as zeros: they stay zero in the state; tokens past a step's last one with k = 0 and decay 1: they
// leave the state as it is, so a group of tokens has no branches and its loads run ahead of its sums).
// Channel of a thread's register 4 i + e: (i * RL + j) * 4 + e, so that a column group's lanes read consecutive 16-byte pieces.
#define GLA_GROUP 4                                            // tokens summed over the lanes together

// Step K of summing NV values over RL lanes (K = 0: lanes RL / 2 apart, and so on): a lane gives half of what it holds away
// and adds its partner's share of the other half; once it holds one value, the two partners add up the same one.
template <int NV, int RL, int K>
__device__ __forceinline__ void lanes_step(float (&v)[NV], int j) {
    constexpr int step = RL >> (K + 1), held = (NV >> K) > 1 ? (NV >> K) : 1;
    if constexpr (step >= 1) {
        if constexpr (held > 1) {
            const bool up = (j & step) != 0;
#pragma unroll
            for (int i = 0; i < held / 2; ++i) {
                const float send = up ? v[i] : v[i + held / 2], keep = up ? v[i + held / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], step);
        }
    }
}
// The first of the values that lane j holds in the end; NV or more: a copy of what another lane holds.
template <int NV, int RL>
__device__ __forceinline__ int lanes_first(int j) {
    int base = 0, n = NV;
#pragma unroll
    for (int step = RL / 2; step >= 1; step >>= 1) {
        if (n > 1) { n >>= 1; base += (j & step) ? n : 0; }
        else if (j & step) base = NV;
    }
    return base;
}

template <typename T, int RL, int R, int C, int CHUNK>
__global__ void __launch_bounds__(256, 1)
gla_scan_kernel(const T* q_in, const T* k_in, const T* v_in, long long ld, const float* decay,
                float scale, float* state, float* y, const int32_t* cu_q,
                const int32_t* slots, int H, int N, int P, int vec, int vec_state) {
    constexpr int NPAD = RL * R;
    constexpr int COLS = 4 * (32 / RL) * C;                    // of a block
    constexpr int BUF = CHUNK * (3 * NPAD + COLS);             // floats per half: k, q, decay, v
    constexpr int VN = 16 / sizeof(T);
    extern __shared__ __align__(16) float gla_sm[];
    pb_grid_dep_launch();
    const int col_blocks = (P + COLS - 1) / COLS;
    const int h = blockIdx.x / col_blocks, p_first = (blockIdx.x % col_blocks) * COLS;
    const int rq = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool computes = warp < 4;
    pb_grid_dep_wait();
    const int first = cu_q[rq], n_tok = cu_q[rq + 1] - first;
    if (n_tok <= 0) return;
    const int n_chunks = (n_tok + CHUNK - 1) / CHUNK;
    const size_t slot_base = ((size_t)slots[rq] * H + h) * N * (size_t)P;

    if (!computes) {
        // A chunk's rows are asked for a whole chunk before they are stored: a trip to memory has as long as the compute warps
        // take for a chunk.  16-byte pieces of k and q, then of the decay, then single values of v.
        const int lt = tid - 128;
        constexpr int PK = NPAD / VN, K_IT = (CHUNK * PK + 127) / 128, PA = NPAD / 4, A_IT = (CHUNK * PA + 127) / 128;
        constexpr int V_IT = (CHUNK * COLS + 127) / 128;
        uint4 kr[K_IT], qr[K_IT], ar[A_IT];
        T vr[V_IT];
        const uint4 zero = make_uint4(0, 0, 0, 0), ones = make_uint4(0x3f800000u, 0x3f800000u, 0x3f800000u, 0x3f800000u);
        auto ask = [&](int ch) {
            const int t0 = ch * CHUNK, cnt = min(CHUNK, n_tok - t0);
            const size_t row0 = (size_t)(first + t0);
            if (vec) {
#pragma unroll
                for (int it = 0; it < K_IT; ++it) {
                    const int idx = lt + it * 128, tt = idx / PK, n = (idx % PK) * VN;
                    const bool ok = tt < cnt && n < N;
                    const size_t off = (row0 + (ok ? tt : 0)) * ld + (size_t)h * N + (ok ? n : 0);
                    kr[it] = ok ? *reinterpret_cast<const uint4*>(k_in + off) : zero;
                    qr[it] = ok ? *reinterpret_cast<const uint4*>(q_in + off) : zero;
                }
#pragma unroll
                for (int it = 0; it < A_IT; ++it) {
                    const int idx = lt + it * 128, tt = idx / PA, n = (idx % PA) * 4;
                    const bool ok = tt < cnt && n < N;
                    ar[it] = ok ? *reinterpret_cast<const uint4*>(decay + ((row0 + tt) * H + h) * N + n) : (tt < cnt ? zero : ones);
                }
            }
#pragma unroll
            for (int it = 0; it < V_IT; ++it) {
                const int idx = lt + it * 128, tt = idx / COLS, cc = idx % COLS;
                const bool ok = tt < cnt && p_first + cc < P;
                vr[it] = v_in[ok ? (row0 + tt) * ld + (size_t)h * P + p_first + cc : (size_t)first * ld];
                if (!ok) pb_st(&vr[it], 0.f);
            }
        };
        auto put = [&](int ch) {
            float* buf = gla_sm + (ch & 1) * BUF;
            float* qs = buf + CHUNK * NPAD;
            float* as = buf + 2 * CHUNK * NPAD;
            float* vs = buf + 3 * CHUNK * NPAD;
            if (vec) {
#pragma unroll
                for (int it = 0; it < K_IT; ++it) {
                    const int idx = lt + it * 128, tt = idx / PK, n = (idx % PK) * VN;
                    if (tt >= CHUNK) continue;
                    float kf[VN], qf[VN];
                    gla_unpack(kr[it], kf);
                    gla_unpack(qr[it], qf);
#pragma unroll
                    for (int e = 0; e < VN; e += 4) {
                        *reinterpret_cast<float4*>(buf + tt * NPAD + n + e) = make_float4(kf[e], kf[e + 1], kf[e + 2], kf[e + 3]);
                        *reinterpret_cast<float4*>(qs + tt * NPAD + n + e) = make_float4(qf[e], qf[e + 1], qf[e + 2], qf[e + 3]);
                    }
                }
#pragma unroll
                for (int it = 0; it < A_IT; ++it) {
                    const int idx = lt + it * 128, tt = idx / PA, n = (idx % PA) * 4;
                    if (tt < CHUNK) *reinterpret_cast<uint4*>(as + tt * NPAD + n) = ar[it];
                }
            } else {                                           // sizes or rows that 16-byte pieces do not fit: element by element
                const int t0 = ch * CHUNK, cnt = min(CHUNK, n_tok - t0);
                const size_t row0 = (size_t)(first + t0);
                for (int idx = lt; idx < CHUNK * NPAD; idx += 128) {
                    const int tt = idx / NPAD, n = idx % NPAD;
                    const bool ok = tt < cnt && n < N;
                    const size_t off = (row0 + (ok ? tt : 0)) * ld + (size_t)h * N + (ok ? n : 0);
                    buf[idx] = ok ? pb_ld(k_in + off) : 0.f;
                    qs[idx] = ok ? pb_ld(q_in + off) : 0.f;
                    as[idx] = ok ? decay[((row0 + tt) * H + h) * N + n] : (tt < cnt ? 0.f : 1.f);
                }
            }
#pragma unroll
            for (int it = 0; it < V_IT; ++it) {
                const int idx = lt + it * 128;
                if (idx < CHUNK * COLS) vs[idx] = pb_ld(&vr[it]);
            }
        };
        ask(0);
        put(0);
        if (n_chunks > 1) ask(1);
        __syncthreads();
        for (int ch = 0; ch < n_chunks; ++ch) {
            if (ch + 1 < n_chunks) put(ch + 1);
            if (ch + 2 < n_chunks) ask(ch + 2);
            __syncthreads();
        }
        return;
    }

    // compute warps
    const int j = lane % RL;
    const int cl = (warp * (32 / RL) + lane / RL) * C;         // the thread's first column within the block
    const int p0 = p_first + cl;
    u64 s[R / 2][C];
    float* S = state + slot_base;
    auto row_of = [&](int r) { return ((r >> 2) * RL + j) * 4 + (r & 3); };
    auto load_row = [&](int n, float (&o)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) o[c] = 0.f;
        if (n >= N) return;
        const float* src = S + (size_t)n * P + p0;
        if (vec_state) {
#pragma unroll
            for (int c = 0; c < C; c += 4)
                if (p0 + c < P) { const float4 f = *reinterpret_cast<const float4*>(src + c); o[c] = f.x; o[c + 1] = f.y; o[c + 2] = f.z; o[c + 3] = f.w; }
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c) if (p0 + c < P) o[c] = src[c];
        }
    };
    auto store_row = [&](int n, const float (&o)[C]) {
        if (n >= N) return;
        float* dst = S + (size_t)n * P + p0;
        if (vec_state) {
#pragma unroll
            for (int c = 0; c < C; c += 4)
                if (p0 + c < P) *reinterpret_cast<float4*>(dst + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c) if (p0 + c < P) dst[c] = o[c];
        }
    };
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        float lo[C], hi[C];
        load_row(row_of(r), lo);
        load_row(row_of(r + 1), hi);
#pragma unroll
        for (int c = 0; c < C; ++c) s[r / 2][c] = pk2(lo[c], hi[c]);
    }
    __syncthreads();
    const size_t y_ld = (size_t)H * P;
    float* yb = y + (size_t)first * y_ld + (size_t)h * P + p0;
    // The sums of one group of tokens over the lanes run between the next group's tokens, a step a token: their exchanges wait
    // while the state moves on.
    constexpr int NV = GLA_GROUP * C, LEFT = NV / RL > 1 ? NV / RL : 1;        // LEFT: values a lane holds in the end
    const int base = lanes_first<NV, RL>(j);
    float prev[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) prev[i] = 0.f;
    int prev_t = -GLA_GROUP;
    auto store = [&]() {
        if (base < NV) {
#pragma unroll
            for (int e = 0; e < LEFT; ++e) {
                const int t = prev_t + (base + e) / C, c = (base + e) % C;
                if (t >= 0 && t < n_tok && p0 + c < P) yb[(size_t)t * y_ld + c] = prev[e] * scale;
            }
        }
    };
    for (int ch = 0; ch < n_chunks; ++ch) {
        const float* buf = gla_sm + (ch & 1) * BUF;
        const int t0 = ch * CHUNK, cnt = min(CHUNK, n_tok - t0);
#pragma unroll 2
        for (int g0 = 0; g0 < cnt; g0 += GLA_GROUP) {
            float o[NV];
#pragma unroll
            for (int u = 0; u < GLA_GROUP; ++u) {
                const int tt = g0 + u;
                const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(buf + tt * NPAD) + j;
                const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(buf + CHUNK * NPAD + tt * NPAD) + j;
                const ulonglong2* a4 = reinterpret_cast<const ulonglong2*>(buf + 2 * CHUNK * NPAD + tt * NPAD) + j;
                const float* vp = buf + 3 * CHUNK * NPAD + tt * COLS + cl;
                u64 vd[C], acc[C];
#pragma unroll
                for (int c = 0; c < C; c += 4) {
                    const float4 f = *reinterpret_cast<const float4*>(vp + c);
                    vd[c] = pk2(f.x, f.x); vd[c + 1] = pk2(f.y, f.y); vd[c + 2] = pk2(f.z, f.z); vd[c + 3] = pk2(f.w, f.w);
                }
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    const ulonglong2 kk = k4[i * RL], qq = q4[i * RL], aa = a4[i * RL];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        s[2 * i][c] = fma2(aa.x, s[2 * i][c], mul2(kk.x, vd[c]));
                        acc[c] = i == 0 ? mul2(s[2 * i][c], qq.x) : fma2(s[2 * i][c], qq.x, acc[c]);
                        s[2 * i + 1][c] = fma2(aa.y, s[2 * i + 1][c], mul2(kk.y, vd[c]));
                        acc[c] = fma2(s[2 * i + 1][c], qq.y, acc[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < C; ++c) { const float2 f = up2(acc[c]); o[u * C + c] = f.x + f.y; }
                if (u == 0) lanes_step<NV, RL, 0>(prev, j);
                else if (u == 1) lanes_step<NV, RL, 1>(prev, j);
                else if (u == 2) lanes_step<NV, RL, 2>(prev, j);
                else { lanes_step<NV, RL, 3>(prev, j); lanes_step<NV, RL, 4>(prev, j); }
            }
            store();
#pragma unroll
            for (int i = 0; i < NV; ++i) prev[i] = o[i];
            prev_t = t0 + g0;
        }
        __syncthreads();
    }
    lanes_step<NV, RL, 0>(prev, j);
    lanes_step<NV, RL, 1>(prev, j);
    lanes_step<NV, RL, 2>(prev, j);
    lanes_step<NV, RL, 3>(prev, j);
    lanes_step<NV, RL, 4>(prev, j);
    store();
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        float lo[C], hi[C];
#pragma unroll
        for (int c = 0; c < C; ++c) { const float2 f = up2(s[r / 2][c]); lo[c] = f.x; hi[c] = f.y; }
        store_row(row_of(r), lo);
        store_row(row_of(r + 1), hi);
    }
}

// ---------------------------------------------------------------------------------------------------------
// One token per sequence.  A block owns a head's whole state: STEP_THREADS threads, P / 4 column groups of four and as many
// channels at a time as fit; a thread asks for eight of its rows before it makes the channels' decays, so the state is on its
// way meanwhile.  Behind the sums: the head's norm over its P outputs, the shared weight, silu of the gate, one rounding.
#define STEP_THREADS 512
#define STEP_ROWS 8
template <typename T>
__global__ void __launch_bounds__(STEP_THREADS)
gla_step_kernel(const T* q_in, const T* k_in, const T* v_in, const T* x1,
                const T* gate, long long ld, const T* w2, const float* bias, float inv_tau, float scale,
                const float* norm_w, float eps, float* state, T* out, const int32_t* cu_q,
                const int32_t* slots, int H, int N, int P, int rank, int vec) {
    extern __shared__ __align__(16) float step_sm[];           // k, q, decay [N] each; outputs [row groups][P]; sums
    __shared__ float red[STEP_THREADS / 32];
    pb_grid_dep_launch();
    const int h = blockIdx.x, rq = blockIdx.y, tid = threadIdx.x;
    const int CG = P >> 2, RG = STEP_THREADS / CG;
    const int cg = tid % CG, rg = tid / CG;
    float* ks = step_sm;
    float* qs = ks + N;
    float* as = qs + N;
    float* os = step_sm + ((3 * N + 3) & ~3);
    pb_grid_dep_wait();
    const int t = cu_q[rq];
    if (cu_q[rq + 1] - t <= 0) return;
    float* S = state + ((size_t)slots[rq] * H + h) * N * (size_t)P + 4 * cg;
    const bool works = rg < RG;
    const int n_rows = works ? (N - rg + RG - 1) / RG : 0;     // channels rg, rg + RG, ...
    float4 s[STEP_ROWS];
#pragma unroll
    for (int i = 0; i < STEP_ROWS; ++i)
        if (i < n_rows) s[i] = *reinterpret_cast<const float4*>(S + (size_t)(rg + i * RG) * P);
    const T* xr = x1 + (size_t)t * ld;
    for (int n = tid; n < N; n += STEP_THREADS) {
        const size_t c = (size_t)h * N + n;
        ks[n] = pb_ld(k_in + (size_t)t * ld + c);
        qs[n] = pb_ld(q_in + (size_t)t * ld + c);
        const T* w = w2 + c * rank;
        float z = 0.f;
        constexpr int VN = 16 / sizeof(T);
        int r = 0;
        if (vec) {
#pragma unroll 2
            for (; r + VN <= rank; r += VN) {
                float wv[VN];
                gla_unpack(*reinterpret_cast<const uint4*>(w + r), wv);
#pragma unroll
                for (int e = 0; e < VN; ++e) z = fmaf(pb_ld(xr + r + e), wv[e], z);
            }
        }
        for (; r < rank; ++r) z = fmaf(pb_ld(xr + r), pb_ld(w + r), z);
        as[n] = gla_decay(z + bias[c], inv_tau);
    }
    float v[4] = {0.f, 0.f, 0.f, 0.f}, o[4] = {0.f, 0.f, 0.f, 0.f};
    if (works) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = pb_ld(v_in + (size_t)t * ld + (size_t)h * P + 4 * cg + e);
    }
    __syncthreads();
    for (int i0 = 0; i0 < n_rows; i0 += STEP_ROWS) {
        if (i0 > 0) {
#pragma unroll
            for (int i = 0; i < STEP_ROWS; ++i)
                if (i0 + i < n_rows) s[i] = *reinterpret_cast<const float4*>(S + (size_t)(rg + (i0 + i) * RG) * P);
        }
#pragma unroll
        for (int i = 0; i < STEP_ROWS; ++i) {
            if (i0 + i < n_rows) {
                const int n = rg + (i0 + i) * RG;
                const float a = as[n], k = ks[n], q = qs[n];
                s[i].x = fmaf(a, s[i].x, k * v[0]); s[i].y = fmaf(a, s[i].y, k * v[1]);
                s[i].z = fmaf(a, s[i].z, k * v[2]); s[i].w = fmaf(a, s[i].w, k * v[3]);
                o[0] = fmaf(s[i].x, q, o[0]); o[1] = fmaf(s[i].y, q, o[1]); o[2] = fmaf(s[i].z, q, o[2]); o[3] = fmaf(s[i].w, q, o[3]);
                *reinterpret_cast<float4*>(S + (size_t)n * P) = s[i];
            }
        }
    }
    if (works) *reinterpret_cast<float4*>(os + (size_t)rg * P + 4 * cg) = make_float4(o[0], o[1], o[2], o[3]);
    __syncthreads();
    // the row groups' sums, then the norm over the head (a thread has at most P / STEP_THREADS + 1 outputs)
    float ss = 0.f;
    for (int p = tid; p < P; p += STEP_THREADS) {
        float acc = 0.f;
        for (int g = 0; g < RG; ++g) acc += os[(size_t)g * P + p];
        acc *= scale;
        os[p] = acc;                                           // row group 0's place: read by this thread alone
        ss += acc * acc;
    }
    ss = pb_warp_sum(ss);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < STEP_THREADS / 32; ++i) total += red[i];
    const float inv = 1.0f / sqrtf(total / (float)P + eps);
    for (int p = tid; p < P; p += STEP_THREADS) {
        const float g = pb_ld(gate + (size_t)t * ld + (size_t)h * P + p);
        pb_st(out + (size_t)t * H * P + (size_t)h * P + p, os[p] * inv * norm_w[p] * (g / (1.0f + expf(-g))));
    }
}

}  // namespace

// x1 [n_tokens, rank] of type dtype, row stride ld_x1; w2 [channels, rank] dense of type dtype; bias float32 [channels];
// out float32 [n_tokens, channels] dense.
PB_API int pb_channel_decay(const void* x1, long long ld_x1, const void* w2, const float* bias, float tau, float* out, int dtype, int n_tokens,
                            int channels, int rank, cudaStream_t stream) {
    PB_REQUIRE(n_tokens >= 0 && channels > 0 && rank > 0 && ld_x1 >= rank && tau > 0.f, "channel_decay: bad sizes");
    PB_REQUIRE(x1 && w2 && bias && out, "channel_decay: null pointer");
    const size_t smem = (size_t)DECAY_TOKENS * rank * sizeof(float);
    PB_REQUIRE(smem <= 48 * 1024, "channel_decay: a rank of %d (at most %d)", rank, 48 * 1024 / DECAY_TOKENS / 4);
    PB_REQUIRE((channels + 127) / 128 < 65536, "channel_decay: %d channels", channels);
    if (n_tokens == 0) return 0;
    if (dtype == PB_BF16 && rank % 8 == 0 && rank <= 64 && n_tokens >= 64 && pb_aligned(w2, 16) && pb_aligned(x1, 16) && ld_x1 % 8 == 0) {
        // A block's time grows with its tokens, and with the rank the registers, so that fewer blocks are on a multiprocessor: many tokens a
        // block (the row of the matrix is fetched once) where there are several waves of such blocks.  us with 8 / 16 / 32 / 64 tokens a
        // block, behind them a block of eight on the kernel below: rank 32, 500 tokens of 4,096 channels 13.1 / 9.8 / 10.0 / 24.7, 17.0;
        // 2,048 of 2,048 27.6 / 20.3 / 17.4 / 18.9, 30.1; 2,048 of 4,096 52 / 40 / 33 / 31, 56; rank 16, 2,048 of 2,048 12.9 / 12.2 /
        // 16.4 / 27.6, 16.8; 200 of 4,096 5.2 / 7.6 / 9.8 / 9.7, 6.4; 2,048 of 4,096 24.0 / 22.6 / 22.6 / 30.6, 30.9.
        const int cols = (channels + 127) / 128;
        const long long blocks = (long long)((n_tokens + 63) / 64) * cols;
        const int tokens = rank >= 32 ? (blocks >= 960 ? 64 : blocks >= 256 ? 32 : 16) : (blocks >= 960 ? 16 : 8);
        const dim3 grid((n_tokens + tokens - 1) / tokens, cols);
        const size_t bytes = (size_t)rank * (tokens + 4) * sizeof(float);
#define DECAY_ROWS(RANK)                                                                                                      \
    case RANK:                                                                                                               \
        pb_launch(channel_decay_rows_kernel<RANK>, grid, dim3(128), bytes, stream, (const __nv_bfloat16*)x1, ld_x1, (const __nv_bfloat16*)w2, bias, \
                  1.0f / tau, out, n_tokens, channels, tokens);                                                              \
        break;
        switch (rank) { DECAY_ROWS(8) DECAY_ROWS(16) DECAY_ROWS(24) DECAY_ROWS(32) DECAY_ROWS(40) DECAY_ROWS(48) DECAY_ROWS(56) DECAY_ROWS(64) }
#undef DECAY_ROWS
        PB_CHECK_LAUNCH("channel_decay");
        return 0;
    }
    const int vec = rank % (dtype == PB_BF16 ? 8 : 4) == 0 && pb_aligned(w2, 16) ? 1 : 0;
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(channel_decay_kernel<T>, dim3((n_tokens + DECAY_TOKENS - 1) / DECAY_TOKENS, (channels + 127) / 128), dim3(128),
                                           smem, stream, (const T*)x1, ld_x1, (const T*)w2, bias, 1.0f / tau, out, n_tokens, channels, rank, vec)));
    PB_CHECK_LAUNCH("channel_decay");
    return 0;
}

template <typename T, int RL, int R, int C, int CHUNK>
static int gla_launch(const void* q, const void* k, const void* v, long long ld, const float* decay, float scale, float* state, float* y,
                      const int32_t* cu_q, const int32_t* slots, int n_seqs, int H, int N, int P, int vec, cudaStream_t stream) {
    constexpr int COLS = 4 * (32 / RL) * C;
    constexpr int smem = 2 * CHUNK * (3 * RL * R + COLS) * (int)sizeof(float);
    if (smem > 48 * 1024) {
        static bool set = false;
        if (!set) {
            const cudaError_t e = cudaFuncSetAttribute(gla_scan_kernel<T, RL, R, C, CHUNK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return pb_fail("gla_scan: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
            set = true;
        }
    }
    const int vec_state = P % 4 == 0 && pb_aligned(state, 16) ? 1 : 0;
    pb_launch(gla_scan_kernel<T, RL, R, C, CHUNK>, dim3(H * ((P + COLS - 1) / COLS), n_seqs), dim3(256), (size_t)smem, stream, (const T*)q, (const T*)k,
              (const T*)v, ld, decay, scale, state, y, cu_q, slots, H, N, P, vec, vec_state);
    return 0;
}

#define GLA_MAX_N 512

// q, k [n_tokens, H * N] and v [n_tokens, H * P]: columns of one projection, rows ld apart; decay float32 [n_tokens, H * N]
// dense; state float32 [slots, H, N, P]; y float32 [n_tokens, H * P] dense; cu_q [n_seqs + 1], slots [n_seqs].
PB_API int pb_gla_scan(const void* q, const void* k, const void* v, long long ld, int dtype, const float* decay, float scale, float* state, float* y,
                       const int32_t* cu_q, const int32_t* slots, int n_seqs, int H, int N, int P, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && H > 0 && N > 0 && P > 0, "gla_scan: bad sizes");
    PB_REQUIRE(N <= GLA_MAX_N, "gla_scan: keys of %d elements (at most %d)", N, GLA_MAX_N);
    PB_REQUIRE(q && k && v && decay && state && y && cu_q && slots && ld >= (long long)H * N && ld >= (long long)H * P, "gla_scan: null pointer or short rows");
    if (n_seqs == 0) return 0;
    PB_REQUIRE(n_seqs < 65536, "gla_scan: %d sequences in one launch", n_seqs);
    const int vn = dtype == PB_BF16 ? 8 : 4;
    const int vec = N % vn == 0 && ld % vn == 0 && pb_aligned(q, 16) && pb_aligned(k, 16) && pb_aligned(decay, 16) ? 1 : 0;
    // four channels (more above 128) x four columns a thread, or eight columns where that still leaves enough blocks to fill
    // the device: the wider a thread's piece, the fewer numbers it reads from shared memory per state element
    const int cols8 = N <= 16 ? 256 : (N <= 32 ? 128 : (N <= 64 ? 64 : 32));
    const bool wide = N <= 128 && (long long)H * ((P + cols8 - 1) / cols8) * n_seqs >= 120 && P > cols8 / 2;
    int e = 0;
#define GLA_LAUNCH(RL, R, C, CHUNK) \
    PB_DISPATCH_DTYPE(dtype, T, (e = gla_launch<T, RL, R, C, CHUNK>(q, k, v, ld, decay, scale, state, y, cu_q, slots, n_seqs, H, N, P, vec, stream)))
    if (N <= 16) { if (wide) GLA_LAUNCH(4, 4, 8, 16); else GLA_LAUNCH(4, 4, 4, 16); }
    else if (N <= 32) { if (wide) GLA_LAUNCH(8, 4, 8, 16); else GLA_LAUNCH(8, 4, 4, 16); }
    else if (N <= 64) { if (wide) GLA_LAUNCH(16, 4, 8, 16); else GLA_LAUNCH(16, 4, 4, 16); }
    else if (N <= 128) { if (wide) GLA_LAUNCH(32, 4, 8, 16); else GLA_LAUNCH(32, 4, 4, 16); }
    else if (N <= 256) GLA_LAUNCH(32, 8, 4, 8);
    else GLA_LAUNCH(32, 16, 4, 4);
#undef GLA_LAUNCH
    if (e) return e;
    PB_CHECK_LAUNCH("gla_scan");
    return 0;
}

static size_t gla_step_smem(int N, int P) { return ((size_t)((3 * N + 3) & ~3) + (size_t)(STEP_THREADS / (P / 4)) * P) * sizeof(float); }

PB_API int pb_gla_step_supported(int N, int P) {
    return N > 0 && P > 0 && P % 4 == 0 && P / 4 <= STEP_THREADS && gla_step_smem(N, P) <= 48 * 1024 ? 1 : 0;
}

// A step of at most one token per sequence: what pb_channel_decay, pb_gla_scan and the norm with its gate do, in one kernel.
// q, k, v, x1, gate: columns of one projection, rows ld apart; norm_w float32 [P] (the heads share it); out [n_tokens, H * P]
// of type dtype, dense.
PB_API int pb_gla_step(const void* q, const void* k, const void* v, const void* x1, const void* gate, long long ld, int dtype, const void* w2,
                       const float* bias, float tau, float scale, const float* norm_w, float eps, float* state, void* out, const int32_t* cu_q,
                       const int32_t* slots, int n_seqs, int H, int N, int P, int rank, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && H > 0 && rank > 0 && tau > 0.f && pb_gla_step_supported(N, P), "gla_step: sizes N=%d P=%d rank=%d not taken", N, P, rank);
    PB_REQUIRE(q && k && v && x1 && gate && w2 && bias && norm_w && state && out && cu_q && slots && pb_aligned(state, 16), "gla_step: null or unaligned pointer");
    if (n_seqs == 0) return 0;
    PB_REQUIRE(n_seqs < 65536, "gla_step: %d sequences in one launch", n_seqs);
    const int vec = rank % (dtype == PB_BF16 ? 8 : 4) == 0 && pb_aligned(w2, 16) ? 1 : 0;
    PB_DISPATCH_DTYPE(dtype, T, (pb_launch(gla_step_kernel<T>, dim3(H, n_seqs), dim3(STEP_THREADS), gla_step_smem(N, P), stream, (const T*)q, (const T*)k,
                                           (const T*)v, (const T*)x1, (const T*)gate, ld, (const T*)w2, bias, 1.0f / tau, scale, norm_w, eps, state,
                                           (T*)out, cu_q, slots, H, N, P, rank, vec)));
    PB_CHECK_LAUNCH("gla_step");
    return 0;
}
