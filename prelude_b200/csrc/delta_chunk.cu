// The gated delta rule of a prompt step by chunks of 64 tokens, on the tensor cores:
//
//   pb_gated_delta_scan_chunked   as pb_gated_delta_scan (delta_rule.cu)
//
// With l_t the sum of the logarithms of the decays up to token t of the chunk, k' and q' the unit keys and queries, S the state
// before the chunk and u_t what token t writes along its key,
//     u_t = beta_t (v_t - exp(l_t) S^T k'_t - sum_{s < t} exp(l_t - l_s) (k'_t . k'_s) u_s)
//     o_t = exp(l_t) S^T q'_t + sum_{s <= t} exp(l_t - l_s) (q'_t . k'_s) u_s
//     S'  = exp(l_last) S + sum_s exp(l_last - l_s) k'_s u_s^T
// The first line is a triangular system (I + A) U = R whose matrix does not depend on the state.  One kernel makes, for every
// chunk and head at once, (I + A)^-1 and the weights of the second line; a second walks the chunks of a head, each of them five
// small products: K S, Q S, (I + A)^-1 R, the weights times U, and K^T times the weighted U.
// K and Q enter the products as they are (bfloat16: exact) and their norms as factors of the sums; everything that is float32
// enters as three bfloat16 numbers whose sum it is (mma_sync.cuh; of nine products of two such operands the six that reach
// float32's last bit are taken); sums of logarithms are taken in 64-bit and kept as a float32 pair; the inverse is made in float32
// by substitution.  No exponent is positive; a decay below exp(-110) counts as exp(-110), which is zero in float32.
//
// What bounds it: the chain of chunks, with three barriers in each.  A block therefore takes few columns of a head's state (16
// or 32), and whatever does not depend on the state is taken out of the chain.  2,048 tokens of one sequence, heads of 128 x 128:
// 16 heads (128 blocks of 16 columns) 111 us against 733 token by token (pb_gated_delta_scan), 32 heads (128 of 32) 196 against 750;
// sequences of 592 and 1,185 tokens, 16 heads, 118 against 432; 64 tokens from memory 25 against 31, 32 tokens 25 against 21.  Error against
// 64-bit where decays are slow (a step of 1e-3): output 1.0 to 2.1e-7 (token by token 2.1e-7 to 3.2e-6), state 0.4 to 2.9e-7 (0.7e-7 to
// 9e-6); where they are fast (0.05 and more) it is up to 1.7 times the tokens' in their place: 0.9 to 1.9e-7 (1.1 to 1.6e-7), state 0.4
// to 1.3e-7 (0.5 to 1.4e-7).
#include "mma_sync.cuh"
#include "sequences.cuh"

#include <math.h>

namespace {

typedef __nv_bfloat16 bf16;

constexpr int DC_L = 64;                                    // tokens of a chunk
constexpr int DC_MUL = 256, DC_ALL = 384;                   // multiplying threads, all threads of the walk
// What the first kernel leaves for a chunk and head: ten 16 x 16 tiles of the lower triangle, row by row, of (I + A)^-1 and of the
// weights, each as three parts of 32 lanes x 16 bytes in the order of an A operand; then four numbers a token - exp(l) / |k|,
// beta, exp(l) / (|q| sqrt(D)), exp(l_last - l) / |k| - exp(l_last), and the first token whose key, beta or decay is not finite
constexpr int DC_TILE = 3 * 32 * 16, DC_TRI = 10 * DC_TILE, DC_NUM = 2 * DC_TRI, DC_BLOB = DC_NUM + 4 * DC_L * 4 + 16;

__device__ __forceinline__ int dc_tri(int i) { return i * (i + 1) / 2; }

template <int D>
struct DcPrep {
    static constexpr int LDK = D + 8, LDA = DC_L + 4, LDX = 36;
    static constexpr int k = 0, q = k + DC_L * LDK * 2;
    // the inverse is made where the keys and queries lay once their products are there: four blocks a multiprocessor
    static constexpr int t = 0, x = t + DC_L * LDA * 4, rows = q + DC_L * LDK * 2, work = x + 32 * LDX * 4, a = rows > work ? rows : work;
    static constexpr int num = a + DC_L * LDA * 4, bytes = num + (6 * DC_L + 4) * 4;
};

template <int D>
__global__ void __launch_bounds__(256, 4)
delta_prepare_kernel(const bf16* u, long long ld_u, const bf16* b_in, long long ld_b, const bf16* a_in, long long ld_a, const float* a_log,
                     const float* dt_bias, const int32_t* cu_q, unsigned char* blobs, int n_seqs, int least, int few, int beside, int H, int G) {
    using Z = DcPrep<D>;
    extern __shared__ __align__(16) unsigned char dp_sm[];
    pb_grid_dep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, g = h / (H / G);
    const float rate = expf(a_log[h]), bias = dt_bias[h];       // written by no kernel: before the wait
    pb_grid_dep_wait();
    int t_first = 0;
    if (beside > 0) least = pb_length_limit(cu_q, n_seqs, least, few, beside, lane);
    const int cnt = pb_find_chunk<DC_L>(cu_q, n_seqs, least, blockIdx.x, lane, t_first);
    if (cnt <= 0) return;
    bf16* ks = reinterpret_cast<bf16*>(dp_sm + Z::k);
    bf16* qs = reinterpret_cast<bf16*>(dp_sm + Z::q);
    float* A = reinterpret_cast<float*>(dp_sm + Z::a);
    float* Ti = reinterpret_cast<float*>(dp_sm + Z::t);
    float* X = reinterpret_cast<float*>(dp_sm + Z::x);
    float* ik = reinterpret_cast<float*>(dp_sm + Z::num);
    float *iq = ik + DC_L, *beta = iq + DC_L, *lh = beta + DC_L, *ll = lh + DC_L, *bad = ll + DC_L;   // bad: 1 where a token is not finite
    int* first_bad = reinterpret_cast<int*>(bad + DC_L);
    unsigned char* blob = blobs + ((size_t)blockIdx.x * H + h) * DC_BLOB;

    for (int idx = tid; idx < DC_L * (D / 8); idx += 256) {
        const int tt = idx / (D / 8), n = idx % (D / 8) * 8;
        if (tt < cnt) {
            const bf16* row = u + (size_t)(t_first + tt) * ld_u + (size_t)g * D + n;
            pb_cp_async16(qs + tt * Z::LDK + n, row);
            pb_cp_async16(ks + tt * Z::LDK + n, row + (size_t)G * D);
        } else {
            *reinterpret_cast<uint4*>(qs + tt * Z::LDK + n) = *reinterpret_cast<uint4*>(ks + tt * Z::LDK + n) = make_uint4(0, 0, 0, 0);
        }
    }
    float braw = 0.f, araw = 0.f;                               // lane e < 8: of token 8 warp + e
    if (lane < 8 && warp * 8 + lane < cnt) {
        braw = pb_ld(b_in + (size_t)(t_first + warp * 8 + lane) * ld_b + h);
        araw = pb_ld(a_in + (size_t)(t_first + warp * 8 + lane) * ld_a + h);
    }
    pb_cp_async_wait();
    __syncthreads();
    const float q_scale = 1.0f / sqrtf((float)D);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int tt = warp * 8 + e;
        float sq = 0.f, sk = 0.f;
        bool finite = true;
#pragma unroll
        for (int i = 0; i < D / 32; ++i) {
            const float qv = __bfloat162float(qs[tt * Z::LDK + lane + 32 * i]), kv = __bfloat162float(ks[tt * Z::LDK + lane + 32 * i]);
            sq = fmaf(qv, qv, sq);
            sk = fmaf(kv, kv, sk);
            finite = finite && isfinite(kv);
        }
        sq = pb_warp_sum(sq);
        sk = pb_warp_sum(sk);
        finite = __all_sync(0xffffffffu, finite);
        if (lane == e) {
            const float bt = tt < cnt ? 1.0f / (1.0f + expf(-braw)) : 0.f;
            const float lg = tt < cnt ? -rate * pb_softplus(araw + bias) : 0.f;      // a token past the end: decay 1, nothing written
            ik[tt] = 1.0f / sqrtf(sk + 1e-6f);
            iq[tt] = q_scale / sqrtf(sq + 1e-6f);
            beta[tt] = bt;
            lh[tt] = lg;
            bad[tt] = finite && !isnan(bt) && !isnan(lg) ? 0.f : 1.f;
        }
    }
    __syncthreads();
    if (warp == 0) {
        double l[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) { const float lg = lh[2 * lane + e]; l[e] = lg < -110.0f ? -110.0 : (double)lg; }
        l[1] += l[0];
        double before = l[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        const double last = __shfl_sync(0xffffffffu, before, 31);
        before = __shfl_up_sync(0xffffffffu, before, 1);        // not before - l[1]: a NaN in l[1] would reach l[0]
        if (lane == 0) before = 0.0;
        float* num = reinterpret_cast<float*>(blob + DC_NUM);
        int fb = bad[2 * lane] != 0.f ? 2 * lane : bad[2 * lane + 1] != 0.f ? 2 * lane + 1 : DC_L;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) fb = min(fb, __shfl_xor_sync(0xffffffffu, fb, o));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int tt = 2 * lane + e;
            const double le = before + l[e];
            const float ex = expf((float)le);
            lh[tt] = (float)le;
            ll[tt] = (float)(le - (double)(float)le);
            num[tt] = ex * ik[tt];
            num[DC_L + tt] = beta[tt];
            num[2 * DC_L + tt] = ex * iq[tt];
            num[3 * DC_L + tt] = expf((float)(last - le)) * ik[tt];
        }
        if (lane == 0) {
            *first_bad = fb;
            num[4 * DC_L] = expf((float)last);
            reinterpret_cast<int*>(num)[4 * DC_L + 1] = fb;
        }
    }
    __syncthreads();
    const int fb = *first_bad;                                  // from that token on nothing is used: the walk sets the results
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
    for (int job = warp; job < 20; job += 8) {
        const int tile = job >> 1, weights = job & 1;           // K K^T, or Q K^T
        const int i = tile < 1 ? 0 : tile < 3 ? 1 : tile < 6 ? 2 : 3, j = tile - dc_tri(i);
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        const unsigned a_addr = pb_smem_addr((weights ? qs : ks) + 16 * i * Z::LDK + pb_a_offset(lane, Z::LDK));
        const unsigned b_addr = pb_smem_addr(ks + 16 * j * Z::LDK + pb_b_offset(lane, Z::LDK));
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            unsigned a[4], b[4];
            pb_ldmatrix_x4(a, a_addr + k * 32);
            pb_ldmatrix_x4(b, b_addr + k * 32);
            pb_mma(acc[0], a, b[0], b[1]);
            pb_mma(acc[1], a, b[2], b[3]);
        }
        unsigned m[3][4];
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            float out[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 16 * i + r0 + (e >> 1) * 8, s = 16 * j + 8 * v + c0 + (e & 1);
                float f = 0.f;
                if ((weights ? s <= t : s < t) && t < fb) f = expf((lh[t] - lh[s]) + (ll[t] - ll[s])) * (weights ? iq[t] : beta[t] * ik[t]) * ik[s];
                out[e] = f == 0.f ? 0.f : f * acc[v][e];
                if (!weights) A[t * Z::LDA + s] = out[e];
            }
            if (weights) {
                unsigned a[3], b[3];
                pb_split3(out[0], out[1], a);
                pb_split3(out[2], out[3], b);
#pragma unroll
                for (int p = 0; p < 3; ++p) { m[p][2 * v] = a[p]; m[p][2 * v + 1] = b[p]; }
            }
        }
        if (weights) {
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(blob + DC_TRI + tile * DC_TILE + (p * 32 + lane) * 16) = make_uint4(m[p][0], m[p][1], m[p][2], m[p][3]);
        }
    }
    __syncthreads();
    // (I + A)^-1: the 16 x 16 blocks of the diagonal a column a thread, then what lies below them block by block
    if (tid < 64) {
        const int b = tid >> 4, c = tid & 15;
        const float* Ab = A + (16 * b) * Z::LDA + 16 * b;
        float* Tb = Ti + (16 * b) * Z::LDA + 16 * b + c;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float s = r == c ? 1.f : 0.f;
#pragma unroll
            for (int k = 0; k < r; ++k) s = fmaf(-Ab[r * Z::LDA + k], x[k], s);
            x[r] = s;
            Tb[r * Z::LDA] = s;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 2; ++it) {                            // block rows 1 and 3: 16 x 16 below the diagonal of each pair
        const int r = tid >> 4, c = tid & 15, o = 32 * it;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) s = fmaf(A[(o + 16 + r) * Z::LDA + o + k], Ti[(o + k) * Z::LDA + o + c], s);
        X[(16 * it + r) * Z::LDX + c] = s;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const int r = tid >> 4, c = tid & 15, o = 32 * it;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) s = fmaf(-Ti[(o + 16 + r) * Z::LDA + o + 16 + k], X[(16 * it + k) * Z::LDX + c], s);
        Ti[(o + 16 + r) * Z::LDA + o + c] = s;
    }
    for (int idx = tid; idx < 256; idx += 256) {                // above the diagonal of each pair: zeros
        const int r = idx >> 4, c = idx & 15;
        Ti[r * Z::LDA + 16 + c] = 0.f;
        Ti[(32 + r) * Z::LDA + 48 + c] = 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int r = (tid >> 5) + 8 * it, c = tid & 31;
        float s = 0.f;
#pragma unroll 8
        for (int k = 0; k < 32; ++k) s = fmaf(A[(32 + r) * Z::LDA + k], Ti[k * Z::LDA + c], s);
        X[r * Z::LDX + c] = s;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int r = (tid >> 5) + 8 * it, c = tid & 31;
        float s = 0.f;
#pragma unroll 8
        for (int k = 0; k < 32; ++k) s = fmaf(-Ti[(32 + r) * Z::LDA + 32 + k], X[k * Z::LDX + c], s);
        Ti[(32 + r) * Z::LDA + c] = s;
    }
    __syncthreads();
    for (int idx = tid; idx < 10 * 32; idx += 256) {
        const int tile = idx >> 5;
        const int i = tile < 1 ? 0 : tile < 3 ? 1 : tile < 6 ? 2 : 3, j = tile - dc_tri(i);
        const float* src = Ti + (16 * i + r0) * Z::LDA + 16 * j + c0;      // idx & 31 is the lane
        unsigned m[4][3];
        pb_split3(src[0], src[1], m[0]);
        pb_split3(src[8 * Z::LDA], src[8 * Z::LDA + 1], m[1]);
        pb_split3(src[8], src[9], m[2]);
        pb_split3(src[8 * Z::LDA + 8], src[8 * Z::LDA + 9], m[3]);
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint4*>(blob + tile * DC_TILE + (p * 32 + lane) * 16) = make_uint4(m[0][p], m[1][p], m[2][p], m[3][p]);
    }
}

template <int D, int PB>
struct DcLayout {
    static constexpr int LDK = D + 8, LDP = PB + 8;
    static constexpr int k = 0, q = k + DC_L * LDK * 2, v = q + DC_L * LDK * 2, blob = v + DC_L * LDP * 2, half = blob + DC_BLOB;
    static constexpr int s = 2 * half, r = s + 3 * D * LDP * 2, u = r + 3 * DC_L * LDP * 2, w = u + 3 * DC_L * LDP * 2, bad = w + 3 * DC_L * LDP * 2;
    static constexpr int bytes = bad + 2 * PB * 4;
    static_assert(half % 16 == 0 && blob % 16 == 0 && s % 16 == 0 && bytes <= 227 * 1024, "shared memory");
};

// The walk over a head's chunks.  A block is one head's state [D, PB columns] and twelve warps.  Warps 8-11 fetch the next
// chunk's K, Q, V and what the first kernel left while the others work.  Warps 0-3 make K S and from it R, warps 4-7 Q S; all
// eight make U (a row tile and half of the columns each); then warps 4-7 finish the outputs and warps 0-3 the state, which lives in
// their registers from chunk to chunk.
template <int D, int PB>
__device__ __forceinline__ void dc_sequence(unsigned char* dw_sm, const bf16* u, long long ld_u, const unsigned char* blobs, float* state, float* y, const int32_t* cu_q,
                                            int seq, int least, int slot, int h, int p_first, int H, int G, int E) {
    using Z = DcLayout<D, PB>;
    const int g = h / (H / G);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int first = cu_q[seq], n_tok = cu_q[seq + 1] - first;
    const int n_chunks = (n_tok + DC_L - 1) / DC_L;

    if (tid >= DC_MUL) {
        const int pt = tid - DC_MUL;
        const unsigned char* blob = blobs + ((size_t)pb_chunks_before<DC_L>(cu_q, seq, least, lane) * H + h) * DC_BLOB;
        auto fetch = [&](int ch) {
            unsigned char* buf = dw_sm + (ch & 1) * Z::half;
            const int t0 = ch * DC_L, cnt = min(DC_L, n_tok - t0);
            const bf16* rows = u + (size_t)(first + t0) * ld_u;
            const unsigned char* from = blob + (size_t)ch * H * DC_BLOB;
            for (int o = pt * 16; o < DC_BLOB; o += 128 * 16) pb_cp_async16(buf + Z::blob + o, from + o);
            bf16* ks = reinterpret_cast<bf16*>(buf + Z::k);
            bf16* qs = reinterpret_cast<bf16*>(buf + Z::q);
            bf16* vs = reinterpret_cast<bf16*>(buf + Z::v);
            for (int idx = pt; idx < DC_L * (D / 8); idx += 128) {
                const int tt = idx / (D / 8), n = idx % (D / 8) * 8;
                if (tt < cnt) {
                    const bf16* row = rows + (size_t)tt * ld_u + (size_t)g * D + n;
                    pb_cp_async16(qs + tt * Z::LDK + n, row);
                    pb_cp_async16(ks + tt * Z::LDK + n, row + (size_t)G * D);
                } else {
                    *reinterpret_cast<uint4*>(qs + tt * Z::LDK + n) = *reinterpret_cast<uint4*>(ks + tt * Z::LDK + n) = make_uint4(0, 0, 0, 0);
                }
            }
            for (int idx = pt; idx < DC_L * (PB / 8); idx += 128) {
                const int tt = idx / (PB / 8), p = idx % (PB / 8) * 8;
                if (tt < cnt) pb_cp_async16(vs + tt * Z::LDP + p, rows + (size_t)tt * ld_u + (size_t)2 * G * D + (size_t)h * E + p_first + p);
                else *reinterpret_cast<uint4*>(vs + tt * Z::LDP + p) = make_uint4(0, 0, 0, 0);
            }
            pb_cp_async_wait();
        };
        fetch(0);
        __syncthreads();
        for (int ch = 0; ch < n_chunks; ++ch) {
            if (ch + 1 < n_chunks) fetch(ch + 1);
            __syncthreads();
        }
        return;
    }

    constexpr int PT = PB / 8, HT = PT / 2, ST = D / 64;        // n8 tiles of the columns, of half of them; 16-row state tiles of a warp 0-3
    const bool keys = warp < 4;
    const int i = keys ? warp : 7 - warp, half = warp >> 2;     // the long and the short row tiles share the schedulers
    const int r0 = lane >> 2, c0 = (lane & 3) * 2, ta = 16 * i + r0, tb = ta + 8;
    bf16* ss = reinterpret_cast<bf16*>(dw_sm + Z::s);
    bf16* rs = reinterpret_cast<bf16*>(dw_sm + Z::r);
    bf16* us = reinterpret_cast<bf16*>(dw_sm + Z::u);
    bf16* ws = reinterpret_cast<bf16*>(dw_sm + Z::w);
    int* bads = reinterpret_cast<int*>(dw_sm + Z::bad);
    const int n0 = ST * 16 * warp;                              // warps 0-3: first row of the state
    float* S = state + (((size_t)slot * H + h) * D + n0 + r0) * E + p_first + c0;
    float st[ST][PT][4];
#pragma unroll
    for (int a = 0; a < ST; ++a)
#pragma unroll
        for (int q = 0; q < PT; ++q) {
            const float2 x = keys ? *reinterpret_cast<const float2*>(S + (size_t)16 * a * E + q * 8) : make_float2(0.f, 0.f);
            const float2 z = keys ? *reinterpret_cast<const float2*>(S + (size_t)(16 * a + 8) * E + q * 8) : make_float2(0.f, 0.f);
            st[a][q][0] = x.x; st[a][q][1] = x.y; st[a][q][2] = z.x; st[a][q][3] = z.y;
        }
    // rows r, r + 8 of columns q * 8 + c0, + 1 of a [3 parts][rows][LDP] matrix
    auto put = [&](bf16* m, int rows, int r, int q, float x0, float x1, float z0, float z1) {
        unsigned a[3], b[3];
        pb_split3(x0, x1, a);
        pb_split3(z0, z1, b);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            unsigned* dst = reinterpret_cast<unsigned*>(m + (p * rows + r) * Z::LDP + q * 8 + c0);
            dst[0] = a[p];
            dst[8 * Z::LDP / 2] = b[p];
        }
    };
    auto put_state = [&]() {
#pragma unroll
        for (int a = 0; a < ST; ++a)
#pragma unroll
            for (int q = 0; q < PT; ++q) put(ss, D, n0 + 16 * a + r0, q, st[a][q][0], st[a][q][1], st[a][q][2], st[a][q][3]);
    };
    if (keys) put_state();
    for (int idx = tid; idx < 2 * PB; idx += DC_MUL) bads[idx] = DC_L;
    __syncthreads();
    const unsigned bt = pb_bt_offset(lane, Z::LDP) * 2;
    const unsigned s_addr = pb_smem_addr(ss) + bt, r_addr = pb_smem_addr(rs) + bt + half * HT * 16, u_addr = pb_smem_addr(us) + bt, w_addr = pb_smem_addr(ws) + bt;
    for (int ch = 0; ch < n_chunks; ++ch) {
        const unsigned char* buf = dw_sm + (ch & 1) * Z::half;
        const uint4* tri = reinterpret_cast<const uint4*>(buf + Z::blob);
        const float* num = reinterpret_cast<const float*>(buf + Z::blob + DC_NUM);
        int* bad = bads + (ch & 1) * PB;
        const int t0 = ch * DC_L, cnt = min(DC_L, n_tok - t0);
        const int fb = reinterpret_cast<const int*>(num)[4 * DC_L + 1];
        // K S (warps 0-3) and Q S (warps 4-7), the small parts of the state summed on their own
        float o[PT][4];
        {
            float part[2][PT][4];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int q = 0; q < PT; ++q) part[p][q][0] = part[p][q][1] = part[p][q][2] = part[p][q][3] = 0.f;
            const unsigned a_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + (keys ? Z::k : Z::q)) + 16 * i * Z::LDK + pb_a_offset(lane, Z::LDK));
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
                unsigned a[4];
                pb_ldmatrix_x4(a, a_addr + k * 32);
#pragma unroll
                for (int p = 2; p >= 0; --p)
#pragma unroll
                    for (int q = 0; q < PT; q += 2) {
                        unsigned b[4];
                        pb_ldmatrix_x4_trans(b, s_addr + ((p * D + k * 16) * Z::LDP + q * 8) * 2);
                        pb_mma(part[p ? 1 : 0][q], a, b[0], b[1]);
                        pb_mma(part[p ? 1 : 0][q + 1], a, b[2], b[3]);
                    }
            }
            const float fa = num[(keys ? 0 : 2 * DC_L) + ta], fb2 = num[(keys ? 0 : 2 * DC_L) + tb];
#pragma unroll
            for (int q = 0; q < PT; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[q][e] = (part[1][q][e] + part[0][q][e]) * (e < 2 ? fa : fb2);
        }
        if (keys) {
            const float ba = num[DC_L + ta], bb = num[DC_L + tb];
            const bf16* vs = reinterpret_cast<const bf16*>(buf + Z::v) + c0;
#pragma unroll
            for (int q = 0; q < PT; ++q) {
                const float2 va = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vs + ta * Z::LDP + q * 8));
                const float2 vb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vs + tb * Z::LDP + q * 8));
                float r[4] = {ba * (va.x - o[q][0]), ba * (va.y - o[q][1]), bb * (vb.x - o[q][2]), bb * (vb.y - o[q][3])};
                // a number that is not finite would reach earlier tokens through the zeros above the diagonal: it is taken out
                // here, and its column's results from its token on are set when they are stored
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!isfinite(r[e])) { r[e] = 0.f; atomicMin(bad + q * 8 + c0 + (e & 1), e < 2 ? ta : tb); }
                put(rs, DC_L, ta, q, r[0], r[1], r[2], r[3]);
            }
        }
        pb_named_barrier(1, DC_MUL);                                               // R is there; the state's parts have been read
        {
            float big[HT][4], small[HT][4];
#pragma unroll
            for (int q = 0; q < HT; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) big[q][e] = small[q][e] = 0.f;
            const uint4* row = tri + dc_tri(i) * (DC_TILE / 16) + lane;
            for (int j = 0; j <= i; ++j) {
                unsigned a[3][4], b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const uint4 f = row[(j * 3 + p) * 32];
                    a[p][0] = f.x; a[p][1] = f.y; a[p][2] = f.z; a[p][3] = f.w;
                    if constexpr (HT == 2) pb_ldmatrix_x4_trans(b[p], r_addr + (p * DC_L + j * 16) * Z::LDP * 2);
                    else pb_ldmatrix_x2_trans(b[p][0], b[p][1], r_addr + (p * DC_L + j * 16) * Z::LDP * 2);
                }
#pragma unroll
                for (int q = 0; q < HT; ++q) {
                    const unsigned bq[3][2] = {{b[0][2 * q], b[0][2 * q + 1]}, {b[1][2 * q], b[1][2 * q + 1]}, {b[2][2 * q], b[2][2 * q + 1]}};
                    pb_mma6(big[q], small[q], a, bq);
                }
            }
            const float wa = num[3 * DC_L + ta], wb = num[3 * DC_L + tb];
#pragma unroll
            for (int q = 0; q < HT; ++q) {
                float x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = small[q][e] + big[q][e];
                put(us, DC_L, ta, half * HT + q, x[0], x[1], x[2], x[3]);
                put(ws, DC_L, ta, half * HT + q, x[0] * wa, x[1] * wa, x[2] * wb, x[3] * wb);
            }
            if (tid < PB) bads[((ch + 1) & 1) * PB + tid] = DC_L;                  // read last in the chunk before
        }
        pb_named_barrier(1, DC_MUL);                                               // U is there
        if (!keys) {
            if (16 * i < cnt) {
                float big[PT][4], small[PT][4];
#pragma unroll
                for (int q = 0; q < PT; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) big[q][e] = small[q][e] = 0.f;
                const uint4* row = tri + (DC_TRI / 16) + dc_tri(i) * (DC_TILE / 16) + lane;
                for (int j = 0; j <= i; ++j) {
                    unsigned a[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 f = row[(j * 3 + p) * 32];
                        a[p][0] = f.x; a[p][1] = f.y; a[p][2] = f.z; a[p][3] = f.w;
                    }
#pragma unroll
                    for (int q = 0; q < PT; q += 2) {
                        unsigned b[3][4];
#pragma unroll
                        for (int p = 0; p < 3; ++p) pb_ldmatrix_x4_trans(b[p], u_addr + ((p * DC_L + j * 16) * Z::LDP + q * 8) * 2);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const unsigned bq[3][2] = {{b[0][2 * e], b[0][2 * e + 1]}, {b[1][2 * e], b[1][2 * e + 1]}, {b[2][2 * e], b[2][2 * e + 1]}};
                            pb_mma6(big[q + e], small[q + e], a, bq);
                        }
                    }
                }
                float* dst = y + (size_t)(first + t0 + ta) * ((size_t)H * E) + (size_t)h * E + p_first + c0;
#pragma unroll
                for (int q = 0; q < PT; ++q) {
                    const int fx = min(fb, bad[q * 8 + c0]), fy = min(fb, bad[q * 8 + c0 + 1]);
                    float x[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] = o[q][e] + (small[q][e] + big[q][e]);
                    if (ta >= fx) x[0] = NAN;
                    if (ta >= fy) x[1] = NAN;
                    if (tb >= fx) x[2] = NAN;
                    if (tb >= fy) x[3] = NAN;
                    if (ta < cnt) *reinterpret_cast<float2*>(dst + q * 8) = make_float2(x[0], x[1]);
                    if (tb < cnt) *reinterpret_cast<float2*>(dst + (size_t)8 * H * E + q * 8) = make_float2(x[2], x[3]);
                }
            }
        } else {
            const float tot = num[4 * DC_L];
#pragma unroll
            for (int a = 0; a < ST; ++a) {
                float big[PT][4], small[PT][4];
#pragma unroll
                for (int q = 0; q < PT; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) big[q][e] = small[q][e] = 0.f;
                const unsigned k_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::k) + n0 + 16 * a + pb_at_offset(lane, Z::LDK));
#pragma unroll
                for (int k = 0; k < DC_L / 16; ++k) {
                    unsigned f[4];
                    pb_ldmatrix_x4_trans(f, k_addr + k * 16 * Z::LDK * 2);
#pragma unroll
                    for (int p = 2; p >= 0; --p)
#pragma unroll
                        for (int q = 0; q < PT; q += 2) {
                            unsigned b[4];
                            pb_ldmatrix_x4_trans(b, w_addr + ((p * DC_L + k * 16) * Z::LDP + q * 8) * 2);
                            pb_mma(p ? small[q] : big[q], f, b[0], b[1]);
                            pb_mma(p ? small[q + 1] : big[q + 1], f, b[2], b[3]);
                        }
                }
#pragma unroll
                for (int q = 0; q < PT; ++q) {
                    const bool bx = min(fb, bad[q * 8 + c0]) < DC_L, by = min(fb, bad[q * 8 + c0 + 1]) < DC_L;
#pragma unroll
                    for (int e = 0; e < 4; ++e) st[a][q][e] = ((e & 1) ? by : bx) ? NAN : fmaf(tot, st[a][q][e], small[q][e] + big[q][e]);
                }
            }
            put_state();
        }
        __syncthreads();
    }
    if (keys) {
#pragma unroll
        for (int a = 0; a < ST; ++a)
#pragma unroll
            for (int q = 0; q < PT; ++q) {
                *reinterpret_cast<float2*>(S + (size_t)16 * a * E + q * 8) = make_float2(st[a][q][0], st[a][q][1]);
                *reinterpret_cast<float2*>(S + (size_t)(16 * a + 8) * E + q * 8) = make_float2(st[a][q][2], st[a][q][3]);
            }
    }
}

template <int D, int PB, bool RECORDED>
__global__ void __launch_bounds__(DC_ALL, 1)
delta_walk_kernel(const bf16* u, long long ld_u, const unsigned char* blobs, float* state, float* y, const int32_t* cu_q, const int32_t* slots, PbSequences which,
                  int H, int G, int E) {
    extern __shared__ __align__(16) unsigned char dw_sm[];
    pb_grid_dep_launch();
    const int slices = E / PB;
    const int h = blockIdx.x / slices, p_first = (blockIdx.x % slices) * PB;
    pb_grid_dep_wait();
    pb_for_sequences<RECORDED>(cu_q, which, [&](int seq, int least) {
        dc_sequence<D, PB>(dw_sm, u, ld_u, blobs, state, y, cu_q, seq, least, slots[seq], h, p_first, H, G, E);
    });
}

struct DcCall {
    const void *u, *b, *a;
    long long ld_u, ld_b, ld_a;
    const float *a_log, *dt_bias;
    float *state, *y;
    const int32_t *cu_q, *slots;
    void* scratch;
    int n_chunks, n_long, counted, longest, H, G, E;
    PbSequences all;
    cudaStream_t stream;
};

template <int D, int PB, bool RECORDED>
int dc_walk(const DcCall& c, int rows, const PbSequences& which) {
    constexpr int bytes = DcLayout<D, PB>::bytes;
    static const cudaError_t set = cudaFuncSetAttribute(delta_walk_kernel<D, PB, RECORDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    PB_REQUIRE(set == cudaSuccess, "gated_delta_scan_chunked: %s", cudaGetErrorString(set));
    pb_launch(delta_walk_kernel<D, PB, RECORDED>, dim3(c.H * (c.E / PB), rows), dim3(DC_ALL), bytes, c.stream, (const bf16*)c.u, c.ld_u, (const unsigned char*)c.scratch,
              c.state, c.y, c.cu_q, c.slots, which, c.H, c.G, c.E);
    PB_CHECK_LAUNCH("gated_delta_scan_chunked");
    return 0;
}

template <int D>
int dc_run(const DcCall& c) {
    constexpr int bytes = DcPrep<D>::bytes;
    static const cudaError_t set = cudaFuncSetAttribute(delta_prepare_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    PB_REQUIRE(set == cudaSuccess, "gated_delta_scan_chunked: %s", cudaGetErrorString(set));
    pb_launch(delta_prepare_kernel<D>, dim3(c.n_chunks, c.H), dim3(256), bytes, c.stream, (const bf16*)c.u, c.ld_u, (const bf16*)c.b, c.ld_b, (const bf16*)c.a,
              c.ld_a, c.a_log, c.dt_bias, c.cu_q, (unsigned char*)c.scratch, c.all.n_seqs, c.all.from, c.all.few, c.all.beside, c.H, c.G);
    PB_CHECK_LAUNCH("gated_delta_scan_chunked");
    // Where the lengths are at hand: the slices for which the longest chain, or all chains over the multiprocessors, takes less.  A chunk of 16 columns
    // takes 0.62 of what one of 32 does.  us, slices of 16 / 32 columns: 16 heads, 592 and 1,185 tokens 74 / 86; 1,333 and 2,667 158 / 191; one of
    // 1,000 41 / 72; 32 heads, 592 and 1,185 145 / 132, one of 1,000 80 / 73.
    int narrowest = 16, widest = 32;
    if (c.counted && c.longest > 0 && c.E % 32 == 0) {
        auto takes = [&](int width) {
            const double chain = (c.longest + DC_L - 1) / DC_L, all = (double)c.n_chunks * c.H * (c.E / width) / pb_multiprocessors();
            return (width == 16 ? 0.62 : 1.0) * (chain > all ? chain : all);
        };
        narrowest = widest = takes(16) < takes(32) ? 16 : 32;
    }
    return pb_for_widths(c.H, c.E, narrowest, widest, c.all, c.n_long, c.counted, [&](int width, int rows, const PbSequences& which) {
        if (which.recorded) return width == 32 ? dc_walk<D, 32, true>(c, rows, which) : dc_walk<D, 16, true>(c, rows, which);
        return width == 32 ? dc_walk<D, 32, false>(c, rows, which) : dc_walk<D, 16, false>(c, rows, which);
    });
}

}  // namespace

// Whether pb_gated_delta_scan_chunked takes these sizes and operands: rows and values in 16-byte pieces, keys of 64 or 128 elements,
// state and result in 8-byte pieces (pb_gated_delta_scan takes any).
PB_API int pb_gated_delta_chunked_takes(const void* u, long long ld_u, const float* state, const float* y, int H, int G, int D, int E) {
    return (D == 64 || D == 128) && E > 0 && E % 16 == 0 && H > 0 && H < 65536 && G > 0 && H % G == 0 && ld_u % 8 == 0 && pb_aligned(u, 16) &&
                   pb_aligned(state, 8) && pb_aligned(y, 8)
               ? 1
               : 0;
}
// Most chunks that n_tokens of n_long sequences can form, and the scratch memory (16-byte aligned) that the call needs for them.
PB_API int pb_gated_delta_chunks(int n_tokens, int n_long) { return n_tokens / DC_L + (n_long < n_tokens ? n_long : n_tokens); }
PB_API long long pb_gated_delta_chunk_bytes(int n_chunks, int H) { return (long long)n_chunks * H * DC_BLOB; }

// Operands as for pb_gated_delta_scan, bfloat16, for the sequences of at least `least` tokens; pb_gated_delta_scan with `below` = least
// does the others.  n_chunks and scratch as the two functions above say; n_long: how many such sequences there are (`counted`), or the
// most there can be, for a step that is being recorded (few, beside: sequences.cuh).
PB_API int pb_gated_delta_scan_chunked(const void* u, long long ld_u, const void* b_in, long long ld_b, const void* a_in, long long ld_a, const float* a_log,
                                       const float* dt_bias, float* state, float* y, const int32_t* cu_q, const int32_t* slots, void* scratch, int n_chunks,
                                       int n_seqs, int least, int few, int beside, int n_long, int counted, long long order, int longest, int H, int G, int D, int E,
                                       cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && n_chunks >= 0 && pb_gated_delta_chunked_takes(u, ld_u, state, y, H, G, D, E), "gated_delta_scan_chunked: %d over %d heads of %d, %d", H, G, D, E);
    PB_REQUIRE(u && b_in && a_in && a_log && dt_bias && state && y && cu_q && slots && scratch, "gated_delta_scan_chunked: null pointer");
    PB_REQUIRE(ld_u >= 2ll * G * D + (long long)H * E && ld_b >= H && ld_a >= H, "gated_delta_scan_chunked: rows too short");
    PB_REQUIRE(pb_aligned(scratch, 16), "gated_delta_scan_chunked: misaligned operands");
    PB_REQUIRE(least > 0 && n_long >= 0 && n_long <= n_seqs && n_long < 65536, "gated_delta_scan_chunked: %d of %d sequences in one launch", n_long, n_seqs);
    if (n_long == 0 || n_chunks == 0) return 0;
    const DcCall c{u, b_in, a_in, ld_u, ld_b, ld_a, a_log, dt_bias, state, y, cu_q, slots, scratch, n_chunks, n_long, counted, longest, H, G, E,
                   PbSequences{n_seqs, least, INT_MAX, few, beside, 0, 0, 0, 0, longest > 0, (unsigned long long)order}, stream};
    return D == 128 ? dc_run<128>(c) : dc_run<64>(c);
}
