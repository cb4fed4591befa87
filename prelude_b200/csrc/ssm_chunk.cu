// The state-space recurrence of a prompt step by chunks of 64 tokens, on the tensor cores:
//
//   pb_ssm_scan_chunked   as pb_ssm_scan: dt = softplus(dt + bias); S <- exp(-exp(A_log) dt) S + dt B x^T; y = S^T C + D x
//
// With l_t the sum of the logarithms of the decays up to token t of the chunk and S the state before it,
//     y_t = exp(l_t) S^T C_t + sum_{s <= t} (C_t . B_s) exp(l_t - l_s) dt_s x_s + D x_t
//     S'  = exp(l_last) S + sum_s exp(l_last - l_s) dt_s B_s x_s^T
// four products a chunk: C B^T (operands as they are, bfloat16: exact products), the masked weights times x, C times the state,
// and B^T times the weighted x.  Everything that is not bfloat16 in memory - the weights, the state, the weighted x - enters
// a product as three bfloat16 numbers whose sum it is (mma_sync.cuh), every sum is float32, and the sums of logarithms are taken
// in 64-bit and kept as a float32 pair, so that the difference of two large ones is as good as the decays' product.
// No exponent is positive.  A decay below exp(-110) counts as exp(-110), which is zero in float32.
//
// What bounds it: the chain of chunks (a block owns a head's state and cannot start a chunk before the one ahead is done) and, in
// a chunk, the warp products and the operand loads from shared memory that feed them.  2,048 tokens, state 128 x 64: 64 heads
// (128 blocks of 32 columns) 114 us against 481 token by token on the float32 units (pb_ssm_scan), 128 heads (128 blocks of 64)
// 164 against 962; 64 heads, 64 tokens from memory 14 against 27, 32 tokens 12 against 18.  Error against 64-bit where decays are slow (a
// step of 1e-3): output 1.4 to 1.8e-7 (token by token 1.6e-7 to 1.3e-6: the more tokens a decay leaves, the more roundings pile up
// there), state 0.3 to 2.6e-7 (2.2e-7 to 5.6e-6); where they are fast (0.05 and more) it is up to twice the tokens' in their place:
// 0.9 to 1.7e-7 (0.9 to 1.1e-7), state 0.5 to 1.3e-7 (0.5 to 1.2e-7).
//
// A block is one head's state [N, PB columns] and twelve warps.  Warps 8-11 fetch: while the others work on one chunk they
// bring the next chunk's B, C and x into the other half of shared memory and make its sums of logarithms and its weighted x.
// Warps 0-7 multiply: warp (i, f) makes rows 16 i .. 16 i + 15 of y from half f of the state's rows and from the 16-token tiles
// f and f + 2 of x (what lies above the diagonal is skipped; tiles i are dealt to the schedulers long with short); the two halves
// are added through shared memory.  For the state warp w owns rows 16 w .. 16 w + 15, in registers from chunk to chunk.
#include "mma_sync.cuh"
#include "sequences.cuh"

#include <math.h>

namespace {

typedef __nv_bfloat16 bf16;

constexpr int SC_L = 64;                        // tokens of a chunk
constexpr int SC_MUL = 256, SC_ALL = 384;       // multiplying threads, all threads

template <int N, int PB>
struct ScLayout {
    static constexpr int LDN = N + 8, LDP = PB + 8, LDY = PB + 4;                  // row strides: 16-byte pieces of eight rows in eight bank groups
    static constexpr int b = 0, c = b + SC_L * LDN * 2, x = c + SC_L * LDN * 2, xw = x + SC_L * LDP * 2, num = xw + 3 * SC_L * LDP * 2;
    static constexpr int bad = num + (4 * SC_L + 4) * 4, half = bad + PB * 4;      // l (high, low), dt, exp(l), exp(l_last); first token that is not finite
    static constexpr int s = 2 * half, yx = s + 3 * N * LDP * 2, bytes = yx + SC_L * LDY * 4;
    static_assert(half % 16 == 0 && bytes <= 227 * 1024, "shared memory");
};

// One sequence's tokens through one head's columns p_first ..; all threads of the block.
template <int N, int PB>
__device__ __forceinline__ void sc_sequence(unsigned char* sc_sm, const bf16* u, const bf16* dt_in, long long ld_dt, float neg_a, float bias, float skip, float* state,
                                            float* y, int first, int n_tok, int slot, int h, int p_first, int heads, int P, int groups) {
    using Z = ScLayout<N, PB>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int inner = heads * P, channels = inner + 2 * groups * N;
    const int g = h / (heads / groups);
    const int n_chunks = (n_tok + SC_L - 1) / SC_L;

    if (tid >= SC_MUL) {
        const int pw = warp - SC_MUL / 32, pt = tid - SC_MUL;
        auto fetch = [&](int ch) {
            unsigned char* buf = sc_sm + (ch & 1) * Z::half;
            const int t0 = ch * SC_L, cnt = min(SC_L, n_tok - t0);
            const bf16* rows = u + (size_t)(first + t0) * channels;
            bf16* bs = reinterpret_cast<bf16*>(buf + Z::b);
            bf16* cs = reinterpret_cast<bf16*>(buf + Z::c);
            for (int idx = pt; idx < SC_L * (N / 8); idx += 128) {
                const int tt = idx / (N / 8), n = idx % (N / 8) * 8;
                bf16* bd = bs + tt * Z::LDN + n;
                bf16* cd = cs + tt * Z::LDN + n;
                if (tt < cnt) {
                    const bf16* row = rows + (size_t)tt * channels + inner + g * N + n;
                    pb_cp_async16(bd, row);
                    pb_cp_async16(cd, row + groups * N);
                } else {
                    *reinterpret_cast<uint4*>(bd) = *reinterpret_cast<uint4*>(cd) = make_uint4(0, 0, 0, 0);
                }
            }
            // x: warp pw has tokens 16 pw .. + 15
            constexpr int PIECES = PB / 8, X_IT = 16 * PIECES / 32;
            uint4 xr[X_IT];
#pragma unroll
            for (int it = 0; it < X_IT; ++it) {
                const int idx = it * 32 + lane, tt = pw * 16 + idx / PIECES, p = idx % PIECES * 8;
                xr[it] = tt < cnt ? *reinterpret_cast<const uint4*>(rows + (size_t)tt * channels + h * P + p_first + p) : make_uint4(0, 0, 0, 0);
            }
            // step sizes of tokens 2 lane, 2 lane + 1 and the sums of logarithms up to them (every warp makes them for itself)
            float dt[2];
            double l[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tt = 2 * lane + e;
                dt[e] = tt < cnt ? pb_softplus(pb_ld(dt_in + (size_t)(first + t0 + tt) * ld_dt + h) + bias) : 0.f;
                const float a = neg_a * dt[e];
                l[e] = a < -110.0f ? -110.0 : (double)a;                          // a token past the end: decay 1
            }
            l[1] += l[0];
            double before = l[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double v = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += v;
            }
            const double last = __shfl_sync(0xffffffffu, before, 31);
            before = __shfl_up_sync(0xffffffffu, before, 1);                      // not before - l[1]: a NaN in l[1] would reach l[0]
            if (lane == 0) before = 0.0;
            float w[2];
            float* num = reinterpret_cast<float*>(buf + Z::num);
            int* bad = reinterpret_cast<int*>(buf + Z::bad);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double le = before + l[e];
                w[e] = expf((float)(last - le)) * dt[e];
                if (pw == 0) {
                    const int tt = 2 * lane + e;
                    num[tt] = (float)le;
                    num[SC_L + tt] = (float)(le - (double)(float)le);
                    num[2 * SC_L + tt] = dt[e];
                    num[3 * SC_L + tt] = expf((float)le);
                    if (tt == SC_L - 1) num[4 * SC_L] = expf((float)last);
                }
            }
            for (int p = pt; p < PB; p += 128) bad[p] = SC_L;
            pb_named_barrier(2, SC_ALL - SC_MUL);
            bf16* xs = reinterpret_cast<bf16*>(buf + Z::x);
            bf16* xw = reinterpret_cast<bf16*>(buf + Z::xw);
#pragma unroll
            for (int it = 0; it < X_IT; ++it) {
                const int idx = it * 32 + lane, tt = pw * 16 + idx / PIECES, p = idx % PIECES * 8;
                const float w0 = __shfl_sync(0xffffffffu, w[0], tt >> 1), w1 = __shfl_sync(0xffffffffu, w[1], tt >> 1);
                const float wt = (tt & 1) ? w1 : w0;
                unsigned raw[4] = {xr[it].x, xr[it].y, xr[it].z, xr[it].w};
                unsigned parts[3][4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[e]));
                    unsigned part[3];
                    pb_split3(f.x * wt, f.y * wt, part);
                    parts[0][e] = part[0]; parts[1][e] = part[1]; parts[2][e] = part[2];
                    // a value that is not finite would reach the tokens before it through the masked weights' zeros: it is
                    // taken out here, and the outputs from its token on are set when they are stored
                    if (!isfinite(f.x)) { raw[e] &= 0xffff0000u; atomicMin(bad + p + 2 * e, tt); }
                    if (!isfinite(f.y)) { raw[e] &= 0x0000ffffu; atomicMin(bad + p + 2 * e + 1, tt); }
                }
                *reinterpret_cast<uint4*>(xs + tt * Z::LDP + p) = make_uint4(raw[0], raw[1], raw[2], raw[3]);
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    *reinterpret_cast<uint4*>(xw + (k * SC_L + tt) * Z::LDP + p) = make_uint4(parts[k][0], parts[k][1], parts[k][2], parts[k][3]);
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

    constexpr int PT = PB / 8, NK = N / 16;                                        // n8 tiles of columns; 16-wide pieces of the state's rows
    const int f = warp & 1, i = warp < 4 ? warp >> 1 : 3 - ((warp - 4) >> 1);
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
    const bool owns = warp < NK;                                                   // rows 16 warp .. + 15 of the state
    bf16* ss = reinterpret_cast<bf16*>(sc_sm + Z::s);
    float* yx = reinterpret_cast<float*>(sc_sm + Z::yx);
    float* S = state + (((size_t)slot * heads + h) * N + warp * 16 + r0) * P + p_first + c0;
    float st[PT][4];
#pragma unroll
    for (int q = 0; q < PT; ++q) {
        const float2 a = owns ? *reinterpret_cast<const float2*>(S + q * 8) : make_float2(0.f, 0.f);
        const float2 b = owns ? *reinterpret_cast<const float2*>(S + (size_t)8 * P + q * 8) : make_float2(0.f, 0.f);
        st[q][0] = a.x; st[q][1] = a.y; st[q][2] = b.x; st[q][3] = b.y;
    }
    auto put_state = [&]() {
        if (!owns) return;
#pragma unroll
        for (int q = 0; q < PT; ++q) {
            unsigned a[3], b[3];
            pb_split3(st[q][0], st[q][1], a);
            pb_split3(st[q][2], st[q][3], b);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                unsigned* dst = reinterpret_cast<unsigned*>(ss + (k * N + warp * 16 + r0) * Z::LDP + q * 8 + c0);
                dst[0] = a[k];
                dst[8 * Z::LDP / 2] = b[k];
            }
        }
    };
    put_state();
    __syncthreads();
    const unsigned s_addr = pb_smem_addr(ss + pb_bt_offset(lane, Z::LDP));
    for (int ch = 0; ch < n_chunks; ++ch) {
        const unsigned char* buf = sc_sm + (ch & 1) * Z::half;
        const float* num = reinterpret_cast<const float*>(buf + Z::num);
        const int t0 = ch * SC_L, cnt = min(SC_L, n_tok - t0);
        float acc[PT][4];
#pragma unroll
        for (int q = 0; q < PT; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.f;
        if (16 * i < cnt) {
            // C B^T of the warp's rows and its tiles of tokens; the half of C's columns that meets its half of the state stays
            float gt[2][2][4];
#pragma unroll
            for (int e = 0; e < 16; ++e) gt[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
            unsigned cf[NK / 2][4];
            const unsigned c_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::c) + 16 * i * Z::LDN + pb_a_offset(lane, Z::LDN));
            const unsigned b_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::b) + 16 * f * Z::LDN + pb_b_offset(lane, Z::LDN));
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int k0 = (half == 0 ? 1 - f : f) * (NK / 2);                 // the half that stays comes last
#pragma unroll
                for (int k = 0; k < NK / 2; ++k) {
                    pb_ldmatrix_x4(cf[k], c_addr + (k0 + k) * 32);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (f + 2 * j <= i) {
                            unsigned b[4];
                            pb_ldmatrix_x4(b, b_addr + j * 32 * Z::LDN * 2 + (k0 + k) * 32);
                            pb_mma(gt[j][0], cf[k], b[0], b[1]);
                            pb_mma(gt[j][1], cf[k], b[2], b[3]);
                        }
                }
            }
            // C times the state before the chunk, the small parts first
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int k = 0; k < NK / 2; ++k)
#pragma unroll
                    for (int q = 0; q < PT; q += 2) {
                        unsigned b[4];
                        pb_ldmatrix_x4_trans(b, s_addr + ((part * N + (f * (NK / 2) + k) * 16) * Z::LDP + q * 8) * 2);
                        pb_mma(acc[q], cf[k], b[0], b[1]);
                        pb_mma(acc[q + 1], cf[k], b[2], b[3]);
                    }
            const int ta = 16 * i + r0, tb = ta + 8;
            const float ea = num[3 * SC_L + ta], eb = num[3 * SC_L + tb];
#pragma unroll
            for (int q = 0; q < PT; ++q) { acc[q][0] *= ea; acc[q][1] *= ea; acc[q][2] *= eb; acc[q][3] *= eb; }
            // the weights of the tokens up to each, times x
            const float ha = num[ta], la = num[SC_L + ta], hb = num[tb], lb = num[SC_L + tb];
            const unsigned x_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::x) + pb_bt_offset(lane, Z::LDP));
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int tile = f + 2 * j;
                if (tile > i) continue;
                unsigned m[3][4];
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    float wgt[4];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int s = tile * 16 + v * 8 + c0 + e;
                        const float hs = num[s], ls = num[SC_L + s], dt = num[2 * SC_L + s];
                        wgt[e] = s <= ta ? gt[j][v][e] * (expf((ha - hs) + (la - ls)) * dt) : 0.f;
                        wgt[2 + e] = s <= tb ? gt[j][v][2 + e] * (expf((hb - hs) + (lb - ls)) * dt) : 0.f;
                        if (s == ta) wgt[e] += skip;
                        if (s == tb) wgt[2 + e] += skip;
                    }
                    unsigned a[3], b[3];
                    pb_split3(wgt[0], wgt[1], a);
                    pb_split3(wgt[2], wgt[3], b);
#pragma unroll
                    for (int k = 0; k < 3; ++k) { m[k][2 * v] = a[k]; m[k][2 * v + 1] = b[k]; }
                }
#pragma unroll
                for (int q = 0; q < PT; q += 2) {
                    unsigned b[4];
                    pb_ldmatrix_x4_trans(b, x_addr + (tile * 16 * Z::LDP + q * 8) * 2);
#pragma unroll
                    for (int k = 2; k >= 0; --k) {
                        pb_mma(acc[q], m[k], b[0], b[1]);
                        pb_mma(acc[q + 1], m[k], b[2], b[3]);
                    }
                }
            }
            if (f == 1) {
                float* dst = yx + (16 * i + r0) * Z::LDY + c0;
#pragma unroll
                for (int q = 0; q < PT; ++q) {
                    *reinterpret_cast<float2*>(dst + q * 8) = make_float2(acc[q][0], acc[q][1]);
                    *reinterpret_cast<float2*>(dst + 8 * Z::LDY + q * 8) = make_float2(acc[q][2], acc[q][3]);
                }
            }
        }
        // the state behind the chunk: what the chunk adds is summed on its own (the tensor cores cut the sums' last bits off,
        // which must not pile up from chunk to chunk), then joins in one multiply-add
        if (owns) {
            float add[PT][4];
#pragma unroll
            for (int q = 0; q < PT; ++q) add[q][0] = add[q][1] = add[q][2] = add[q][3] = 0.f;
            unsigned bf[SC_L / 16][4];
            const unsigned b_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::b) + 16 * warp + pb_at_offset(lane, Z::LDN));
#pragma unroll
            for (int k = 0; k < SC_L / 16; ++k) pb_ldmatrix_x4_trans(bf[k], b_addr + k * 16 * Z::LDN * 2);
            const unsigned w_addr = pb_smem_addr(reinterpret_cast<const bf16*>(buf + Z::xw) + pb_bt_offset(lane, Z::LDP));
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int k = 0; k < SC_L / 16; ++k)
#pragma unroll
                    for (int q = 0; q < PT; q += 2) {
                        unsigned b[4];
                        pb_ldmatrix_x4_trans(b, w_addr + ((part * SC_L + k * 16) * Z::LDP + q * 8) * 2);
                        pb_mma(add[q], bf[k], b[0], b[1]);
                        pb_mma(add[q + 1], bf[k], b[2], b[3]);
                    }
            const float tot = num[4 * SC_L];
#pragma unroll
            for (int q = 0; q < PT; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) st[q][e] = fmaf(tot, st[q][e], add[q][e]);
        }
        pb_named_barrier(1, SC_MUL);                                               // the state before the chunk has been read, the halves of y are there
        if (f == 0 && 16 * i < cnt) {
            const int* bad = reinterpret_cast<const int*>(buf + Z::bad);
            const float* src = yx + (16 * i + r0) * Z::LDY + c0;
            float* dst = y + (size_t)(first + t0 + 16 * i + r0) * inner + h * P + p_first + c0;
#pragma unroll
            for (int q = 0; q < PT; ++q) {
                const int2 from = *reinterpret_cast<const int2*>(bad + q * 8 + c0);
                const float2 a = *reinterpret_cast<const float2*>(src + q * 8), b = *reinterpret_cast<const float2*>(src + 8 * Z::LDY + q * 8);
                float2 ya = make_float2(acc[q][0] + a.x, acc[q][1] + a.y), yb = make_float2(acc[q][2] + b.x, acc[q][3] + b.y);
                const int ta = 16 * i + r0, tb = ta + 8;
                if (ta >= from.x) ya.x = NAN;
                if (ta >= from.y) ya.y = NAN;
                if (tb >= from.x) yb.x = NAN;
                if (tb >= from.y) yb.y = NAN;
                if (ta < cnt) *reinterpret_cast<float2*>(dst + q * 8) = ya;
                if (tb < cnt) *reinterpret_cast<float2*>(dst + (size_t)8 * inner + q * 8) = yb;
            }
        }
        put_state();
        __syncthreads();
    }
    if (owns) {
#pragma unroll
        for (int q = 0; q < PT; ++q) {
            *reinterpret_cast<float2*>(S + q * 8) = make_float2(st[q][0], st[q][1]);
            *reinterpret_cast<float2*>(S + (size_t)8 * P + q * 8) = make_float2(st[q][2], st[q][3]);
        }
    }
}

template <int N, int PB, bool RECORDED>
__global__ void __launch_bounds__(SC_ALL, 1)
ssm_chunk_kernel(const bf16* u, const bf16* dt_in, long long ld_dt, const float* dt_bias, const float* a_log, const float* d_skip, float* state,
                 float* y, const int32_t* cu_q, const int32_t* slots, PbSequences which, int heads, int P, int groups) {
    extern __shared__ __align__(16) unsigned char sc_sm[];
    pb_grid_dep_launch();
    const int slices = P / PB;
    const int h = blockIdx.x / slices, p_first = (blockIdx.x % slices) * PB;
    const float neg_a = -expf(a_log[h]), bias = dt_bias[h], skip = d_skip[h];     // written by no kernel: before the wait
    pb_grid_dep_wait();
    pb_for_sequences<RECORDED>(cu_q, which, [&](int seq, int) {
        const int first = cu_q[seq];
        sc_sequence<N, PB>(sc_sm, u, dt_in, ld_dt, neg_a, bias, skip, state, y, first, cu_q[seq + 1] - first, slots[seq], h, p_first, heads, P, groups);
    });
}

template <int N, int PB, bool RECORDED>
int sc_launch(const void* u, const void* dt_in, long long ld_dt, const float* dt_bias, const float* a_log, const float* d_skip, float* state, float* y,
              const int32_t* cu_q, const int32_t* slots, const PbSequences& which, int rows, int heads, int P, int groups, cudaStream_t stream) {
    constexpr int bytes = ScLayout<N, PB>::bytes;
    static const cudaError_t set = cudaFuncSetAttribute(ssm_chunk_kernel<N, PB, RECORDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    PB_REQUIRE(set == cudaSuccess, "ssm_scan_chunked: %s", cudaGetErrorString(set));
    pb_launch(ssm_chunk_kernel<N, PB, RECORDED>, dim3(heads * (P / PB), rows), dim3(SC_ALL), bytes, stream, (const bf16*)u, (const bf16*)dt_in, ld_dt, dt_bias,
              a_log, d_skip, state, y, cu_q, slots, which, heads, P, groups);
    PB_CHECK_LAUNCH("ssm_scan_chunked");
    return 0;
}

}  // namespace

// Whether pb_ssm_scan_chunked takes these sizes and operands: rows in 16-byte pieces, state and result in 8-byte ones (pb_ssm_scan
// takes any).
PB_API int pb_ssm_scan_chunked_takes(const void* u, const float* state, const float* y, int heads, int P, int N, int groups) {
    return (N == 64 || N == 128) && P > 0 && P % 16 == 0 && heads > 0 && groups > 0 && heads % groups == 0 && pb_aligned(u, 16) && pb_aligned(state, 8) &&
                   pb_aligned(y, 8)
               ? 1
               : 0;
}

// Operands as for pb_ssm_scan, bfloat16, for the sequences of at least `least` tokens; pb_ssm_step does those of one.  n_long: how many
// there are (`counted`), or the most there can be, for a step that is being recorded (few, beside: sequences.cuh).
PB_API int pb_ssm_scan_chunked(const void* u, const void* dt_in, long long ld_dt, const float* dt_bias, const float* a_log, const float* d_skip,
                               float* state, float* y, const int32_t* cu_q, const int32_t* slots, int n_seqs, int least, int few, int beside, int n_long, int counted,
                               long long order, int longest, int heads, int P, int N, int groups, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && pb_ssm_scan_chunked_takes(u, state, y, heads, P, N, groups), "ssm_scan_chunked: %d heads of %d, state %d, %d groups", heads, P, N, groups);
    PB_REQUIRE(u && dt_in && dt_bias && a_log && d_skip && state && y && cu_q && slots && ld_dt >= heads, "ssm_scan_chunked: null pointer");
    PB_REQUIRE(least > 0 && n_long >= 0 && n_long <= n_seqs && n_long < 65536, "ssm_scan_chunked: %d of %d sequences in one launch", n_long, n_seqs);
    const PbSequences all{n_seqs, least, INT_MAX, few, beside, 0, 0, 0, 0, longest > 0, (unsigned long long)order};
    return pb_for_widths(heads, P, 16, 64, all, n_long, counted, [&](int width, int rows, const PbSequences& which) {
#define SC_ARGS u, dt_in, ld_dt, dt_bias, a_log, d_skip, state, y, cu_q, slots, which, rows, heads, P, groups, stream
#define SC_CASE(NN, PP) if (N == NN && width == PP) return which.recorded ? sc_launch<NN, PP, true>(SC_ARGS) : sc_launch<NN, PP, false>(SC_ARGS)
        SC_CASE(128, 64);
        SC_CASE(128, 32);
        SC_CASE(128, 16);
        SC_CASE(64, 64);
        SC_CASE(64, 32);
        SC_CASE(64, 16);
#undef SC_CASE
#undef SC_ARGS
        return pb_fail("ssm_scan_chunked: state %d", N);
    });
}

// For tests: the launches that pb_for_widths makes of a walk, four numbers each - width, rows, lo, hi; how many there are.
PB_API int pb_walk_launches(int heads, int cols, int narrowest, int widest, int n_long, int counted, int* out) {
    int n = 0;
    pb_for_widths(heads, cols, narrowest, widest, PbSequences{n_long, 1, INT_MAX, 0, 0, 0, 0, 0, 0, 0, 0}, n_long, counted, [&](int width, int rows, const PbSequences& which) {
        int* o = out + 4 * n++;
        o[0] = width; o[1] = rows; o[2] = which.lo; o[3] = which.hi;
        return 0;
    });
    return n;
}
