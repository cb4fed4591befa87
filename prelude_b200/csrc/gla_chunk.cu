// Gated linear attention over a prompt step by 16 tokens at a time, on the tensor cores:
//
//   pb_gla_scan_chunked   as pb_gla_scan (gla.cu): S <- diag(a) S + k v^T ; o = scale * S^T q
//
// With D_t the product of the decays up to token t of the sixteen, E_t that of the decays behind it (both per channel) and S the
// state before them,
//     o_t = S^T (D_t q_t) + sum_{s <= t} w_ts v_s,   w_ts = sum_n q_t[n] k_s[n] a_(s+1)[n] .. a_t[n]
//     S'  = diag(D_16) S + sum_s (E_s k_s) v_s^T
// Nothing but S depends on what lies before: one kernel makes, for all sixteens at once, the weights w - channel by channel on the
// float32 units, by moving every earlier key on by each token's decay: products of decays only, no quotient, so no decay is too
// small - and D_t q_t and E_s k_s in the order in which the products' operands lie in registers.  A second kernel walks a
// sequence's sixteens with three small products each.  v enters as it is (bfloat16: exact), everything that is float32 as three
// bfloat16 numbers whose sum it is (mma_sync.cuh; of nine products of two such operands the six that reach float32's last bit
// are taken); all sums are float32.
//
// What bounds it: the chain of sixteens.  Nothing but registers lies on it: a warp owns 16 channels of the state, transposed, as the
// sums of its own products, and the layout of those sums is the layout of the operand that the next sixteen's product with the
// queries wants.  The warps' shares of the outputs are added up by the fetching warps one sixteen later.  (With the operands made by
// the walk's fetching warps, once for every slice of the columns, 32 heads took 220 us instead of 177.)
//
// Measured against token by token (gla.cu), both kernels, heads of 128 x 128: 2,048 tokens 276 -> 177 us of 32 heads, 298 -> 148 of 16;
// 1,777 tokens of two sequences, 16 heads: 160 -> 100; 256 tokens of 32: 38 -> 31.  Error against 64 bits 0.6 - 1.9e-7 in the outputs and
// 0.01 - 2.0e-7 in the state (token by token 0.6 - 2.5e-7 and 0.01 - 2.6e-7; decays of 0.9 to 1 a tenth farther than they, of 0.99 to 1 a fifth nearer).  The walk issues in 46 % of the cycles, the tensor units work in
// 30 %: the rest is the fixed latencies of its chain.
#include "mma_sync.cuh"
#include "sequences.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int GC_L = 16;                                    // tokens at a time
constexpr int GC_STAGES = 4;                                // sixteens in shared memory: what the walk works on and three on their way
constexpr int GC_MUL = 256, GC_ALL = 384;                   // multiplying threads, all threads of the walk
// What the first kernel leaves for a sixteen and head: for every 16 channels the three parts of D q as an A operand [token][channel],
// then of E k as a B operand [token][channel], then the three parts of the weights as an A operand, 32 lanes x 16 bytes each, then
// the product of all sixteen decays per channel
template <int N>
struct GcBlob {
    static constexpr int q = 0, k = N / 16 * 3 * 512, w = 2 * k, d = w + 3 * 512, bytes = d + N * 4;
};

// Sum over the lanes of sixteen numbers a lane: every exchange halves the numbers a lane still holds.  Lane l ends with number
// (bit 4, bit 3, bit 2, bit 1 of l).
template <int HELD>
__device__ __forceinline__ void gc_halve(float (&v)[16], int lane) {
    const bool up = (lane & HELD) != 0;                     // 16 numbers: lanes 16 apart, 8: 8 apart, and so on
#pragma unroll
    for (int i = 0; i < HELD / 2; ++i) {
        const float send = up ? v[i] : v[i + HELD / 2], keep = up ? v[i + HELD / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, HELD);
    }
}

// Two warps make everything of one sixteen and head, a lane N / 32 channels: the first the weights, the second the operands.
constexpr int GP_SLOTS = 4;                                 // sixteens a block
template <int N>
struct GcRows {
    static constexpr int LD = N + 8;
    static constexpr int q = 0, k = GC_L * N * 2, a = 2 * k, part = a + GC_L * N * 4;           // rows of q, k and the decays; one part of an operand
    static constexpr int slot = part + GC_L * LD * 2, w = GP_SLOTS * slot, bytes = w + GP_SLOTS * GC_L * (GC_L + 1) * 4;
};

template <int N>
__global__ void __launch_bounds__(64 * GP_SLOTS, 2)
gla_prepare_kernel(const bf16* q_in, const bf16* k_in, long long ld, const float* decay, const int32_t* cu_q, unsigned char* blobs, int n_steps,
                   int n_seqs, int H) {
    constexpr int CH = N / 32;
    using Z = GcRows<N>;
    extern __shared__ __align__(16) unsigned char gw_sm[];
    pb_grid_dep_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, at = warp >> 1, slot = blockIdx.x * GP_SLOTS + at, h = blockIdx.y;
    const bool operands = warp & 1;
    pb_grid_dep_wait();
    int first = 0;
    const int cnt = slot < n_steps ? pb_find_chunk<GC_L>(cu_q, n_seqs, 1, slot, lane, first) : 0;      // the same for both warps
    unsigned char* rows = gw_sm + at * Z::slot;
    // all rows at once by way of shared memory: as loads into registers they are put off until a token wants its own, one trip to
    // memory each.  The two warps fetch half of them each.
    if (cnt > 0) {
        for (int idx = lane + 32 * operands; idx < GC_L * (N / 4); idx += 64) {
            const int t = idx / (N / 4), c = idx % (N / 4) * 4;
            const size_t row = (size_t)(first + min(t, cnt - 1));
            pb_cp_async16(rows + Z::a + (t * N + c) * 4, decay + row * ((size_t)H * N) + (size_t)h * N + c);
            if (c < N / 2) {
                pb_cp_async16(rows + Z::q + (t * N + 2 * c) * 2, q_in + row * ld + (size_t)h * N + 2 * c);
                pb_cp_async16(rows + Z::k + (t * N + 2 * c) * 2, k_in + row * ld + (size_t)h * N + 2 * c);
            }
        }
    }
    pb_cp_async_wait();
    __syncthreads();
    if (cnt <= 0) return;
    unsigned char* blob = blobs + ((size_t)slot * H + h) * GcBlob<N>::bytes;
    if (!operands) {
        float r[GC_L][CH];                                  // key s moved on to the token at hand
        float (*w)[GC_L + 1] = reinterpret_cast<float (*)[GC_L + 1]>(gw_sm + Z::w) + at * GC_L;
#pragma unroll
        for (int t = 0; t < GC_L; ++t) {
            float q[CH], d[CH], p[16];
            const unsigned* qr = reinterpret_cast<const unsigned*>(rows + Z::q + (t * N + lane * CH) * 2);
            const unsigned* kr = reinterpret_cast<const unsigned*>(rows + Z::k + (t * N + lane * CH) * 2);
            const float* ar = reinterpret_cast<const float*>(rows + Z::a) + t * N + lane * CH;
#pragma unroll
            for (int c = 0; c < CH; c += 2) {
                const unsigned qb = qr[c / 2], kb = kr[c / 2];
                const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qb)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&kb));
                q[c] = x.x; q[c + 1] = x.y;
                r[t][c] = y.x; r[t][c + 1] = y.y;
                d[c] = ar[c]; d[c + 1] = ar[c + 1];
            }
#pragma unroll
            for (int s = 0; s < 16; ++s) {
                p[s] = 0.f;
                if (s <= t) {
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        if (s < t) r[s][c] *= d[c];
                        p[s] = fmaf(q[c], r[s][c], p[s]);
                    }
                }
            }
            gc_halve<16>(p, lane);
            gc_halve<8>(p, lane);
            gc_halve<4>(p, lane);
            gc_halve<2>(p, lane);
            const float sum = p[0] + __shfl_xor_sync(0xffffffffu, p[0], 1);
            if ((lane & 1) == 0) {
                const int s = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
                w[t][s] = s <= t && t < cnt ? sum : 0.f;
            }
        }
        __syncwarp();
        const int r0 = lane >> 2, c0 = (lane & 3) * 2;
        unsigned m[4][3];
        pb_split3(w[r0][c0], w[r0][c0 + 1], m[0]);
        pb_split3(w[r0 + 8][c0], w[r0 + 8][c0 + 1], m[1]);
        pb_split3(w[r0][c0 + 8], w[r0][c0 + 9], m[2]);
        pb_split3(w[r0 + 8][c0 + 8], w[r0 + 8][c0 + 9], m[3]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(blob + GcBlob<N>::w + (p * 32 + lane) * 16) = make_uint4(m[0][p], m[1][p], m[2][p], m[3][p]);
        return;
    }
    // the queries times the decays up to them, then the keys times those behind them (a token past the end: nothing, decay 1); an
    // operand's three parts one after the other, each turned into register order by way of shared memory
    float x[GC_L][CH], d[CH];
    unsigned char* part = rows + Z::part;
    const unsigned base = pb_smem_addr(part);
    auto lay = [&](bool keys) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            __syncwarp();                                   // the part before has been read
#pragma unroll
            for (int t = 0; t < GC_L; ++t)
#pragma unroll
                for (int c = 0; c < CH; c += 2) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(x[t][c], x[t][c + 1]);
                    const float2 f = __bfloat1622float2(b);
                    x[t][c] -= f.x;
                    x[t][c + 1] -= f.y;
                    *reinterpret_cast<__nv_bfloat162*>(part + (t * Z::LD + lane * CH + c) * 2) = b;
                }
            __syncwarp();
#pragma unroll
            for (int n = 0; n < N / 16; ++n) {
                unsigned f[4];
                if (keys) pb_ldmatrix_x4_trans(f, base + (n * 16 + pb_bt_offset(lane, Z::LD)) * 2);
                else pb_ldmatrix_x4(f, base + (n * 16 + pb_a_offset(lane, Z::LD)) * 2);
                *reinterpret_cast<uint4*>(blob + (keys ? GcBlob<N>::k : GcBlob<N>::q) + ((n * 3 + p) * 32 + lane) * 16) = make_uint4(f[0], f[1], f[2], f[3]);
            }
        }
    };
#pragma unroll
    for (int c = 0; c < CH; ++c) d[c] = 1.f;
#pragma unroll
    for (int t = 0; t < GC_L; ++t) {
        const unsigned* qr = reinterpret_cast<const unsigned*>(rows + Z::q + (t * N + lane * CH) * 2);
        const float* ar = reinterpret_cast<const float*>(rows + Z::a) + t * N + lane * CH;
#pragma unroll
        for (int c = 0; c < CH; c += 2) {
            const unsigned raw = t < cnt ? qr[c / 2] : 0u;
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
            if (t < cnt) { d[c] *= ar[c]; d[c + 1] *= ar[c + 1]; }
            x[t][c] = f.x * d[c];
            x[t][c + 1] = f.y * d[c + 1];
        }
    }
    lay(false);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        reinterpret_cast<float*>(blob + GcBlob<N>::d)[lane * CH + c] = d[c];
        d[c] = 1.f;
    }
#pragma unroll
    for (int t = GC_L - 1; t >= 0; --t) {
        const unsigned* kr = reinterpret_cast<const unsigned*>(rows + Z::k + (t * N + lane * CH) * 2);
        const float* ar = reinterpret_cast<const float*>(rows + Z::a) + t * N + lane * CH;
#pragma unroll
        for (int c = 0; c < CH; c += 2) {
            const unsigned raw = t < cnt ? kr[c / 2] : 0u;
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
            x[t][c] = f.x * d[c];
            x[t][c + 1] = f.y * d[c + 1];
            if (t < cnt) { d[c] *= ar[c]; d[c + 1] *= ar[c + 1]; }
        }
    }
    lay(true);
}

template <int N, int PB>
struct GcLayout {
    static constexpr int LDP = PB + 8, LDO = PB + 8, NW = N / 16;
    static constexpr int blob = 0, v = GcBlob<N>::bytes, half = v + GC_L * LDP * 2;
    static constexpr int part = NW * GC_L * LDO * 4, o = GC_STAGES * half, bad = o + 2 * part, bytes = bad + 4 * PB * 4;
    static_assert(v % 16 == 0 && half % 16 == 0 && o % 16 == 0 && bytes <= 227 * 1024, "shared memory");
};

// The walk.  A block is one head's state [N, PB columns] and twelve warps.  Warps 0-7 multiply: warp (n, g) owns channels 16 n ..
// 16 n + 15 of column group g.  Warps 8-11: while the others work on one sixteen they add up the shares of the outputs of the one
// before and bring what the first kernel left of the next one, and its v, and what is three sixteens ahead on its way, into shared memory.  One barrier a
// sixteen.
template <int N, int PB>
__device__ __forceinline__ void gc_sequence(unsigned char* gc_sm, const bf16* v_in, long long ld, float scale, const unsigned char* blobs, float* state, float* y,
                                            const int32_t* cu_q, int seq, int slot, int h, int p_first, int H, int P) {
    using Z = GcLayout<N, PB>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int first = cu_q[seq], n_tok = cu_q[seq + 1] - first;
    const int n_steps = (n_tok + GC_L - 1) / GC_L;
    int* bads = reinterpret_cast<int*>(gc_sm + Z::bad);         // of four sixteens: the first token whose v is not finite, per column

    if (tid >= GC_MUL) {
        constexpr int FETCH = GC_ALL - GC_MUL;
        const int pt = tid - GC_MUL;
        const unsigned char* blob = blobs + ((size_t)pb_chunks_before<GC_L>(cu_q, seq, 1, lane) * H + h) * GcBlob<N>::bytes;
        constexpr int VP = PB / 8, V_IT = (GC_L * VP + FETCH - 1) / FETCH;
        uint4 vr[V_IT];
        auto ask = [&](int s) {                                 // v two sixteens ahead, in registers: nothing here may wait for it
            const int t0 = s * GC_L, cnt = min(GC_L, n_tok - t0);
#pragma unroll
            for (int it = 0; it < V_IT; ++it) {
                const int idx = min(pt + it * FETCH, GC_L * VP - 1), t = idx / VP, p = idx % VP * 8;
                vr[it] = *reinterpret_cast<const uint4*>(v_in + (size_t)(first + t0 + min(t, cnt - 1)) * ld + (size_t)h * P + p_first + p);
            }
        };
        auto bring = [&](int s) {
            if (s < n_steps) {
                unsigned char* to = gc_sm + s % GC_STAGES * Z::half;
                const unsigned char* from = blob + (size_t)s * H * GcBlob<N>::bytes;
                for (int o = pt * 16; o < GcBlob<N>::bytes; o += FETCH * 16) pb_cp_async16(to + o, from + o);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        auto put = [&](int s) {
            unsigned char* buf = gc_sm + s % GC_STAGES * Z::half;
            const int cnt = n_tok - s * GC_L;                   // a token past the end: nothing
            int* bad = bads + (s & 3) * PB;
#pragma unroll
            for (int it = 0; it < V_IT; ++it) {
                const int idx = pt + it * FETCH, t = idx / VP, p = idx % VP * 8;
                if (t >= GC_L) continue;
                if (t >= cnt) vr[it] = make_uint4(0, 0, 0, 0);
                unsigned raw[4] = {vr[it].x, vr[it].y, vr[it].z, vr[it].w};
                // a value that is not finite would reach earlier tokens through the zeros above the diagonal: it is taken out
                // here, and its column's results from its token on are set when they are stored
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if ((raw[e] & 0x7f80u) == 0x7f80u) { raw[e] &= 0xffff0000u; atomicMin(bad + p + 2 * e, t); }
                    if ((raw[e] & 0x7f800000u) == 0x7f800000u) { raw[e] &= 0x0000ffffu; atomicMin(bad + p + 2 * e + 1, t); }
                }
                *reinterpret_cast<uint4*>(buf + Z::v + (t * Z::LDP + p) * 2) = make_uint4(raw[0], raw[1], raw[2], raw[3]);
            }
        };
        auto add_up = [&](int s) {
            const float* part = reinterpret_cast<const float*>(gc_sm + Z::o + (s & 1) * Z::part);
            const int* bad = bads + (s & 3) * PB;
            const int t0 = s * GC_L, cnt = min(GC_L, n_tok - t0);
            for (int idx = pt; idx < GC_L * PB / 4; idx += FETCH) {
                const int t = idx / (PB / 4), p = idx % (PB / 4) * 4;
                if (t >= cnt) break;
                float4 sum = *reinterpret_cast<const float4*>(part + t * Z::LDO + p);
#pragma unroll
                for (int w = 1; w < Z::NW; ++w) {
                    const float4 f = *reinterpret_cast<const float4*>(part + (w * GC_L + t) * Z::LDO + p);
                    sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
                }
                const int4 from = *reinterpret_cast<const int4*>(bad + p);
                sum.x = t >= from.x ? __int_as_float(0x7fffffff) : sum.x * scale;
                sum.y = t >= from.y ? __int_as_float(0x7fffffff) : sum.y * scale;
                sum.z = t >= from.z ? __int_as_float(0x7fffffff) : sum.z * scale;
                sum.w = t >= from.w ? __int_as_float(0x7fffffff) : sum.w * scale;
                *reinterpret_cast<float4*>(y + (size_t)(first + t0 + t) * ((size_t)H * P) + (size_t)h * P + p_first + p) = sum;
            }
        };
        for (int idx = pt; idx < 4 * PB; idx += FETCH) bads[idx] = GC_L;
        pb_named_barrier(2, FETCH);
        for (int s = 0; s + 1 < GC_STAGES; ++s) bring(s);
        ask(0);
        put(0);
        if (n_steps > 1) ask(1);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(GC_STAGES - 2) : "memory");
        __syncthreads();
        for (int s = 0; s < n_steps; ++s) {
            bring(s + GC_STAGES - 1);                           // over the stage that was read a sixteen ago
            if (s > 0) add_up(s - 1);
            if (s + 1 < n_steps) put(s + 1);
            if (s + 2 < n_steps) ask(s + 2);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(GC_STAGES - 2) : "memory");
            for (int idx = pt; idx < PB; idx += FETCH) bads[((s + 2) & 3) * PB + idx] = GC_L;      // read last a sixteen ago
            __syncthreads();
        }
        add_up(n_steps - 1);
        return;
    }

    constexpr int NW = Z::NW, PG = 8 / NW, PW = PB / PG, PT = PW / 16;           // column groups, columns of one, its 16-row tiles of the transposed state
    static_assert(PT >= 1, "16 columns a warp at least");
    const int nw = warp % NW, pg = warp / NW;
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
    float* S = state + (((size_t)slot * H + h) * N + nw * 16 + c0) * P + p_first + pg * PW + r0;
    float st[PT][2][4];                                         // [16 columns p][8 channels]: rows p = r0, r0 + 8, channels c0, c0 + 1
#pragma unroll
    for (int a = 0; a < PT; ++a)
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
            for (int e = 0; e < 4; ++e) st[a][v][e] = S[(size_t)(8 * v + (e & 1)) * P + 16 * a + (e >> 1) * 8];
    __syncthreads();
    for (int s = 0; s < n_steps; ++s) {
        const unsigned char* buf = gc_sm + s % GC_STAGES * Z::half;
        const unsigned base = pb_smem_addr(buf);
        float big[PT][2][4], small[PT][2][4];
#pragma unroll
        for (int a = 0; a < PT; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int e = 0; e < 4; ++e) big[a][b][e] = small[a][b][e] = 0.f;
        // the warp's share of the outputs: its channels of the queries times its channels of the state
        unsigned qf[3][4];
        auto take = [&](unsigned (&f)[4], int at) {
            const uint4 x = *reinterpret_cast<const uint4*>(buf + Z::blob + at + lane * 16);
            f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
        };
#pragma unroll
        for (int p = 0; p < 3; ++p) take(qf[p], GcBlob<N>::q + (nw * 3 + p) * 512);
#pragma unroll
        for (int a = 0; a < PT; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                unsigned b0[3], b1[3];
                pb_split3(st[a][0][2 * b], st[a][0][2 * b + 1], b0);
                pb_split3(st[a][1][2 * b], st[a][1][2 * b + 1], b1);
                const unsigned sb[3][2] = {{b0[0], b1[0]}, {b0[1], b1[1]}, {b0[2], b1[2]}};
                pb_mma6(big[a][b], small[a][b], qf, sb);
            }
        // the weights times v: 8 columns each from some of the warps
        constexpr int TILES = PW / 8;
#pragma unroll
        for (int a = 0; a < PT; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int tile = 2 * a + b;
                if (nw == tile * NW / TILES % NW) {
                    unsigned b0, b1;
                    pb_ldmatrix_x2_trans(b0, b1, base + Z::v + (pg * PW + tile * 8 + (lane & 15) * Z::LDP) * 2);
#pragma unroll
                    for (int p = 2; p >= 0; --p) {
                        unsigned wf[4];
                        take(wf, GcBlob<N>::w + p * 512);
                        pb_mma(p ? small[a][b] : big[a][b], wf, b0, b1);
                    }
                }
            }
        float* dst = reinterpret_cast<float*>(gc_sm + Z::o + (s & 1) * Z::part) + (nw * GC_L + r0) * Z::LDO + pg * PW + c0;
#pragma unroll
        for (int a = 0; a < PT; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                *reinterpret_cast<float2*>(dst + 16 * a + 8 * b) = make_float2(small[a][b][0] + big[a][b][0], small[a][b][1] + big[a][b][1]);
                *reinterpret_cast<float2*>(dst + 8 * Z::LDO + 16 * a + 8 * b) = make_float2(small[a][b][2] + big[a][b][2], small[a][b][3] + big[a][b][3]);
            }
        // the state behind the sixteen
        unsigned kf[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) take(kf[p], GcBlob<N>::k + (nw * 3 + p) * 512);
        const int* bad = bads + (s & 3) * PB + pg * PW;
        const float2 d0 = *reinterpret_cast<const float2*>(buf + GcBlob<N>::d + (nw * 16 + c0) * 4),
                     d1 = *reinterpret_cast<const float2*>(buf + GcBlob<N>::d + (nw * 16 + 8 + c0) * 4);
#pragma unroll
        for (int a = 0; a < PT; ++a) {
            unsigned vf[4];
            pb_ldmatrix_x4_trans(vf, base + Z::v + (pg * PW + 16 * a + pb_at_offset(lane, Z::LDP)) * 2);
            float more[2][4], less[2][4];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
#pragma unroll
                for (int e = 0; e < 4; ++e) more[v][e] = less[v][e] = 0.f;
                pb_mma(less[v], vf, kf[2][2 * v], kf[2][2 * v + 1]);
                pb_mma(less[v], vf, kf[1][2 * v], kf[1][2 * v + 1]);
                pb_mma(more[v], vf, kf[0][2 * v], kf[0][2 * v + 1]);
            }
            const bool ba = bad[16 * a + r0] < GC_L, bb = bad[16 * a + r0 + 8] < GC_L;
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float d = v == 0 ? (e & 1 ? d0.y : d0.x) : (e & 1 ? d1.y : d1.x);
                    st[a][v][e] = (e < 2 ? ba : bb) ? __int_as_float(0x7fffffff) : fmaf(d, st[a][v][e], less[v][e] + more[v][e]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < PT; ++a)
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[(size_t)(8 * v + (e & 1)) * P + 16 * a + (e >> 1) * 8] = st[a][v][e];
}

template <int N, int PB, bool RECORDED>
__global__ void __launch_bounds__(GC_ALL, 1)
gla_walk_kernel(const bf16* v_in, long long ld, float scale, const unsigned char* blobs, float* state, float* y, const int32_t* cu_q, const int32_t* slots,
                PbSequences which, int H, int P) {
    extern __shared__ __align__(16) unsigned char gc_sm[];
    pb_grid_dep_launch();
    const int slices = P / PB;
    const int h = blockIdx.x / slices, p_first = (blockIdx.x % slices) * PB;
    pb_grid_dep_wait();
    pb_for_sequences<RECORDED>(cu_q, which, [&](int seq, int) {
        gc_sequence<N, PB>(gc_sm, v_in, ld, scale, blobs, state, y, cu_q, seq, slots[seq], h, p_first, H, P);
    });
}

struct GcCall {
    const bf16 *q, *k, *v;
    long long ld;
    const float* decay;
    float scale;
    float *state, *y;
    const int32_t *cu_q, *slots;
    unsigned char* scratch;
    int n_steps, n_seqs, most, counted, longest, H, P;
    long long order;
    cudaStream_t stream;
};

template <int N, int PB, bool RECORDED>
int gc_walk(const GcCall& c, int rows, const PbSequences& which) {
    constexpr int bytes = GcLayout<N, PB>::bytes;
    static const cudaError_t set = cudaFuncSetAttribute(gla_walk_kernel<N, PB, RECORDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    PB_REQUIRE(set == cudaSuccess, "gla_scan_chunked: %s", cudaGetErrorString(set));
    pb_launch(gla_walk_kernel<N, PB, RECORDED>, dim3(c.H * (c.P / PB), rows), dim3(GC_ALL), bytes, c.stream, c.v, c.ld, c.scale, (const unsigned char*)c.scratch, c.state, c.y,
              c.cu_q, c.slots, which, c.H, c.P);
    PB_CHECK_LAUNCH("gla_scan_chunked");
    return 0;
}

template <int N>
int gc_run(const GcCall& c) {
    static const cudaError_t set = cudaFuncSetAttribute(gla_prepare_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, GcRows<N>::bytes);
    PB_REQUIRE(set == cudaSuccess, "gla_scan_chunked: %s", cudaGetErrorString(set));
    pb_launch(gla_prepare_kernel<N>, dim3((c.n_steps + GP_SLOTS - 1) / GP_SLOTS, c.H), dim3(64 * GP_SLOTS), GcRows<N>::bytes, c.stream, c.q, c.k, c.ld, c.decay, c.cu_q,
              c.scratch, c.n_steps, c.n_seqs, c.H);
    PB_CHECK_LAUNCH("gla_scan_chunked");
    // 64 channels: always two column groups of 16
    const PbSequences all{c.n_seqs, 1, INT_MAX, 0, 0, 0, 0, 0, 0, c.longest > 0, (unsigned long long)c.order};
    return pb_for_widths(c.H, c.P, N == 64 ? 32 : 16, 32, all, c.most, c.counted, [&](int width, int rows, const PbSequences& which) {
        if constexpr (N == 64) return which.recorded ? gc_walk<64, 32, true>(c, rows, which) : gc_walk<64, 32, false>(c, rows, which);
        else if (which.recorded) return width == 32 ? gc_walk<128, 32, true>(c, rows, which) : gc_walk<128, 16, true>(c, rows, which);
        else return width == 32 ? gc_walk<128, 32, false>(c, rows, which) : gc_walk<128, 16, false>(c, rows, which);
    });
}

}  // namespace

// Whether pb_gla_scan_chunked takes these sizes and operands: rows and results in 16-byte pieces, 64 or 128 channels, values in 16-column slices
// (64 channels: 32, a column group for each half of the warps).
PB_API int pb_gla_chunked_takes(const void* q, const void* k, const void* v, const void* decay, const float* y, long long ld, int H, int N, int P) {
    return (N == 64 || N == 128) && P > 0 && P % (N == 64 ? 32 : 16) == 0 && H > 0 && H < 65536 && ld % 8 == 0 && pb_aligned(q, 16) && pb_aligned(k, 16) &&
                   pb_aligned(v, 16) && pb_aligned(decay, 16) && pb_aligned(y, 16)
               ? 1
               : 0;
}
// Most sixteens that n_tokens of n_seqs sequences can form, and the scratch memory (16-byte aligned) that the call needs for them.
PB_API int pb_gla_chunks(int n_tokens, int n_seqs) { return n_tokens / GC_L + (n_seqs < n_tokens ? n_seqs : n_tokens); }
PB_API long long pb_gla_chunk_bytes(int n_steps, int H, int N) { return (long long)n_steps * H * (N == 64 ? GcBlob<64>::bytes : GcBlob<128>::bytes); }

// Operands as for pb_gla_scan, bfloat16; n_steps and scratch as the two functions above say.  most: how many sequences there are
// (`counted`), or can be, for a step that is being recorded.  order, longest: PbSequences, and the longest sequence's tokens (0: no order).
PB_API int pb_gla_scan_chunked(const void* q, const void* k, const void* v, long long ld, const float* decay, float scale, float* state, float* y,
                               const int32_t* cu_q, const int32_t* slots, void* scratch, int n_steps, int n_seqs, int most, int counted, long long order, int longest, int H,
                               int N, int P, cudaStream_t stream) {
    PB_REQUIRE(n_seqs >= 0 && n_steps >= 0 && pb_gla_chunked_takes(q, k, v, decay, y, ld, H, N, P), "gla_scan_chunked: %d heads of %d x %d", H, N, P);
    PB_REQUIRE(q && k && v && decay && state && y && cu_q && slots && scratch, "gla_scan_chunked: null pointer");
    PB_REQUIRE(pb_aligned(scratch, 16), "gla_scan_chunked: misaligned operands");
    PB_REQUIRE(most >= 0 && most <= n_seqs && most < 65536, "gla_scan_chunked: %d of %d sequences in one launch", most, n_seqs);
    if (most == 0 || n_steps == 0) return 0;
    const GcCall c{(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, decay, scale, state, y, cu_q, slots, (unsigned char*)scratch, n_steps, n_seqs, most,
                   counted, longest, H, P, order, stream};
    return N == 128 ? gc_run<128>(c) : gc_run<64>(c);
}
