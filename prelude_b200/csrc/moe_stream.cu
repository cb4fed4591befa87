// The routed experts' products of a decode step, where an expert has a row or a few: a stream over the matrices of the experts that were
// chosen, each read once.
//
//   pb_moe_stream   out[slot, n] = sum_k A[slot / a_div, k] * W[e(slot), n, k], or an activation of the sums (MoeAct in moe.cu), for the
//                   slots' choices ids [n_slots]; bfloat16 in, float32 sums, bfloat16 or float32 out
//
// As gemm_stream.cu: one block a multiprocessor, four loader warps bring rows of W through a ring of stages (8 rows by a piece of K, one
// bulk copy a row), eight warps multiply on the tensor cores with the weights as the row operand, their sums meet in shared memory.
// What differs:
//  * The rows to stream are those of the chosen experts: every block counts the choices for itself, lists the experts that were hit in
//    ascending order, one with more than eight rows of A once for every eight, and takes its equal share of all their rows, in units of 8
//    features; a share may span experts.  (With the eights of an expert walked by the blocks that have its share, those take twice as long and all wait:
//    a feed-forward of 64 experts of 4,096 x 2,048, top 6, 12 tokens, nine of them at one expert, 522 us; here 309, the kernel in moe.cu 377.)
//  * The column operand are up to eight rows of A, those that chose the expert at hand.  Where all rows of A fit they lie in shared
//    memory from the start, else those of the next expert are asked for while one is worked on (two buffers where two fit).
//  * Which rows come first is known only when the router is done, so nothing is fetched ahead of the wait for the kernel before - but by
//    the second of two such products in a row, which finds the choices settled: the first one lets the kernel behind it begin only when
//    it has itself waited, so that a block fills its ring while other multiprocessors are still at the first product.  The experts of 8 rows,
//    2,048 x 2,048, both products 79.0 -> 76.6 us.
// Every sum is over k in an order that K alone decides (steps of 16 dealt to eight warps with four chains each, piece by piece), so a token's
// result does not depend on who else chose the expert.  No sum runs on in the tensor cores, which cut what they add up: a step's sixteen products
// are added to a chain in float32, and the eight warps' sums meet in 64 bits.  Error against 64 bits, with running sums / with chains in float32 and the
// warps in 32 bits / here / the kernel in moe.cu: K = 768 7.4e-8, 6.7e-8, 5.4e-8, 6.6e-8; 2,048 9.4e-8, 7.5e-8, 6.3e-8, 7.9e-8; 4,096, gated 2.6e-7, 1.3e-7,
// 1.2e-7, 1.5e-7; 7,168, gated 4.2e-7, 1.5e-7, 1.4e-7, 1.8e-7.  It costs nothing with rows of 2,048 and more, of 768 up to 4 %.
//
// What bounds it: the weights' bytes.  A product alone, us against the kernel in moe.cu, whose warps keep four rows of 2 KB in flight and spend half
// their lives on beginnings and ends: 21 experts hit by 32 choices, 4,096 x 4,096 gated 106 against 115 (6.7 TB/s); 26 hit, 4,096 x 2,048 68 against 77,
// 2,048 x 2,048 37 against 42, eight hit 14 against 19.  Short rows leave it bound by the copies and by each tile's sums (1,000 and 1,300 cycles a tile
// of 16 rows): 2,048 rows of 768, one token 7.4 against 11.6, eight 26 against 24, sixteen 36 against 37; rows of 512 take a fifth more and keep the
// kernel in moe.cu.
#include "attention_common.cuh"

#define MS_WARPS 8                              // multiplying warps
#define MS_LOADERS 4
#define MS_THREADS ((MS_WARPS + MS_LOADERS) * 32)
#define MS_ROWS 8                               // features of a stage; rows of A at a time
#define MS_MAX_STAGES 16
#define MS_CHAINS 4
#define MS_SLOTS 512
#define MS_EXPERTS 1024
#define MS_SMEM_LIMIT (227 * 1024 - 1024)

struct MsParams {
    const __nv_bfloat16* A;
    const __nv_bfloat16* W;
    const int32_t* ids;
    void* out;
    long long lda, w_expert_stride, ldo;
    int n_slots, n_src, a_div, n_experts, N, K;
    int ks, n_chunks, stages, bufs;
    int gated, act, out_f32, settled;       // settled: see pb_moe_stream
    float limit, alpha;
    int* status;
};

// Bytes of shared memory ahead of the rows of A: two sets of the warps' sums, the choices, the counts, the experts hit, four slot lists
struct MsLayout {
    static constexpr int red = 0, ids = red + 2 * MS_WARPS * 16 * 8 * 4, count = ids + MS_SLOTS * 4, hits = count + MS_EXPERTS * 4,
                         slots = hits + MS_SLOTS * 4, x = slots + 4 * MS_ROWS * 4;
};

// One block's share: which entries of the list (an expert, the eight of its rows), which of their features; the loaders and the others walk it alike.
struct MsWalk {
    int hit, f0, f1;
};
#define MS_EIGHT 16                             // an entry: the expert, and from this bit on which eight of its rows

__global__ void __launch_bounds__(MS_THREADS, 1) moe_stream_kernel(MsParams p) {
    extern __shared__ __align__(128) unsigned char ms_sm[];
    __shared__ __align__(8) uint64_t full_bar[MS_MAX_STAGES], empty_bar[MS_MAX_STAGES], x_bar[2];
    __shared__ int s_dead, s_hits;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x_stride = p.K * 2 + 16, w_stride = p.ks * 2 + 16, stage_bytes = MS_ROWS * w_stride;   // 16 bytes more: rows in different bank groups
    float* red = reinterpret_cast<float*>(ms_sm + MsLayout::red);
    int* ids = reinterpret_cast<int*>(ms_sm + MsLayout::ids);
    int* count = reinterpret_cast<int*>(ms_sm + MsLayout::count);
    int* hits = reinterpret_cast<int*>(ms_sm + MsLayout::hits);
    int* slots = reinterpret_cast<int*>(ms_sm + MsLayout::slots);
    unsigned char* sx = ms_sm + MsLayout::x;
    unsigned char* ring = sx + (size_t)p.bufs * MS_ROWS * x_stride;

    for (int e = tid; e < p.n_experts; e += MS_THREADS) count[e] = 0;
    if (tid < 32) {                                            // a thread a stage, as in gemm_stream.cu
        if (lane == 0) {
            s_dead = 0;
            mbar_init(&x_bar[0], 1);
            mbar_init(&x_bar[1], 1);
        }
        if (lane < p.stages) { mbar_init(&full_bar[lane], 1); mbar_init(&empty_bar[lane], MS_WARPS); }
        mbar_fence_init();
    }
    __syncthreads();
    if (!p.settled) pb_grid_dep_wait();
    // Only now: a kernel whose blocks begin behind this finds done whatever was launched ahead of this one
    if (!p.settled) pb_grid_dep_launch();
    for (int i = tid; i < p.n_slots; i += MS_THREADS) {
        const int e = __ldcg(p.ids + i);                       // from L2: written a moment ago
        ids[i] = e;
        if (e >= 0 && e < p.n_experts) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int e0 = 0; e0 < p.n_experts; e0 += 32) {
            const int eights = e0 + lane < p.n_experts ? (count[e0 + lane] + MS_ROWS - 1) / MS_ROWS : 0;
            if (!__any_sync(0xffffffffu, eights > 1)) {
                const unsigned who = __ballot_sync(0xffffffffu, eights > 0);
                if (eights) hits[n + __popc(who & ((1u << lane) - 1u))] = e0 + lane;
                n += __popc(who);
            } else {
                int upto = eights;                             // of this lane's expert and those before it
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += v;
                }
                for (int i = 0; i < eights; ++i) hits[n + upto - eights + i] = (e0 + lane) | (i << MS_EIGHT);
                n += __shfl_sync(0xffffffffu, upto, 31);
            }
        }
        if (lane == 0) s_hits = n;
    }
    __syncthreads();
    const int units = (p.N + MS_ROWS - 1) / MS_ROWS;           // of one entry
    const long long all = (long long)s_hits * units;
    const long long u0 = blockIdx.x * all / gridDim.x, u1 = (blockIdx.x + 1) * all / gridDim.x;
    if (u0 >= u1) {
        if (p.settled) pb_grid_dep_wait();                     // no block ends before the kernel ahead has
        return;
    }
    const int span = p.gated ? MS_ROWS : 16;                   // features of a tile
    auto open = [&](int hit) {
        MsWalk w;
        const long long base = (long long)hit * units;
        w.hit = hit;
        w.f0 = (int)(max(u0 - base, 0ll)) * MS_ROWS;
        w.f1 = min((int)min(u1 - base, (long long)units) * MS_ROWS, p.N);
        return w;
    };
    const int first_hit = (int)(u0 / units), last_hit = (int)((u1 - 1) / units);
    // to the next entry; false: there is none
    auto next = [&](MsWalk& w) {
        if (w.hit == last_hit) return false;
        w = open(w.hit + 1);
        return true;
    };
    auto expert_of = [&](const MsWalk& w) { return hits[w.hit] & ((1 << MS_EIGHT) - 1); };
    auto first_row = [&](const MsWalk& w) { return (hits[w.hit] >> MS_EIGHT) * MS_ROWS; };

    if (warp >= MS_WARPS) {
        // ---------------- loaders: the warps take the stages in turn, a lane copies a row ----------------
        // No more warps than stages: a warp that waits for a stage's tenant of one lap ago then knows that the one of two laps ago has left (it
        // has waited for that or a later one), and a parity tells only two laps apart
        const int lw = warp - MS_WARPS, n_loaders = min(MS_LOADERS, p.stages);
        bool ok = true;
        int stage = 0, phase = 0, i = 0, turn = 0;
        MsWalk w = open(first_hit);
        do {
            const __nv_bfloat16* We = p.W + (size_t)expert_of(w) * p.w_expert_stride;
#pragma unroll 1
            for (int f = w.f0; f < w.f1 && ok; f += span) {
                const int halves = (p.gated || w.f1 - f > MS_ROWS) ? 2 : 1;
#pragma unroll 1
                for (int kc = 0; kc < p.n_chunks && ok; ++kc) {
                    for (int h = 0; h < halves; ++h, ++i) {
                        if (turn == lw) {
                            if (i >= p.stages) {               // the first ring-full finds every stage free
                                ok = mbar_wait_bounded(&empty_bar[stage], phase ^ 1);
                                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                            }
                            const int feat0 = f + (p.gated ? 0 : h * MS_ROWS);
                            const int row0 = feat0 + (p.gated ? h * p.N : 0);    // up rows follow the gate rows
                            const int k0 = kc * p.ks, len = min(p.ks, p.K - k0), rows = min(MS_ROWS, w.f1 - feat0);
                            if (lane == 0) mbar_arrive_expect_tx(&full_bar[stage], (unsigned)rows * len * 2);
                            if (lane < rows)
                                bulk_copy_g2s(ring + (size_t)stage * stage_bytes + (size_t)lane * w_stride, We + (size_t)(row0 + lane) * p.K + k0,
                                              (unsigned)len * 2, &full_bar[stage]);
                        }
                        if (++turn == n_loaders) turn = 0;
                        if (++stage == p.stages) { stage = 0; phase ^= 1; }
                    }
                }
            }
        } while (ok && next(w));
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 13);
        return;
    }

    // ---------------- multiplying warps ----------------
    if (p.settled) {                                           // the weights are on their way; the rows are the kernel's just ahead, and its readers' the results
        pb_grid_dep_wait();
        pb_grid_dep_launch();
    }
    const bool resident = p.n_src <= p.bufs * MS_ROWS;
    // the slots of a segment, and its rows of A on their way (warp 0): segment n uses slot list n % 4 and, where the rows do not all stay, buffer
    // n % bufs, which nobody reads any more
    auto stage_rows = [&](const MsWalk& w, int n) {
        const int e = expert_of(w), first = first_row(w);
        int found = 0;
        for (int s0 = 0; s0 < p.n_slots; s0 += 32) {
            const bool mine = s0 + lane < p.n_slots && ids[s0 + lane] == e;
            const unsigned who = __ballot_sync(0xffffffffu, mine);
            const int at = found + __popc(who & ((1u << lane) - 1u)) - first;
            if (mine && at >= 0 && at < MS_ROWS) slots[(n & 3) * MS_ROWS + at] = s0 + lane;
            found += __popc(who);
        }
        __syncwarp();
        const int rows = min(MS_ROWS, found - first), buf = resident ? 0 : n % p.bufs;
        if (resident && n > 0) return;
        const int bring = resident ? p.n_src : rows;
        if (lane == 0) mbar_arrive_expect_tx(&x_bar[buf], (unsigned)bring * p.K * 2);
        __syncwarp();
        if (lane < bring) {
            const int src = resident ? lane : slots[(n & 3) * MS_ROWS + lane] / p.a_div;
            bulk_copy_g2s(sx + (size_t)(buf * MS_ROWS + lane) * x_stride, p.A + (size_t)src * p.lda, (unsigned)p.K * 2, &x_bar[buf]);
        }
    };
    const int g = lane >> 2, t4 = lane & 3;
    const unsigned sx_a = smem_u32(sx), ring_a = smem_u32(ring);
    const unsigned a_off = (lane & 7) * w_stride + (lane >> 4) * 16;
    const bool upper = (lane & 8) != 0;                        // this lane addresses a row of the second stage
    int stage = 0, phase = 0, n = 0, tile = 0;
    MsWalk w = open(first_hit), ahead = w;
    bool more = true;                                          // of `ahead`, the next segment whose rows are to be asked for
    if (warp == 0) {
        stage_rows(ahead, 0);
        more = next(ahead);
    }
    do {
        if (warp == 0 && more && (n > 0 || p.bufs > 1 || resident)) {
            // two buffers, or all rows there: the segment after this one; one buffer: this one, whose buffer the last one has left
            const int at = (p.bufs > 1 || resident) ? n + 1 : n;
            stage_rows(ahead, at);
            more = next(ahead);
        }
        const int buf = resident ? 0 : n % p.bufs;
        if (!resident || n == 0) {
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&x_bar[buf], resident ? 0 : (n / p.bufs) & 1))) {
                if (lane == 0) { *(volatile int*)&s_dead = 1; if (p.status) atomicExch(p.status, 13); }
            }
        }
        const int rows = min(MS_ROWS, count[expert_of(w)] - first_row(w));
        const int* mine_slots = slots + (n & 3) * MS_ROWS;
        // warp 0 wrote the list before it arrived at the barrier just waited for, or before those of the tiles of the segment before
        const int m_row = min(lane & 7, rows - 1);
        const unsigned b_off = (unsigned)(resident ? mine_slots[m_row] / p.a_div : buf * MS_ROWS + m_row) * x_stride + ((lane >> 3) & 1) * 16;
#pragma unroll 1
        for (int f = w.f0; f < w.f1; f += span, ++tile) {
            const int halves = (p.gated || w.f1 - f > MS_ROWS) ? 2 : 1;
            float acc[MS_CHAINS][4];
#pragma unroll
            for (int c = 0; c < MS_CHAINS; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
#pragma unroll 1
            for (int kc = 0; kc < p.n_chunks; ++kc) {
                const int stage2 = (stage + 1 == p.stages) ? 0 : stage + 1, phase2 = (stage + 1 == p.stages) ? phase ^ 1 : phase;
                bool landed = mbar_wait_bounded(&full_bar[stage], phase);
                if (halves == 2) landed = landed && mbar_wait_bounded(&full_bar[stage2], phase2);
                if (!__all_sync(0xffffffffu, landed)) {
                    if (lane == 0) { *(volatile int*)&s_dead = 1; if (p.status) atomicExch(p.status, 13); }
                    break;
                }
                const int k0 = kc * p.ks, steps = min(p.ks, p.K - k0) >> 4;
                const unsigned a_base = ring_a + ((upper && halves == 2) ? stage2 : stage) * stage_bytes + a_off;
                const unsigned b_base = sx_a + b_off + k0 * 2;
#pragma unroll 1
                for (int s0 = warp; s0 < steps; s0 += MS_WARPS * MS_CHAINS) {
                    unsigned a[MS_CHAINS][4], b[MS_CHAINS][2];
#pragma unroll
                    for (int c = 0; c < MS_CHAINS; ++c) {
                        const int s = s0 + c * MS_WARPS;
                        if (s < steps) {
                            ldsm_x4<0>(a[c], a_base + s * 32);
                            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(b[c][0]), "=r"(b[c][1]) : "r"(b_base + s * 32));
                        }
                    }
#pragma unroll
                    for (int c = 0; c < MS_CHAINS; ++c)
                        if (s0 + c * MS_WARPS < steps) {
                            // sixteen products at a time: what the tensor cores add to a running sum they cut off instead of rounding it
                            float q[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_bf16_free(q, a[c], b[c][0], b[c][1]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[c][e] += q[e];
                        }
                }
                __syncwarp();
                if (lane == 0) {
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&empty_bar[stage])) : "memory");
                    if (halves == 2) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&empty_bar[stage2])) : "memory");
                }
                for (int h = 0; h < halves; ++h)
                    if (++stage == p.stages) { stage = 0; phase ^= 1; }
            }
            // the eight warps' sums: acc[.][e] is feature g (+ 8 for e >= 2), row 2 t4 + (e & 1); two sets, so that one barrier a tile is enough
            float* set = red + (tile & 1) * MS_WARPS * 128;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                set[warp * 128 + (2 * t4 + (e & 1)) * 16 + g + 8 * (e >> 1)] = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
            asm volatile("bar.sync 1, %0;\n" ::"n"(MS_WARPS * 32) : "memory");
            if (*(volatile int*)&s_dead) return;
            const int per = p.gated ? MS_ROWS : 16;
            for (int idx = tid; idx < rows * per; idx += MS_WARPS * 32) {
                const int m = idx / per, rr = idx % per, feat = f + rr;
                if (feat >= w.f1) continue;
                auto sum = [&](int at) {                       // of the warps, in 64 bits: rounded once (in 32 bits these sums alone are half of the error)
                    double w8[MS_WARPS];
#pragma unroll
                    for (int k = 0; k < MS_WARPS; ++k) w8[k] = set[k * 128 + m * 16 + at];
                    return (float)(((w8[0] + w8[1]) + (w8[2] + w8[3])) + ((w8[4] + w8[5]) + (w8[6] + w8[7])));
                };
                float v = sum(rr);
                const float u = p.gated ? sum(rr + 8) : 0.f;
                if (p.gated) v = p.act == PB_ACT_CLAMPED ? pb_clamped_unit(v, u, p.limit, p.alpha) : v / (1.0f + expf(-v)) * u;
                else if (p.act == PB_ACT_RELU2) v = pb_relu2(v);
                const size_t at = (size_t)mine_slots[m] * p.ldo + feat;
                if (p.out_f32) reinterpret_cast<float*>(p.out)[at] = v;
                else reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v);
            }
        }
        ++n;
    } while (next(w));
}

// Piece of K a stage, stages and buffers for rows of K: two buffers of eight rows of A where they take no more than a third of shared memory; the
// longest equal pieces, in steps of 128, of which four stages fit, else three.  (25 experts hit of 2,048 x 4,096, us, by
// pieces of 1,024, 2,048, 4,096: 71, 65, 73 for K = 4,096; uneven ones, 2,560 and 1,536, 83.)
static bool ms_plan(int K, int* ks, int* n_chunks, int* stages, int* bufs, size_t* smem) {
    const size_t x_rows = (size_t)MS_ROWS * ((size_t)K * 2 + 16);
    *bufs = 2 * x_rows <= MS_SMEM_LIMIT / 3 ? 2 : 1;
    const size_t taken = MsLayout::x + *bufs * x_rows;
    if (taken >= MS_SMEM_LIMIT) return false;
    for (int want = 4; want >= 3; --want)
        for (int n = 1; n == 1 || K / n >= 512; ++n) {
            const int piece = n == 1 ? K : ((K + n - 1) / n + 127) / 128 * 128;
            const size_t stage = (size_t)MS_ROWS * ((size_t)piece * 2 + 16), fit = (MS_SMEM_LIMIT - taken) / stage;
            if ((int)fit < want) continue;
            *ks = piece; *n_chunks = (K + piece - 1) / piece; *stages = fit > MS_MAX_STAGES ? MS_MAX_STAGES : (int)fit;
            *smem = taken + *stages * stage;
            return true;
        }
    return false;
}

// Whether pb_moe_stream takes rows of K elements, n_slots choices among n_experts (rows shorter than 768 are left to pb_moe_gemv: see above).
PB_API int pb_moe_stream_supported(int K, int n_slots, int n_experts) {
    int ks, nc, st, bufs;
    size_t smem;
    return K >= 768 && K % 16 == 0 && n_slots > 0 && n_slots <= MS_SLOTS && n_experts > 0 && n_experts <= MS_EXPERTS && ms_plan(K, &ks, &nc, &st, &bufs, &smem) ? 1 : 0;
}

// A [n_slots / a_div, K] with row stride lda; W [n_experts, (2) N, K], w_expert_stride elements from one expert to the next, gate rows
// first; ids int32 [n_slots]; out [n_slots, N] with row stride ldo, float32 or bfloat16.  act, limit, alpha: as in pb_moe_gemv.  settled: ids and W were
// there when the kernel launched before this one passed its own wait, and that one is a pb_moe_stream; they are read ahead of the wait.
PB_API int pb_moe_stream(const void* A, long long lda, int a_div, const void* W, long long w_expert_stride, int N, int K, int gated, int act, float limit,
                         float alpha, const int32_t* ids, int n_slots, int n_experts, int settled, void* out, long long ldo, int out_dtype, int* status, cudaStream_t stream) {
    PB_REQUIRE(pb_moe_stream_supported(K, n_slots, n_experts) && N > 0 && a_div > 0 && n_slots % a_div == 0, "moe_stream: K=%d, %d choices of %d experts", K, n_slots, n_experts);
    PB_REQUIRE(A && W && ids && out && pb_aligned(A, 16) && pb_aligned(W, 16) && lda % 8 == 0 && w_expert_stride % 8 == 0, "moe_stream: null or unaligned pointer");
    PB_REQUIRE(lda >= K && ldo >= N && w_expert_stride >= (long long)(gated ? 2 : 1) * N * K, "moe_stream: a stride is shorter than its row");
    PB_REQUIRE(gated ? act == PB_ACT_SILU || (act == PB_ACT_CLAMPED && limit > 0.f) : act == PB_ACT_NONE || act == PB_ACT_RELU2,
               "moe_stream: activation %d in the %s form, limit %g", act, gated ? "gated" : "plain", (double)limit);
    PB_REQUIRE(out_dtype == PB_F32 || out_dtype == PB_BF16, "moe_stream: unknown output type code %d", out_dtype);
    MsParams p{};
    p.A = (const __nv_bfloat16*)A; p.W = (const __nv_bfloat16*)W; p.ids = ids; p.out = out; p.lda = lda; p.w_expert_stride = w_expert_stride; p.ldo = ldo;
    p.n_slots = n_slots; p.n_src = n_slots / a_div; p.a_div = a_div; p.n_experts = n_experts; p.N = N; p.K = K; p.gated = gated ? 1 : 0; p.act = act;
    p.out_f32 = out_dtype == PB_F32; p.settled = settled ? 1 : 0; p.limit = limit; p.alpha = alpha; p.status = status;
    size_t smem;
    ms_plan(K, &p.ks, &p.n_chunks, &p.stages, &p.bufs, &smem);
    static const cudaError_t set = cudaFuncSetAttribute(moe_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM_LIMIT);
    PB_REQUIRE(set == cudaSuccess, "moe_stream: %s", cudaGetErrorString(set));
    static const int sms = pb_multiprocessors();
    pb_launch(moe_stream_kernel, dim3(sms), dim3(MS_THREADS), smem, stream, p);
    PB_CHECK_LAUNCH("moe_stream");
    return 0;
}
