// Attention of single tokens (a decode step) whose keys and values are one cached row - a latent of `vd` elements with a rotated key part
// behind it, shared by all heads - on the fifth-generation tensor cores.
//
//   q [n_tokens, H, kd] bfloat16      pages [num_pages, G, page_size, kd] bfloat16, the values a row's first vd elements
//   out[t, h] = sum_j softmax_j(scale q[t, h] . k_j) k_j[0 .. vd)      float32 scores, weights and sums
//
// What bounds it are the cached rows, read once: 16 requests behind 3,000 tokens of 576 elements are 55 MB.  A block has one token's
// heads, at most 32 of them, and walks 64 rows at a time.
//   Scores: S = Q K^T with the queries in tensor memory, where each of the four groups of 32 lanes holds all heads' queries: a thread has
// one head and a quarter of the tile's rows, and the products' idle 96 lanes serve to spread the softmax over four warps.
//   Result: O^T = K^T P^T, value elements by heads: the rows are the first operand, read element by element out of the bytes that served as
// keys, so 32 heads cost a quarter of what they would as rows of a 128-row product, and the result takes 128 columns of tensor memory
// and not 512.  A weight goes in as two bfloat16 numbers, its rounding and what that left: the result is then as far from 64 bits as its
// own rounding (1.66e-3 in the 2-norm; weights rounded once 1.67e-3 to 2.04e-3, the more where no row dominates).
// A tile's scores take the tensor cores 1,230 cycles and its result 1,600, less than a tile takes to come from memory with all
// multiprocessors at it (74 KB at 1/148 of 6.5 TB/s: 1.7 us, 3,100 cycles).
//
// The key range of a token is cut among the blocks of a cluster, which put their parts together through distributed shared memory, in
// order, each for its share of the heads: no scratch memory and no second kernel.
//
// Measured against the form on mma.sync with its merge (attention_paged_tc.cu, 32-row tiles with four barriers each), 32 heads, rows of 576
// from memory, us: 16 requests behind 3,000 tokens each 42.4 -> 22.5, 64 of them 130 -> 50 (4.4 TB/s), one 22.2 -> 15.8; behind 512 tokens 16
// requests 17.5 -> 12.3, 2 requests 11.4 -> 9.3; behind 64 tokens 16 requests 10.7 and 10.8, 256 requests 18.5 and 25.  What is left besides the bytes:
// 5,000 cycles until the first scores, and 9,000 from the last tile to the end (two cluster barriers around the parts' way to the block
// that adds them up).  Copies into the L2 cache four tiles ahead were no faster alone and 0.9 us slower between a layer's other kernels.
//
// Warps 0..3: the softmax, the result's rescaling when a maximum has grown by more than 2^8 (up to there the weights may exceed 1: their
// relative rounding is the same), the way out.  Warp 4: the copies.  Warps 5 and 6: the two products.  Rows that do not count (behind the token,
// outside the window, of a page that is not there) are zeroed in shared memory before a product reads them: what another request left in a
// page's rest must not get into the sums, not even times zero.  Every wait is bounded in time.
#include "tcgen05_pair.cuh"

#include <math.h>

namespace {

typedef __nv_bfloat16 bf16;

constexpr int LA_KEYS = 64, LA_HEADS = 32, LA_THREADS = 224, LA_MAX_KD = 576, LA_MAX_SPLITS = 8;
// A tile in shared memory: eight rows at a time (one copy), of them 64 elements at a time, 128-byte rows in the 128-byte swizzle.  Groups
// of eight rows are thus at one distance whichever pages they come from, which is what both products' descriptors ask for.  (Copies of 16
// rows by 64 elements, 36 a tile: the copies alone took 6,400 cycles a tile.)
constexpr int LA_ATOM = 8 * 128, LA_P_BYTES = LA_HEADS * 128;
constexpr float LA_GROWTH = 8.0f;
constexpr int LA_TMEM = 512, LA_O_COL = 0, LA_S_COL = 128, LA_Q_COL = 192, LA_MAX_STAGES = 6;
constexpr float LA_LOG2E = 1.4426950408889634f;

struct LaParts {
    float m[LA_HEADS], l[4][LA_HEADS];                      // this block's: maxima, sums of the four warps
    float part_m[LA_MAX_SPLITS][LA_HEADS], part_l[LA_MAX_SPLITS][LA_HEADS], weight[LA_HEADS][LA_MAX_SPLITS];     // of its heads
};
static_assert(sizeof(LaParts) <= 2 * LA_P_BYTES, "over the weights");

struct LaMaps {
    CUtensorMap q, k;
};

struct LaParams {
    bf16* out;
    const float* sink;
    const int32_t* positions;
    const int32_t* table_row;
    const int32_t* block_table;
    const bf16* gate;
    long long ld_gate;
    int* status;
    int table_stride, page_size, num_pages, H, G, kd, vd, hp, head_tiles, window, splits, stages;
    float scale;
};

__device__ __forceinline__ void la_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void la_bar() { asm volatile("bar.sync 1, 128;\n" ::: "memory"); }
__device__ __forceinline__ void la_st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(addr), "f"(v) : "memory"); }
// Shared-memory descriptors of a tile's rows as the first operand, K-major (rows by elements) and MN-major (elements by rows): groups of
// eight rows `group_bytes` apart, the next 64 elements of the same rows LA_ATOM.
__device__ __forceinline__ uint64_t la_desc_rows(const void* tile, unsigned group_bytes) {
    return (tc_smem_desc(tile) & ~((uint64_t)0x3FFF << 32)) | (uint64_t)(group_bytes >> 4) << 32;
}
__device__ __forceinline__ uint64_t la_desc_elements(const void* tile, unsigned group_bytes) {
    return (tc_smem_desc_mn(tile, LA_ATOM) & ~((uint64_t)0x3FFF << 32)) | (uint64_t)(group_bytes >> 4) << 32;
}
__global__ void __launch_bounds__(LA_THREADS, 1) attention_latent_kernel(const __grid_constant__ LaMaps maps, LaParams p) {
    pb_grid_dep_launch();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_bar[LA_MAX_STAGES], free_bar[LA_MAX_STAGES], q_full, q_ready, s_full, s_free, p_ready, pv_done, fixed_bar;
    __shared__ uint32_t tmem_holder;
    __shared__ int s_ok, s_mask[LA_MAX_STAGES];
    __shared__ float s_max[2][4][LA_HEADS], s_corr[4][LA_HEADS];

    cg::cluster_group cluster = cg::this_cluster();
    const int part = p.splits > 1 ? (int)cluster.block_rank() : 0;
    const int item = blockIdx.x / p.splits;
    const int tok = item / (p.G * p.head_tiles), g = item / p.head_tiles % p.G, ht = item % p.head_tiles;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = p.H / p.G, head0 = g * group + ht * p.hp, heads = min(p.hp, group - ht * p.hp);
    const int ncb = p.kd / 64, group_bytes = ncb * LA_ATOM, stage_bytes = LA_KEYS / 8 * group_bytes;
    // the weights, two parts: [heads][64 rows], 128-byte rows in the 128-byte swizzle; behind the last tile what the parts tell each other
    unsigned char* sp = smem + p.stages * stage_bytes;
    LaParts& parts = *reinterpret_cast<LaParts*>(sp);
    unsigned char* sq = smem + (p.stages - 1) * stage_bytes;        // the queries on their way into tensor memory: where the last stage is, later
    float* so = reinterpret_cast<float*>(smem);             // [parts][this block's heads][vd], over the tiles when the cluster's products are done

    if (threadIdx.x == 0) {
        s_ok = 1;
        for (int i = 0; i < p.stages; ++i) { tc_mbar_init(&full_bar[i], 1); tc_mbar_init(&free_bar[i], 1); }
        tc_mbar_init(&s_full, 1); tc_mbar_init(&s_free, 4); tc_mbar_init(&q_full, 1); tc_mbar_init(&q_ready, 4); tc_mbar_init(&p_ready, 4); tc_mbar_init(&pv_done, 1);
        tc_mbar_init(&fixed_bar, 4);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 5) tc_tmem_alloc(&tmem_holder, LA_TMEM);
    if (warp == 4 && lane == 0) { tc_prefetch_map(&maps.q); tc_prefetch_map(&maps.k); }
    pb_grid_dep_wait();
    const int trow = p.table_row[tok], pos_tok = p.positions[tok];
    // this block's heads of the result: `per` of them from part * per on; thread n has the n-th one's gate and sink
    const int per = (p.hp + p.splits - 1) / p.splits, mine = max(0, min(per, heads - part * per)), my_head = head0 + part * per + (int)threadIdx.x;
    float gate = 0.f, sink = -INFINITY;
    if ((int)threadIdx.x < mine) {
        if (p.gate) gate = __bfloat162float(p.gate[(size_t)tok * p.ld_gate + my_head]);
        if (p.sink) sink = p.sink[my_head] * LA_LOG2E;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_holder;
    const bool live = trow >= 0;                            // else a padding row of a captured step
    const int pos = live ? pos_tok : -1;
    const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    const int first = lo / LA_KEYS, walk = live ? pos / LA_KEYS - first + 1 : 0;
    const int each = (walk + p.splits - 1) / p.splits, begin = min(walk, part * each), nt = min(walk, begin + each) - begin;
    const int page_shift = 31 - __clz(p.page_size), ppt = LA_KEYS >> page_shift, all_pages = (1 << ppt) - 1;
    auto key0 = [&](int i) { return (first + begin + i) * LA_KEYS; };
    auto edge = [&](int i, int mask) { return mask != all_pages || key0(i) + LA_KEYS - 1 > pos || key0(i) < lo; };

    if (warp == 4) {
        // ---------------- copies: eight rows each ----------------
        bool ok = true;
        const int32_t* table = p.block_table + (size_t)max(trow, 0) * p.table_stride;
        int stage = 0;
        unsigned phase = 1;                                 // the first round finds the stages free
        if (nt > 0 && lane == 0) {
            tc_mbar_expect_tx(&q_full, ncb * p.hp * 128);
            tc_tma_load_3d(sq, &maps.q, 0, tok * p.H + head0, 0, &q_full);
        }
        __syncwarp();
        for (int i = 0; i < nt; ++i) {
            ok = __all_sync(0xffffffffu, i == p.stages - 1 ? tc_mbar_wait(&q_ready, 0) : i < p.stages || tc_mbar_wait(&free_bar[stage], phase));
            if (!ok) break;
            int page = -1;
            const int j0 = key0(i) + lane * p.page_size;
            if (lane < ppt && j0 <= pos && j0 + p.page_size > lo) {
                page = table[j0 >> page_shift];
                if (page >= p.num_pages) { page = -1; if (p.status) atomicExch(p.status, 6); }
            }
            const int mask = (int)__ballot_sync(0xffffffffu, page >= 0);
            if (lane == 0) {
                s_mask[stage] = mask;
                tc_mbar_expect_tx(&full_bar[stage], __popc(mask) * p.page_size * p.kd * 2);
            }
            __syncwarp();
            const int id = __shfl_sync(0xffffffffu, page, min(lane * 8 >> page_shift, ppt - 1));
            if (lane < LA_KEYS / 8 && id >= 0)
                tc_tma_load_3d(smem + stage * stage_bytes + lane * group_bytes, &maps.k, 0, (id * p.G + g) * p.page_size + (lane * 8 & (p.page_size - 1)), 0, &full_bar[stage]);
            if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 14);
    } else if (warp == 5) {
        // ---------------- scores ----------------
        // (the whole warp walks, one thread issues: descriptors stay in uniform registers)
        bool ok = true;
        if (nt > 0) {
            const uint32_t idesc = tc_instr_desc(LA_KEYS);
            const uint64_t dk0 = la_desc_rows(smem, group_bytes);
            auto wait = [&](uint64_t* bar, unsigned phase) { ok = ok && __all_sync(0xffffffffu, tc_mbar_wait(bar, phase)); };
            int n_fixed = 0, stage = 0;
            unsigned phase = 0;
            wait(&q_ready, 0);
            for (int i = 0; i < nt && ok; ++i) {
                wait(&full_bar[stage], phase);
                if (edge(i, s_mask[stage])) wait(&fixed_bar, n_fixed++ & 1);
                if (i > 0) wait(&s_free, (i - 1) & 1);
                if (!ok) break;
                tc_fence_after();
                if (tc_elect_one()) {
                    uint64_t dk = dk0 + (unsigned)(stage * stage_bytes >> 4);
                    uint32_t q = tmem + LA_Q_COL;
                    for (int cb = 0; cb < ncb; ++cb) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc_mma_ts(tmem + LA_S_COL, q + 8 * k, dk + 2 * k, idesc, (cb > 0 || k > 0) ? 1u : 0u);
                        dk += LA_ATOM >> 4;
                        q += 32;
                    }
                    tc_commit(&s_full);
                }
                __syncwarp();
                if (++stage == p.stages) { stage = 0; phase ^= 1; }
            }
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 15);
    } else if (warp == 6) {
        // ---------------- result: a warp of its own, so that no tile's result stands behind the next tile's scores ----------------
        const uint32_t idesc = tc_instr_desc(p.hp) | (1u << 15);            // (the rows as elements: MN-major)
        const uint64_t dp = tc_smem_desc(sp), dv0 = la_desc_elements(smem, group_bytes);
        const int o_tiles = p.vd / 128;
        bool ok = true;
        int stage = 0;
        for (int i = 0; i < nt && ok; ++i) {
            ok = __all_sync(0xffffffffu, tc_mbar_wait(&p_ready, i & 1));
            if (!ok) break;
            tc_fence_after();
            if (tc_elect_one()) {
                const uint64_t dv = dv0 + (unsigned)(stage * stage_bytes >> 4);
                for (int m = 0; m < o_tiles; ++m)
#pragma unroll
                    for (int k = 0; k < LA_KEYS / 16; ++k)
#pragma unroll
                        for (int v = 1; v >= 0; --v)        // the small parts first
                            tc_mma(tmem + LA_O_COL + m * LA_HEADS, dv + (unsigned)((2 * m * LA_ATOM + 2 * k * group_bytes) >> 4), dp + (v * LA_P_BYTES >> 4) + 2 * k, idesc,
                                   (i > 0 || k > 0 || v == 0) ? 1u : 0u);
                tc_commit(&free_bar[stage]);
                tc_commit(&pv_done);
            }
            __syncwarp();
            if (++stage == p.stages) stage = 0;
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 17);
    } else {
        // ---------------- softmax and result: a thread has head `lane` and rows 16 warp .. 16 warp + 15 of a tile ----------------
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
        const int o_tiles = p.vd / 128;
        const float scale2 = p.scale * LA_LOG2E;            // scores in units of log 2
        float l = 0.f, m = -INFINITY;                       // the maximum that the head's weights are taken against: the same in all four warps
        bool ok = true;
        if (nt > 0) {
            // all heads' queries into this warp's lanes, two elements a column
            ok = tc_mbar_wait(&q_full, 0);
            const int r = lane & (p.hp - 1);
            for (int cb = 0; cb < ncb; ++cb) {
                uint32_t raw[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(sq + cb * p.hp * 128 + r * 128 + ((c ^ (r & 7)) << 4));
                    raw[4 * c] = v.x; raw[4 * c + 1] = v.y; raw[4 * c + 2] = v.z; raw[4 * c + 3] = v.w;
                }
                tc_tmem_st32(taddr + LA_Q_COL + cb * 32, raw);
            }
            la_proxy_fence();                               // the next to write there is a copy
            tc_tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(&q_ready);
        }
        int stage = 0;
        unsigned phase = 0;
        for (int i = 0; i < nt; ++i) {
            const int base = key0(i);
            ok = ok && tc_mbar_wait(&full_bar[stage], phase);
            const int mask = s_mask[stage];
            auto counts = [&](int r) { return base + r <= pos && base + r >= lo && (mask >> (r >> page_shift) & 1); };
            const bool partial = edge(i, mask);
            if (ok && partial) {
                for (int r = warp; r < LA_KEYS; r += 4)
                    if (!counts(r))
                        for (int c = lane; c < ncb * 8; c += 32)
                            *reinterpret_cast<uint4*>(smem + stage * stage_bytes + (r >> 3) * group_bytes + (c >> 3) * LA_ATOM + (r & 7) * 128 + (c & 7) * 16) =
                                make_uint4(0, 0, 0, 0);
                la_proxy_fence();
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&fixed_bar);
            }
            if (++stage == p.stages) { stage = 0; phase ^= 1; }
            ok = ok && tc_mbar_wait(&s_full, i & 1);
            tc_fence_after();
            float s[16];
            tc_tmem_ld16(taddr + LA_S_COL + warp * 16, s);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(&s_free);
            float top = -INFINITY;
#pragma unroll
            for (int c = 0; c < 16; ++c) s[c] *= scale2;
            if (partial) {
#pragma unroll
                for (int c = 0; c < 16; ++c) s[c] = counts(warp * 16 + c) ? s[c] : -INFINITY;
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) top = fmaxf(top, s[c]);
            s_max[i & 1][warp][lane] = top;
            la_bar();
            top = fmaxf(fmaxf(s_max[i & 1][0][lane], s_max[i & 1][1][lane]), fmaxf(s_max[i & 1][2][lane], s_max[i & 1][3][lane]));
            const bool grown = top > m + LA_GROWTH || (m == -INFINITY && top > -INFINITY);
            if (__any_sync(0xffffffffu, grown)) {           // the same in all four warps
                const float m_new = fmaxf(m, top), corr = m == -INFINITY ? 0.f : exp2f(m - m_new);
                s_corr[warp][lane] = corr;
                l *= corr;
                m = m_new;
                __syncwarp();
                if (i > 0) {
                    ok = ok && tc_mbar_wait(&pv_done, (i - 1) & 1);
                    tc_fence_after();
                    for (int o = 0; o < o_tiles; ++o) {
                        uint32_t raw[32];
                        tc_tmem_ld32(taddr + LA_O_COL + o * LA_HEADS, raw);
                        tc_tmem_ld_wait();
#pragma unroll
                        for (int h = 0; h < LA_HEADS; ++h) raw[h] = __float_as_uint(__uint_as_float(raw[h]) * s_corr[warp][h]);
                        tc_tmem_st32(taddr + LA_O_COL + o * LA_HEADS, raw);
                    }
                    tc_tmem_st_wait();
                }
                __syncwarp();
            }
            const float ref = m == -INFINITY ? 0.f : m;
            unsigned w[2][8];                               // the weights in two parts: rounded, and what that left
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
                const float e0 = exp2f(s[c] - ref), e1 = exp2f(s[c + 1] - ref);
                l += e0 + e1;
                const __nv_bfloat162 b = __floats2bfloat162_rn(e0, e1);
                const float2 taken = __bfloat1622float2(b);
                const __nv_bfloat162 r = __floats2bfloat162_rn(e0 - taken.x, e1 - taken.y);
                w[0][c / 2] = *reinterpret_cast<const unsigned*>(&b);
                w[1][c / 2] = *reinterpret_cast<const unsigned*>(&r);
            }
            if (i > 0) ok = ok && tc_mbar_wait(&pv_done, (i - 1) & 1);           // the weights' place is free
            if (lane < p.hp) {
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    unsigned char* row = sp + v * LA_P_BYTES + lane * 128;
                    *reinterpret_cast<uint4*>(row + (((2 * warp) ^ (lane & 7)) << 4)) = make_uint4(w[v][0], w[v][1], w[v][2], w[v][3]);
                    *reinterpret_cast<uint4*>(row + (((2 * warp + 1) ^ (lane & 7)) << 4)) = make_uint4(w[v][4], w[v][5], w[v][6], w[v][7]);
                }
            }
            la_proxy_fence();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(&p_ready);
        }
        if (nt > 0) ok = ok && tc_mbar_wait(&pv_done, (nt - 1) & 1);
        tc_fence_after();
        parts.l[warp][lane] = l;
        if (warp == 0) parts.m[lane] = m;
        if (!ok) {
            s_ok = 0;
            if (lane == 0 && p.status) atomicExch(p.status, 16);
        }
    }
    if (p.splits > 1) cluster.sync();                       // nobody's tiles are needed any more
    else __syncthreads();
    // Every head's maximum, sum and result go to the block that puts the head together, over the cluster's tiles.
    if (warp < 4 && live && s_ok) {
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + LA_O_COL, to = tc_smem(so) + (warp * 32 + lane) * 4;
        if (warp == 0 && lane < heads) {
            const int owner = lane / per, n = lane - owner * per;
            la_st_cluster(gp_map_to_rank(tc_smem(&parts.part_m[part][n]), owner), parts.m[lane]);
            la_st_cluster(gp_map_to_rank(tc_smem(&parts.part_l[part][n]), owner), (parts.l[0][lane] + parts.l[1][lane]) + (parts.l[2][lane] + parts.l[3][lane]));
        }
#pragma unroll 1
        for (int o = 0; o < p.vd / 128; ++o) {
            uint32_t raw[32];
            tc_tmem_ld32(taddr + o * LA_HEADS, raw);
            tc_tmem_ld_wait();
            const uint32_t first_row = to + (part * per * p.vd + o * 128) * 4;
            uint32_t at = gp_map_to_rank(first_row, 0);
            int owner = 0, n = 0;
#pragma unroll
            for (int h = 0; h < LA_HEADS; ++h) {
                if (h < heads) la_st_cluster(at, nt > 0 ? __uint_as_float(raw[h]) : 0.f);
                at += p.vd * 4;
                if (++n == per) { n = 0; ++owner; at = gp_map_to_rank(first_row, min(owner, p.splits - 1)); }
            }
        }
    }
    if (p.splits > 1) cluster.sync();
    else __syncthreads();
    if (live && s_ok) {
        if ((int)threadIdx.x < mine) {
            float w[LA_MAX_SPLITS], l[LA_MAX_SPLITS], M = sink, L = 0.f;
#pragma unroll
            for (int s = 0; s < LA_MAX_SPLITS; ++s) {
                w[s] = s < p.splits ? parts.part_m[s][threadIdx.x] : -INFINITY;
                l[s] = s < p.splits ? parts.part_l[s][threadIdx.x] : 0.f;
            }
#pragma unroll
            for (int s = 0; s < LA_MAX_SPLITS; ++s) M = fmaxf(M, w[s]);
            const float top = M == -INFINITY ? 0.f : M;
#pragma unroll
            for (int s = 0; s < LA_MAX_SPLITS; ++s) {
                w[s] = exp2f(w[s] - top);
                L += l[s] * w[s];
            }
            if (p.sink) L += exp2f(sink - top);
            const float inv = (L > 0.f || L != L ? 1.0f / L : 0.f) * (p.gate ? 1.0f / (1.0f + expf(-gate)) : 1.0f);
#pragma unroll
            for (int s = 0; s < LA_MAX_SPLITS; ++s) parts.weight[threadIdx.x][s] = w[s] * inv;
        }
        __syncthreads();
        const int d = threadIdx.x * 4;
        if (d < p.vd) {
            bf16* dst = p.out + ((size_t)tok * p.H + head0 + part * per) * p.vd + d;
            const float* src = so + d;
#pragma unroll 2
            for (int n = 0; n < mine; ++n) {
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                for (int s = 0; s < p.splits; ++s) {
                    const float4 v = *reinterpret_cast<const float4*>(src + (s * per + n) * p.vd);
                    const float w = parts.weight[n][s];
                    acc.x = fmaf(v.x, w, acc.x); acc.y = fmaf(v.y, w, acc.y); acc.z = fmaf(v.z, w, acc.z); acc.w = fmaf(v.w, w, acc.w);
                }
                const __nv_bfloat162 a = __floats2bfloat162_rn(acc.x, acc.y), b = __floats2bfloat162_rn(acc.z, acc.w);
                uint2 raw;
                raw.x = *reinterpret_cast<const uint32_t*>(&a);
                raw.y = *reinterpret_cast<const uint32_t*>(&b);
                *reinterpret_cast<uint2*>(dst + n * p.vd) = raw;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        __syncwarp();
        tc_fence_after();
        tc_tmem_dealloc(tmem, LA_TMEM);
    }
}

int la_stages(int kd) {
    const int n = 220 * 1024 / (LA_KEYS * kd * 2);
    return n < LA_MAX_STAGES ? n : LA_MAX_STAGES;
}
// (never so little that two blocks share a multiprocessor: each has all of its tensor memory, and blocks of two clusters could wait for each
// other's)
size_t la_smem(int kd) {
    const size_t n = 1024 + (size_t)la_stages(kd) * LA_KEYS * kd * 2 + 2 * LA_P_BYTES;
    return n > 120 * 1024 ? n : 120 * 1024;
}

// Blocks that run at once in clusters of `splits`, one a multiprocessor.
int la_slots(int splits) {
    static const struct Slots {
        int n[LA_MAX_SPLITS + 1] = {};
        Slots() {
            int dev = 0, sms = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaFuncSetAttribute(attention_latent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)la_smem(LA_MAX_KD));
            n[1] = sms;
            for (int s = 2; s <= LA_MAX_SPLITS; ++s) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3((unsigned)(sms / s * s));
                cfg.blockDim = dim3(LA_THREADS);
                cfg.dynamicSmemBytes = la_smem(LA_MAX_KD);
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = s; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
                cfg.attrs = attr; cfg.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, attention_latent_kernel, &cfg) != cudaSuccess) { clusters = 0; (void)cudaGetLastError(); }
                n[s] = clusters * s;
            }
        }
    } slots;
    return slots.n[splits];
}

int la_heads(int H, int G) { return H / G <= 16 ? 16 : LA_HEADS; }

// [rows, cols] as {64 elements, rows, cols / 64}: a copy brings 64 elements of `box_rows` rows, `box_blocks` times
int la_map(CUtensorMap* map, const void* ptr, long long rows, int cols, int box_rows, int box_blocks) {
    cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(cols / 64)};
    cuuint64_t strides[2] = {(cuuint64_t)cols * 2, 128};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)box_blocks}, estr[3] = {1, 1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : pb_fail("attention_latent: cuTensorMapEncodeTiled failed with code %d (%lld rows of %d)", (int)r, rows, cols);
}

}  // namespace

// Rows of whole 64-element blocks, values of whole 128-row tiles of the result, pages that divide a tile.
PB_API int pb_attention_latent_supported(int H, int G, int kd, int vd, int page_size) {
    return H > 0 && G > 0 && H % G == 0 && kd > 0 && kd % 64 == 0 && kd <= LA_MAX_KD && vd > 0 && vd % 128 == 0 && vd <= 512 && vd <= kd &&
           (page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64);
}

// q [n_tokens, H, kd], out [n_tokens, H, vd], pages [num_pages, G, page_size, kd]; token t's rows are those at block_table[table_row[t]]
// of positions max(0, positions[t] - window + 1) (window 0: 0) .. positions[t]; table_row[t] < 0: no such token.  sink: float32 [H] or null;
// gate [n_tokens, H] with row stride ld_gate, or null: sigmoid(gate) multiplies a head's output.  max_context: no position is larger.
// force_splits (tests): into how many parts a token's rows are cut, 0 for the kernel's choice.
PB_API int pb_attention_latent_bf16(const void* q, const void* pages, void* out, const float* sink, const int32_t* positions, const int32_t* table_row,
                                    const int32_t* block_table, int table_stride, int page_size, int num_pages, int n_tokens, int H, int G, int kd, int vd,
                                    float scale, int window, const void* gate, long long ld_gate, int max_context, int force_splits, int* status,
                                    cudaStream_t stream) {
    PB_REQUIRE(pb_attention_latent_supported(H, G, kd, vd, page_size), "attention_latent: H=%d G=%d kd=%d vd=%d pages of %d not taken", H, G, kd, vd, page_size);
    PB_REQUIRE(q && pages && out && positions && table_row && block_table && table_stride > 0 && num_pages > 0 && n_tokens >= 0 && window >= 0 &&
                   (!gate || ld_gate >= H) && force_splits >= 0 && force_splits <= LA_MAX_SPLITS,
               "attention_latent: null pointer or bad geometry");
    PB_REQUIRE(pb_aligned(q, 16) && pb_aligned(pages, 16) && pb_aligned(out, 8), "attention_latent: operands must be 16-byte aligned");
    if (n_tokens == 0) return 0;
    if (int e = get_encode()) return e;
    LaParams p{};
    p.out = (bf16*)out; p.sink = sink; p.stages = la_stages(kd); p.positions = positions; p.table_row = table_row; p.block_table = block_table; p.gate = (const bf16*)gate;
    p.ld_gate = ld_gate; p.status = status; p.table_stride = table_stride; p.page_size = page_size; p.num_pages = num_pages; p.H = H; p.G = G; p.kd = kd;
    p.vd = vd; p.hp = la_heads(H, G); p.head_tiles = (H / G + p.hp - 1) / p.hp; p.window = window; p.scale = scale;
    const long long items = (long long)n_tokens * G * p.head_tiles;
    const int rows = window > 0 && window < max_context ? window : max_context, tiles = max(1, (rows + LA_KEYS - 1) / LA_KEYS);
    // as many parts as still run all at once
    p.splits = 1;
    for (int s = 2; s <= LA_MAX_SPLITS && s <= tiles; ++s)
        if (items * s <= la_slots(s)) p.splits = s;
    if (force_splits) p.splits = force_splits;
    PB_REQUIRE(la_slots(p.splits) >= p.splits && items * p.splits < (1ll << 31), "attention_latent: %d parts, %lld blocks", p.splits, items * p.splits);
    LaMaps maps;
    if (int e = la_map(&maps.q, q, (long long)n_tokens * H, kd, p.hp, kd / 64)) return e;
    if (int e = la_map(&maps.k, pages, (long long)num_pages * G * page_size, kd, 8, kd / 64)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items * p.splits));
    cfg.blockDim = dim3(LA_THREADS);
    cfg.dynamicSmemBytes = la_smem(kd);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pb_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = p.splits; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, attention_latent_kernel, maps, p);
    PB_CHECK_LAUNCH("attention_latent");
    return 0;
}
