// Products of routed experts in prompt steps, on paired blocks of the fifth-generation tensor cores (tcgen05.mma.cta_group::2):
//
//   A: [places, K] bfloat16, the rows sorted by expert     B: [n_experts * R, K] bfloat16, the experts' matrices one below the other
//   out[i, j] = sum_k A[i, k] * B[e(i) R + j, k]           gated: silu (or the clamped unit) of the gate sums times the up sums
//
// For experts with fewer rows than fill the tiles of gemm_pair.cu's grouped form: the weights are the product's 256 rows, the tokens its
// columns, 64 to 256 of them, and the down projection's result is float32.  What bounds it are the weights, each of which is read once:
// 64 experts of 4,096 x 2,048 with 16 rows each, both products and the rows' copy, 529 us for 3.2 GB (6.1 TB/s) against 1,452 on the 64-row
// tiles of moe.cu; with 32 rows 542 against 1,509, with 128 610 against 1,826 on its 128-row tiles.  (From 192 rows on the form with the tokens
// as rows takes them, the products alone 637 against 659 with the float32 result here.)
//
// A pair's tile is 256 rows of an expert's matrix (gated: 128 gate rows and the 128 up rows of the same features, 64 of each in each
// block) by at most 256 of its tokens.  Each block holds its 128 weight rows and half of the tokens; its tensor memory receives its rows'
// sums for all tokens.  Tiles run along an expert's features first: the pairs of a wave share a few experts' tokens, which stay in the
// L2 cache.
//
// In each block: warp 8 issues the tensor-map copies (three stages), warp 9 of the leading block the products for both, warps 0..7
// read the sums out of tensor memory (two accumulators: one's stores overlap the next one's products).  A thread has one row, that is
// one feature: 32 lanes write 64 bytes of a token's row.  In the gated form gate and up sums of a feature lie in
// lanes 64 apart; the warps swap halves of every 32 columns through shared memory.  Every wait is bounded in time; a
// block that gives up raises the status word, and both leave through the cluster's last barrier with their tensor memory freed.
#include "tcgen05_pair.cuh"

namespace {

constexpr int GG_STEP = 64;                                 // tokens come in steps of this many, half of them in each block
// A stage holds two copies of 64 of K: what it costs the warp that issues the products - wait, vote, election, commit - is 500 to 600 cycles,
// longer than four products of fewer than 256 columns take.  (Stages of one copy, six of them, both products, us: 64 experts of 4,096 x 2,048
// with 4 rows each 571, now 504; with 64 rows 584, now 536; with 160 rows 773, now 645.  gemm_pair.cu's products have 256 columns, and gained nothing.)
constexpr int GG_STAGES = 3, GG_SUB = 2, GG_STAGE_BYTES = GG_SUB * GP_STAGE_BYTES;
constexpr int GG_SWAP = 2 * 2 * 16 * 64 * 4;                // two sets of epilogue warps, two halves of 32 columns, 64 features

// Copy boxes: a block's 128 weight rows, or 64 gate rows and 64 up rows; its tokens, 128, 64 or 32 of them.  (In copies of 16 rows, with
// columns in steps of 32, 64 experts with 96 rows took 456 + 221 us instead of 408 + 203.)
struct GgMaps {
    CUtensorMap w, x[3];
};

struct GgParams {
    void* out;                                              // [places, out_cols] bfloat16, or float32 (plain form)
    int* status;
    long long ldo;
    int out_cols, expert_rows, tiles_m, tiles_n, kblocks, gated, act, wide;          // wide: float32 out
    float limit, alpha;
    // row tile tm: rows tile_row0[tm] .. of expert tile_expert[tm] (negative: no such tile), at most 256, which end before offsets[expert + 1]
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* offsets;
};

// Where row tile tm lies, and how many columns its product has; false when there is no such tile.
__device__ __forceinline__ bool gg_tile(const GgParams& p, int tm, int& expert, int& row0, int& rows, int& columns) {
    expert = p.tile_expert[tm];
    if (expert < 0) return false;
    row0 = p.tile_row0[tm];
    rows = min(256, p.offsets[expert + 1] - row0);
    columns = max(GG_STEP, (rows + GG_STEP - 1) / GG_STEP * GG_STEP);
    return true;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_grouped_kernel(const __grid_constant__ GgMaps maps, GgParams p) {
    pb_grid_dep_launch();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full_bar[GG_STAGES], empty_bar[GG_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_holder;
    __shared__ int s_ok;

    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();             // 0: the leading block of the pair
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_tiles = p.tiles_m * p.tiles_n;

    if (threadIdx.x == 0) {
        s_ok = 1;
        for (int s = 0; s < GG_STAGES; ++s) { tc_mbar_init(&full_bar[s], 1); tc_mbar_init(&empty_bar[s], 1); }
        for (int a = 0; a < 2; ++a) { tc_mbar_init(&acc_full[a], 1); tc_mbar_init(&acc_empty[a], 2 * GP_EPI_WARPS); }   // the epilogue warps of both blocks
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 9) gp_tmem_alloc2(&tmem_holder, 512);       // one warp of each block, the same warp in both
    if (warp == 8 && lane == 0) { tc_prefetch_map(&maps.w); for (int i = 0; i < 3; ++i) tc_prefetch_map(&maps.x[i]); }
    tc_fence_before();
    cluster.sync();                                         // both blocks' barriers and tensor memory are set up
    tc_fence_after();
    const uint32_t tmem_base = tmem_holder;
    pb_grid_dep_wait();                                     // the tile map and the rows are earlier kernels'

    if (warp == 8) {
        if (lane == 0) {
            bool ok = true;
            int fill = 0;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                const int tm = tile / p.tiles_n, tn = tile % p.tiles_n;
                int expert, row0, rows, columns;
                if (!gg_tile(p, tm, expert, row0, rows, columns)) continue;
                const int half = columns / 2, x_row = row0 + rank * half;
                const int w_row = expert * p.expert_rows + (p.gated ? tn * 128 + rank * 64 : tn * 256 + rank * 128);
                for (int kb = 0; kb < p.kblocks; ++kb, ++fill) {
                    const int stage = fill % GG_STAGES;
                    ok = tc_mbar_wait(&empty_bar[stage], ((fill / GG_STAGES) & 1) ^ 1);
                    if (!ok) break;
                    const uint32_t leader_full = gp_map_to_rank(tc_smem(&full_bar[stage]), 0);
                    if (rank == 0) tc_mbar_expect_tx(&full_bar[stage], GG_SUB * (2 * GP_A_BYTES + columns * GP_BK * 2));   // both blocks' copies land on this barrier
#pragma unroll
                    for (int sub = 0; sub < GG_SUB; ++sub) {
                        unsigned char* sw = smem + stage * GG_STAGE_BYTES + sub * GP_STAGE_BYTES;
                        const int k = (kb * GG_SUB + sub) * GP_BK;
                        gp_tma_load_2d(sw, &maps.w, k, w_row, leader_full);
                        if (p.gated) gp_tma_load_2d(sw + 64 * GP_BK * 2, &maps.w, k, w_row + p.out_cols, leader_full);
                        int r = 0;
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            if (half & (128 >> i)) {
                                gp_tma_load_2d(sw + GP_A_BYTES + r * GP_BK * 2, &maps.x[i], k, x_row + r, leader_full);
                                r += 128 >> i;
                            }
                    }
                }
            }
            if (!ok && p.status) atomicExch(p.status, 8);
        }
    } else if (warp == 9) {
        // ---------------- products: the leading block issues for the pair ----------------
        if (rank == 0) {
            int fill = 0, seg = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                int expert, row0, rows, columns;
                if (!gg_tile(p, tile / p.tiles_n, expert, row0, rows, columns)) continue;       // seg counts the tiles that exist
                const uint32_t idesc = gp_idesc(columns);
                const int acc = seg & 1;
                ok = __all_sync(0xffffffffu, tc_mbar_wait(&acc_empty[acc], ((seg >> 1) & 1) ^ 1));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * 256;
                for (int kb = 0; kb < p.kblocks; ++kb, ++fill) {
                    const int stage = fill % GG_STAGES;
                    ok = __all_sync(0xffffffffu, tc_mbar_wait(&full_bar[stage], (fill / GG_STAGES) & 1));
                    if (!ok) break;
                    tc_fence_after();
                    if (tc_elect_one()) {
#pragma unroll
                        for (int sub = 0; sub < GG_SUB; ++sub) {
                            const unsigned char* sw = smem + stage * GG_STAGE_BYTES + sub * GP_STAGE_BYTES;
                            const uint64_t dw = tc_smem_desc(sw), dx = tc_smem_desc(sw + GP_A_BYTES);
#pragma unroll
                            for (int k = 0; k < GP_BK / 16; ++k)
                                gp_mma2(d_tmem, dw + 2 * k, dx + 2 * k, idesc, (kb > 0 || sub > 0 || k > 0) ? 1u : 0u);
                        }
                        gp_commit_both(&empty_bar[stage]);               // the stage is free in both blocks when these finish
                        if (kb + 1 == p.kblocks) gp_commit_both(&acc_full[acc]);
                    }
                    __syncwarp();
                }
                ++seg;
            }
            if (!ok && lane == 0 && p.status) atomicExch(p.status, 9);
        }
    } else {
        // ---------------- epilogue: eight warps, this block's 128 accumulator rows ----------------
        // A warp reads the 32 tensor-memory lanes of its number modulo four; warps 0..3 and 4..7 take turns at a tile's columns, 32 at a time.
        const int quarter = warp & 3, side = warp >> 2;
        const int row = quarter * 32 + lane;                // row of the block's half = tensor-memory lane
        const bool up_row = p.gated && quarter >= 2;
        float* swap = reinterpret_cast<float*>(smem + GG_STAGES * GG_STAGE_BYTES) + side * (2 * 16 * 64) + (row & 63);
        int seg = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles; tile += n_pairs) {
            const int tm = tile / p.tiles_n, tn = tile % p.tiles_n;
            int expert, row0, rows, columns;
            if (!gg_tile(p, tm, expert, row0, rows, columns)) continue;
            const int acc = seg & 1;
            if (ok) ok = tc_mbar_wait(&acc_full[acc], (seg >> 1) & 1);
            if (!ok) s_ok = 0;
            gp_bar_epilogue();
            if (!s_ok) { ok = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + acc * 256 + ((uint32_t)(quarter * 32) << 16);
            const int feature = p.gated ? tn * 128 + rank * 64 + (row & 63) : tn * 256 + rank * 128 + row;
            const bool live = feature < p.out_cols;
            const size_t at = (size_t)row0 * p.ldo + (live ? feature : 0);
            __nv_bfloat16* dst = (__nv_bfloat16*)p.out + at;
            float* dst32 = (float*)p.out + at;
#pragma unroll 1
            for (int c0 = side * 32; c0 < columns; c0 += 64) {
                float v[32];
                gp_row_chunk(taddr + c0, v);
                if (p.gated) {
                    // the gate rows' threads finish the first 16 columns, the up rows' threads the others
#pragma unroll
                    for (int j = 0; j < 16; ++j) swap[((up_row ? 16 : 0) + j) * 64] = up_row ? v[j] : v[16 + j];
                    asm volatile("bar.sync %0, 128;\n" ::"r"(2 + side) : "memory");
                    const int first = c0 + (up_row ? 16 : 0);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float theirs = swap[((up_row ? 0 : 16) + j) * 64];
                        float g = up_row ? theirs : v[j];
                        const float up = up_row ? v[16 + j] : theirs;
                        // the exponential as in moe.cu's tiles, which take the same rows at other sizes
                        if (p.act == PB_ACT_CLAMPED) g = pb_clamped_unit(g, up, p.limit, p.alpha);
                        else g = g / (1.0f + expf(-g)) * up;
                        if (live && first + j < rows) dst[(size_t)(first + j) * p.ldo] = __float2bfloat16_rn(g);
                    }
                    asm volatile("bar.sync %0, 128;\n" ::"r"(2 + side) : "memory");        // the halves have been read
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float f = p.act == PB_ACT_RELU2 ? pb_relu2(v[j]) : v[j];
                        if (live && c0 + j < rows) {
                            if (p.wide) dst32[(size_t)(c0 + j) * p.ldo] = f;
                            else dst[(size_t)(c0 + j) * p.ldo] = __float2bfloat16_rn(f);
                        }
                    }
                    __syncwarp();
                }
            }
            // the accumulator may be overwritten: tell the leading block, which issues the products
            tc_fence_before();
            __syncwarp();
            if (lane == 0) gp_arrive_cluster(gp_map_to_rank(tc_smem(&acc_empty[acc]), 0));
            ++seg;
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 10);
    }
    // nobody touches the other block's shared memory, barriers or tensor memory after this
    tc_fence_before();
    cluster.sync();
    if (warp == 9) {
        __syncwarp();
        tc_fence_after();
        gp_tmem_dealloc2(tmem_base, 512);
    }
}

}  // namespace

// A [places, K] holds the rows sorted by expert; B [n_experts * expert_rows_b, K] the experts' matrices one below the other; the
// device-side map (tile_expert, tile_row0 over max_m_tiles row tiles of 256, offsets) says which rows are whose.  out [places, N]
// bfloat16 (or float32: wide, plain form) with N = expert_rows_b, or, gated, N = expert_rows_b / 2 and silu(gate sums) * up sums (an expert's matrix: N gate rows,
// then N up rows); act: PbAct (plain: PB_ACT_NONE or PB_ACT_RELU2; gated: PB_ACT_SILU, or PB_ACT_CLAMPED with limit and alpha).
PB_API int pb_gemm_grouped_bf16(const void* A, const void* B, void* out, int places, int expert_rows_b, int n_experts, int K,
                                long long lda, long long ldb, long long ldo, int gated, int wide, int act, float limit, float alpha, const int32_t* tile_expert,
                                const int32_t* tile_row0, const int32_t* offsets, int max_m_tiles, int max_pairs,
                                int* status, cudaStream_t stream) {
    PB_REQUIRE(n_experts > 0 && max_m_tiles >= 0 && places > 0 && expert_rows_b > 0 && K >= 8 && K % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0 &&
                   (!gated || (expert_rows_b % 2 == 0 && !wide)),
               "gemm_grouped: places=%d rows per expert=%d K=%d lda=%lld ldb=%lld not taken", places, expert_rows_b, K, lda, ldb);
    PB_REQUIRE((long long)n_experts * expert_rows_b < (1ll << 31), "gemm_grouped: too many rows of B");
    PB_REQUIRE(A && B && out && tile_expert && tile_row0 && offsets && pb_aligned(A, 16) && pb_aligned(B, 16), "gemm_grouped: null or unaligned pointer");
    PB_REQUIRE(gated ? act == PB_ACT_SILU || (act == PB_ACT_CLAMPED && limit > 0.f) : act == PB_ACT_NONE || act == PB_ACT_RELU2,
               "gemm_grouped: activation %d in the %s form, limit %g", act, gated ? "gated" : "plain", (double)limit);
    if (max_m_tiles == 0) return 0;
    if (int e = get_encode()) return e;
    GgParams p{};
    p.out = out; p.wide = wide; p.status = status; p.ldo = ldo;
    p.out_cols = gated ? expert_rows_b / 2 : expert_rows_b;
    p.expert_rows = expert_rows_b; p.gated = gated ? 1 : 0; p.act = act; p.limit = limit; p.alpha = alpha;
    p.tiles_m = max_m_tiles;
    p.tiles_n = gated ? (p.out_cols + 127) / 128 : (p.out_cols + 255) / 256;
    p.kblocks = (K + GG_SUB * GP_BK - 1) / (GG_SUB * GP_BK);          // (a copy that starts behind K brings zeros)
    p.tile_expert = tile_expert; p.tile_row0 = tile_row0; p.offsets = offsets;
    const long long tiles = (long long)p.tiles_m * p.tiles_n;
    PB_REQUIRE(tiles < (1ll << 30), "gemm_grouped: %lld tiles are too many", tiles);
    long long pairs = gp_max_pairs();
    if (max_pairs > 0 && max_pairs < pairs) pairs = max_pairs;
    if (tiles < pairs) pairs = tiles;
    GgMaps maps;
    if (int e = gp_make_map(&maps.w, B, n_experts * expert_rows_b, K, ldb, gated ? 64 : 128)) return e;
    for (int i = 0; i < 3; ++i)
        if (int e = gp_make_map(&maps.x[i], A, places, K, lda, 128 >> i)) return e;
    const size_t smem = (size_t)GG_STAGES * GG_STAGE_BYTES + GG_SWAP + 1024;
    static const cudaError_t set = cudaFuncSetAttribute(gemm_grouped_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    PB_REQUIRE(set == cudaSuccess, "gemm_grouped: cannot get %zu bytes of shared memory: %s", smem, cudaGetErrorString(set));
    pb_launch(gemm_grouped_kernel, dim3((unsigned)(2 * pairs)), dim3(GP_THREADS), smem, stream, maps, p);
    PB_CHECK_LAUNCH("gemm_grouped");
    return 0;
}
