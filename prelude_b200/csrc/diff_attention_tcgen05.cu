// Differential attention of prompt portions on the fifth-generation tensor cores (tcgen05), bfloat16 operands, float32 scores, weights, sums
// and epilogue: for a query at position p and head h
//     o = softmax(temp(p) scale q1 . k1_j) v_j  -  lambda softmax(temp(p) scale q2 . k2_j) v_j     over max(0, p - window + 1) <= j <= p
// brought to unit root mean square, times a scale and the sigmoid of a gate.
//
// A block takes 128 query rows - 128 / G tokens of one request times the G query heads of one key/value head - as two row tiles of 128: the
// rows' first and their second queries.  It walks the visible keys in tiles of 128; the maps have keys of their own and share the values,
// which are fetched once.  The two maps are to each other what the two row tiles of attention_prefill_tc.cu are: warps 0-3 and 4-7
// are their softmax groups (thread = row = tensor-memory lane), warp 8 brings the tiles, warp 9 issues the products, one map's while
// the other is in its softmax: S_0(0) S_1(0) | PV_0(j) S_0(j+1) PV_1(j) S_1(j+1) | ..  (Two threads a row, sixteen warps: the units are no less
// busy and everybody waits longer, 45 us for 34.)
//
// The weights enter the second product as two bfloat16 numbers, their rounding and what that left, which together take the 128
// columns of tensor memory that their scores had: the difference of two nearly equal maps inherits no rounding of its weights, and a
// maximum may grow by 2^8 before the sums are rescaled.  Tensor memory: S_0, S_1, O_0, O_1, 128 columns each (O: value size).
//
// At the end a row's two results lie in the same lane: each of its two threads makes half of the columns of the difference, the
// halves' sums of squares meet in shared memory, and each writes its half.
//
// What bounds it: a map's chain from tile to tile - scores out of tensor memory and their maximum 450 cycles, exponentials and conversions
// 2,300 (with the other map's beside them), the two products 1,460 - 5,100 cycles in all, in which the tensor cores work half of the time.
//
// Measured against the mma.sync kernel (diff_attention_tc.cu), us: 16 heads over 4 of 64 and 128, 1,024 tokens 106 -> 34, 4,096 tokens
// 720 -> 198, 64 tokens 23 -> 14, 64 behind 2,000 90 -> 57; 32 heads over 8, 1,024 tokens 181 -> 46.  512 tokens beside 16 single ones behind
// 2,000: 129 -> 57 with all of them here (165 with the single ones there).  Distance from 64 bits of a layer of 1,024 tokens 4.3e-3 -> 4.0e-3.
#include "attention_common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int DT_KEYS = 128, DT_THREADS = 320, DT_SLAB = 128 * 128;          // a slab: 128 rows of 64 elements
constexpr float DT_GROWTH = 8.0f;

// KH, VH: 64-column slabs of a query or key row, of a value row.
template <int KH, int VH>
struct DtTiling {
    static constexpr int Q_BYTES = 2 * KH * DT_SLAB, K_BYTES = 2 * KH * DT_SLAB, V_BYTES = VH * DT_SLAB;   // queries and keys of both maps
    static constexpr int STAGES = 2, VD = VH * 64, O_COL = 256;
    static constexpr int SMEM = Q_BYTES + STAGES * (K_BYTES + V_BYTES) + 1024;
};

struct DtParams {
    __nv_bfloat16* out;                                     // [T, heads, vdim]
    const __nv_bfloat16* gate; long long gate_stride;       // [T, heads * vdim] or null
    const int32_t* block_table; const int32_t* token_row; const int32_t* cu_q; const int32_t* q_start; const int32_t* tile_seq; const int32_t* tile_tok0;
    int table_stride, page_size, num_pages, n_heads, n_kv_heads, window, tok, kv_rows;       // tok: tokens of a block, 128 / group
    float scale_log2, temp_coef; int temp_every;
    float lambda, norm_eps, out_scale;
    int* status;
};

__device__ __forceinline__ void dt_bar_groups() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }
__device__ __forceinline__ void dt_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

template <int KH, int VH>
__global__ void __launch_bounds__(DT_THREADS, 1)
diff_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, DtParams p) {
    pb_grid_dep_launch();
    using T = DtTiling<KH, VH>;
    constexpr int ST = T::STAGES, HALF = T::VD / 2;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* sQ = smem;
    unsigned char* sKr = smem + T::Q_BYTES;
    unsigned char* sVr = sKr + ST * T::K_BYTES;
    __shared__ __align__(8) uint64_t q_full, k_full[ST], v_full[ST], k_empty[ST], v_empty[ST], s_full[2], p_full[2], o_full[2];
    __shared__ uint32_t tmem_holder;
    __shared__ float s_inv[2][128], s_ss[2][128];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int TOK = p.tok, G = 128 / TOK, ps = p.page_size;
    const int tile = blockIdx.x / p.n_kv_heads, kvh = blockIdx.x - tile * p.n_kv_heads;
    const int r = p.tile_seq[tile], tok0 = p.tile_tok0[tile];
    const int q_base = p.cu_q[r], pos0 = p.q_start[r];
    const int n_tok = min(TOK, p.cu_q[r + 1] - q_base - tok0);   // tokens of this block
    const int p_min = pos0 + tok0, p_max = p_min + n_tok - 1;
    const int lo = p.window > 0 ? max(0, p_min - p.window + 1) : 0;
    const int kt0 = lo / DT_KEYS, n_tiles = p_max / DT_KEYS - kt0 + 1;
    const int lo_run = lo / p.kv_rows * p.kv_rows;               // first key of the first run that holds a visible key

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        for (int s = 0; s < ST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        for (int m = 0; m < 2; ++m) { mbar_init(&s_full[m], 1); mbar_init(&p_full[m], 128); mbar_init(&o_full[m], 1); }
        mbar_fence_init();
    }
    if (warp == 9) tc_tmem_alloc(&tmem_holder, 512);
    if (warp == 8 && lane == 0) { tc_prefetch_map(&map_q); tc_prefetch_map(&map_k); tc_prefetch_map(&map_v); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_holder;

    if (warp == 8) {
        // ---------------- loads: lane u brings the u-th run of a tile ----------------
        const int32_t* table = p.block_table + (size_t)p.token_row[q_base + tok0] * p.table_stride;
        const int runs = DT_KEYS / p.kv_rows;
        const int hi_run = p_max / p.kv_rows * p.kv_rows;        // first key of the last run that holds a visible key
        pb_grid_dep_wait();                                      // the queries and the newest keys and values are earlier kernels'
        if (lane == 0) {
            mbar_arrive_expect_tx(&q_full, T::Q_BYTES);
            for (int hg = 0; hg < G; ++hg)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int h = 0; h < KH; ++h)
                        tc_tma_load_3d(sQ + (m * KH + h) * DT_SLAB + hg * TOK * 128, &map_q, h * 64, (kvh * G + hg) * 2 + m, q_base + tok0, &q_full);
        }
        __syncwarp();
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < n_tiles; ++j) {
            // Runs without a visible key (before the window, after the last key) are read from the nearest run that has one: their
            // weights are zero, and the value rows are cleared by the softmax threads.
            const int j0 = min(max((kt0 + j) * DT_KEYS + min(lane, runs - 1) * p.kv_rows, lo_run), hi_run);
            int page = table[j0 / ps];
            const int row = j0 % ps;
            if (page < 0 || page >= p.num_pages) {               // never read outside the pool; the step is reported as bad
                page = 0;
                if (lane < runs && p.status) atomicExch(p.status, 6);
            }
            const int stage = j % ST;
            const unsigned phase = (j / ST) & 1;
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&k_empty[stage], phase ^ 1));
            if (!ok) break;
            if (lane == 0) mbar_arrive_expect_tx(&k_full[stage], T::K_BYTES);
            __syncwarp();
            if (lane < runs) {
                unsigned char* dst = sKr + stage * T::K_BYTES + lane * p.kv_rows * 128;
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int h = 0; h < KH; ++h) tc_tma_load_5d(dst + (m * KH + h) * DT_SLAB, &map_k, 0, h, row, 2 * kvh + m, page, &k_full[stage]);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&v_empty[stage], phase ^ 1));
            if (!ok) break;
            if (lane == 0) mbar_arrive_expect_tx(&v_full[stage], T::V_BYTES);
            __syncwarp();
            if (lane < runs) {
                unsigned char* dst = sVr + stage * T::V_BYTES + lane * p.kv_rows * 128;
#pragma unroll
                for (int h = 0; h < VH; ++h) tc_tma_load_5d(dst + h * DT_SLAB, &map_v, 0, h, row, kvh, page, &v_full[stage]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 7);
    } else if (warp == 9) {
        // ---------------- products: the whole warp walks, one thread issues ----------------
        const uint32_t idesc_s = tc_instr_desc(DT_KEYS), idesc_o = tc_instr_desc(T::VD, true);
        bool ok = true;
        auto wait_all = [&](uint64_t* bar, unsigned parity) {
            ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(bar, parity));
            return ok;
        };
        auto issue_s = [&](int m, int stage) {
            tc_fence_after();
            if (tc_elect_one()) {
                const uint64_t dq = tc_smem_desc(sQ + m * KH * DT_SLAB), dk = tc_smem_desc(sKr + stage * T::K_BYTES + m * KH * DT_SLAB);
#pragma unroll
                for (int ks = 0; ks < KH * 4; ++ks) {
                    const unsigned off = ((ks >> 2) * DT_SLAB + (ks & 3) * 32) >> 4;
                    tc_mma(tmem_base + m * 128, dq + off, dk + off, idesc_s, ks > 0 ? 1u : 0u);
                }
                tc_commit(&s_full[m]);
                if (m == 1) tc_commit(&k_empty[stage]);
            }
            __syncwarp();
        };
        auto issue_o = [&](int m, int stage, bool first, bool last) {
            tc_fence_after();
            if (tc_elect_one()) {
                const uint64_t dv = tc_smem_desc_mn(sVr + stage * T::V_BYTES, DT_SLAB);
                const uint32_t d = tmem_base + T::O_COL + m * T::VD, w = tmem_base + m * 128;
#pragma unroll
                for (int part = 1; part >= 0; --part)            // the small parts first
#pragma unroll
                    for (int ks = 0; ks < DT_KEYS / 16; ++ks)
                        tc_mma_ts(d, w + part * 64 + ks * 8, dv + ((ks * 16 * 128) >> 4), idesc_o, (!first || part == 0 || ks > 0) ? 1u : 0u);
                if (last) tc_commit(&o_full[m]);
                if (m == 1) tc_commit(&v_empty[stage]);
            }
            __syncwarp();
        };
        if (wait_all(&q_full, 0) && wait_all(&k_full[0], 0)) {
            issue_s(0, 0);
            issue_s(1, 0);
        }
#pragma unroll 1
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int stage = j % ST, next = (j + 1) % ST;
            for (int m = 0; m < 2 && ok; ++m) {
                if (!wait_all(&p_full[m], j & 1)) break;
                if (m == 0 && !wait_all(&v_full[stage], (j / ST) & 1)) break;
                issue_o(m, stage, j == 0, j == n_tiles - 1);
                if (j + 1 < n_tiles) {
                    if (m == 0 && !wait_all(&k_full[next], ((j + 1) / ST) & 1)) break;
                    issue_s(m, next);
                }
            }
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 9);
    } else {
        // ---------------- softmax: thread = row ----------------
        const int m = warp >> 2, R = (warp & 3) * 32 + lane;
        const int hg = R / TOK, tl = R - hg * TOK;
        const bool valid = tl < n_tok;
        const int row_pos = p_min + min(tl, n_tok - 1);          // rows without a token behave like the last token
        const int row_lo = p.window > 0 ? row_pos - p.window + 1 : 0;
        const float sc = p.scale_log2 * (p.temp_coef == 0.f ? 1.0f : 1.0f + p.temp_coef * logf((float)((row_pos + 1) / p.temp_every + 1)));
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t s_addr = lane_base + m * 128, o_addr = lane_base + T::O_COL;
        float m_ref = -INFINITY, l = 0.f;
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < n_tiles; ++j) {
            ok = ok && mbar_wait_bounded(&s_full[m], j & 1);
            tc_fence_after();
            uint32_t sr[DT_KEYS];
#pragma unroll
            for (int c = 0; c < DT_KEYS; c += 32) tc_tmem_ld32(s_addr + c, sr + c);
            tc_tmem_ld_wait();
            const int key0 = (kt0 + j) * DT_KEYS;
            if (key0 + DT_KEYS - 1 > row_pos || key0 < row_lo) {
#pragma unroll
                for (int c = 0; c < DT_KEYS; ++c)
                    if (key0 + c > row_pos || key0 + c < row_lo) sr[c] = __float_as_uint(-INFINITY);
            }
            float mx[8];                                         // eight chains side by side
#pragma unroll
            for (int i = 0; i < 8; ++i) mx[i] = __uint_as_float(sr[i]);
#pragma unroll
            for (int c = 8; c < DT_KEYS; ++c) mx[c & 7] = fmaxf(mx[c & 7], __uint_as_float(sr[c]));
            const float rmax = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
            const float cand = fmaxf(m_ref, rmax * sc);          // the factor is positive: the maximum commutes with it
            if (__any_sync(0xffffffffu, cand > m_ref + DT_GROWTH)) {       // (also from -inf to a number)
                const float corr = m_ref == -INFINITY ? 0.f : ex2_approx(m_ref - cand);
                m_ref = cand;
                l *= corr;
                if (j > 0) {                                     // the sums hold something: no product is writing them now
#pragma unroll 1
                    for (int c = 0; c < T::VD; c += 32) {
                        uint32_t orr[32];
                        tc_tmem_ld32(o_addr + m * T::VD + c, orr);
                        tc_tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * corr);
                        tc_tmem_st32(o_addr + m * T::VD + c, orr);
                    }
                }
            }
            const float mref = m_ref == -INFINITY ? 0.f : m_ref;
            float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < DT_KEYS; c += 32) {
                uint32_t hi[16], rest[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float p0 = ex2_approx(fmaf(__uint_as_float(sr[c + 2 * i]), sc, -mref));
                    const float p1 = ex2_approx(fmaf(__uint_as_float(sr[c + 2 * i + 1]), sc, -mref));
                    ls[i & 3] += p0 + p1;
                    const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
                    const float2 f = __bfloat1622float2(b);
                    hi[i] = *reinterpret_cast<const uint32_t*>(&b);
                    rest[i] = pack_bf16(p0 - f.x, p1 - f.y);
                }
                tc_tmem_st16(s_addr + (c >> 1), hi);
                tc_tmem_st16(s_addr + 64 + (c >> 1), rest);
            }
            l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
            // Value rows of keys that nobody may see hold whatever their page holds, and 0 x NaN is NaN: each group clears them once
            // the tile has landed and before it lets its product start.  Only the first and the last tile have such rows.
            const int clear_below = j == 0 ? lo_run - key0 : 0, clear_from = j == n_tiles - 1 ? p_max + 1 - key0 : DT_KEYS;
            if (clear_below > 0 || clear_from < DT_KEYS) {
                const int stage = j % ST;
                ok = ok && mbar_wait_bounded(&v_full[stage], (j / ST) & 1);
                unsigned char* sV = sVr + stage * T::V_BYTES;
#pragma unroll 1
                for (int idx = R; idx < DT_KEYS * VH * 8; idx += 128) {
                    const int row = idx / (VH * 8), rest = idx - row * (VH * 8);
                    if (ok && (row < clear_below || row >= clear_from))
                        *reinterpret_cast<uint4*>(sV + (rest >> 3) * DT_SLAB + row * 128 + (rest & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
            }
            tc_tmem_st_wait();
            tc_fence_before();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&p_full[m])) : "memory");
        }
        // ---------------- the head's epilogue: this group's half of the columns ----------------
        // (Eight columns at a time, in loops that stay loops: what runs once in a block waits for its instructions.)
        const int col0 = m * HALF;
        const int token = q_base + tok0 + (valid ? tl : 0), head = kvh * G + hg;
        const __nv_bfloat16* gate = p.gate == nullptr ? nullptr : p.gate + (size_t)token * p.gate_stride + (size_t)head * T::VD + col0;
        uint4 g = gate ? *reinterpret_cast<const uint4*>(gate) : make_uint4(0u, 0u, 0u, 0u);       // asked for while the last products run
        s_inv[m][R] = l > 0.f ? 1.0f / l : 0.f;
        ok = ok && mbar_wait_bounded(&o_full[0], 0) && mbar_wait_bounded(&o_full[1], 0);
        tc_fence_after();
        dt_bar_groups();
        const float inv0 = s_inv[0][R], inv1 = s_inv[1][R] * p.lambda;
        auto columns = [&](int c, float (&v)[8]) {
            uint32_t a[8], b[8];
            dt_ld8(o_addr + col0 + c, a);
            dt_ld8(o_addr + T::VD + col0 + c, b);
            tc_tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(a[i]) * inv0 - __uint_as_float(b[i]) * inv1;
        };
        float ss = 0.f;
#pragma unroll 1
        for (int c = 0; c < HALF; c += 8) {
            float v[8];
            columns(c, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
        }
        s_ss[m][R] = ss;
        dt_bar_groups();
        const float f = p.out_scale / sqrtf((s_ss[0][R] + s_ss[1][R]) / (float)T::VD + p.norm_eps);
        __nv_bfloat16* dst = p.out + ((size_t)token * p.n_heads + head) * T::VD + col0;
#pragma unroll 1
        for (int c = 0; c < HALF; c += 8) {
            float v[8];
            columns(c, v);
            const uint4 now = g;
            if (gate && c + 8 < HALF) g = *reinterpret_cast<const uint4*>(gate + c + 8);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&now);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 z = __bfloat1622float2(h[u]);
                v[2 * u] *= gate ? f * pb_sigmoid_for<__nv_bfloat16>(z.x) : f;
                v[2 * u + 1] *= gate ? f * pb_sigmoid_for<__nv_bfloat16>(z.y) : f;
            }
            if (valid && ok)
                *reinterpret_cast<uint4*>(dst + c) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 10);
    }
    // everybody is done with tensor memory
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        __syncwarp();
        tc_fence_after();
        tc_tmem_dealloc(tmem_base, 512);
    }
}

int dt_encode(CUtensorMap* map, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
              CUtensorMapSwizzle swizzle, const char* what) {
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : pb_fail("diff_attention_tcgen05: cuTensorMapEncodeTiled failed with code %d for %s", (int)r, what);
}

template <int KH, int VH>
int dt_launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const DtParams& p, int n_tiles, cudaStream_t stream) {
    using T = DtTiling<KH, VH>;
    static const cudaError_t set = cudaFuncSetAttribute(diff_attention_tcgen05_kernel<KH, VH>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
    PB_REQUIRE(set == cudaSuccess, "diff_attention_tcgen05: cannot get %d bytes of shared memory: %s", T::SMEM, cudaGetErrorString(set));
    pb_launch(diff_attention_tcgen05_kernel<KH, VH>, dim3((unsigned)n_tiles * p.n_kv_heads), dim3(DT_THREADS), (size_t)T::SMEM, stream, mq, mk, mv, p);
    PB_CHECK_LAUNCH("diff_attention_tcgen05");
    return 0;
}

}  // namespace

// Keys of 64, values of 64 or 128, a power of two of at most 16 query heads per key/value head, pages whose runs tile 128 keys evenly,
// rows in 16-byte pieces.
PB_API int pb_diff_attention_tcgen05_supported(int n_heads, int n_kv_heads, int dim, int vdim, int page_size, long long q_stride, const void* q,
                                               long long gate_stride, const void* gate) {
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads) return 0;
    const int g = n_heads / n_kv_heads;
    return (g & (g - 1)) == 0 && g <= 16 && dim == 64 && (vdim == 64 || vdim == 128) && page_size > 0 && page_size % 8 == 0 &&
           (DT_KEYS % page_size == 0 || page_size % DT_KEYS == 0) && q_stride % 8 == 0 && pb_aligned(q, 16) && (!gate || (gate_stride % 8 == 0 && pb_aligned(gate, 16)));
}

// Tokens of one tile of the host's list for this kernel.
PB_API int pb_diff_attention_tcgen05_tile_tokens(int n_heads, int n_kv_heads) { return 128 / (n_heads / n_kv_heads); }

// Operands as for pb_diff_attention_tc_bf16; q_start [requests] the position of each portion's first token; tiles: of prompt portions, 128 /
// (n_heads / n_kv_heads) tokens each.  scale > 0, temp_coef >= 0.
PB_API int pb_diff_attention_tcgen05_bf16(const void* q, long long q_stride, const void* gate, long long gate_stride, const void* k_pages,
                                          const void* v_pages, void* out, const int32_t* block_table, int table_stride, const int32_t* token_row,
                                          const int32_t* cu_q, const int32_t* q_start, const int32_t* tile_seq, const int32_t* tile_tok0, int n_tiles,
                                          int page_size, int num_pages, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim, float scale,
                                          float temp_coef, int temp_every, float lambda, float norm_eps, float out_scale, int window, int k_swizzle,
                                          int v_swizzle, int* status, cudaStream_t stream) {
    PB_REQUIRE(pb_diff_attention_tcgen05_supported(n_heads, n_kv_heads, dim, vdim, page_size, q_stride, q, gate_stride, gate),
               "diff_attention_tcgen05: heads %d over %d, dim %d, vdim %d, pages of %d not taken", n_heads, n_kv_heads, dim, vdim, page_size);
    PB_REQUIRE(q && k_pages && v_pages && out && block_table && token_row && cu_q && q_start && (n_tiles == 0 || (tile_seq && tile_tok0)) && num_pages > 0 &&
                   table_stride > 0 && temp_every > 0 && window >= 0,
               "diff_attention_tcgen05: null pointer or bad geometry");
    PB_REQUIRE(scale > 0.f && temp_coef >= 0.f, "diff_attention_tcgen05: scale %g, temperature %g: the kernel takes the maximum before them", (double)scale, (double)temp_coef);
    PB_REQUIRE(pb_aligned(k_pages, 16) && pb_aligned(v_pages, 16) && pb_aligned(out, 16), "diff_attention_tcgen05: unaligned pages or result");
    PB_REQUIRE(n_tiles >= 0 && (long long)n_tiles * n_kv_heads < (1ll << 31), "diff_attention_tcgen05: bad grid");
    if (n_tiles == 0 || n_tokens == 0) return 0;
    if (int e = get_encode()) return e;
    DtParams p{};
    p.out = (__nv_bfloat16*)out; p.gate = (const __nv_bfloat16*)gate; p.gate_stride = gate_stride; p.block_table = block_table; p.token_row = token_row;
    p.cu_q = cu_q; p.q_start = q_start; p.tile_seq = tile_seq; p.tile_tok0 = tile_tok0; p.table_stride = table_stride; p.page_size = page_size;
    p.num_pages = num_pages; p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.window = window; p.tok = 128 / (n_heads / n_kv_heads);
    p.kv_rows = page_size < DT_KEYS ? page_size : DT_KEYS;
    p.scale_log2 = scale * 1.4426950408889634f; p.temp_coef = temp_coef; p.temp_every = temp_every; p.lambda = lambda; p.norm_eps = norm_eps;
    p.out_scale = out_scale; p.status = status;
    CUtensorMap mq, mk, mv;
    {
        cuuint64_t dims[3] = {(cuuint64_t)dim, (cuuint64_t)n_heads * 2, (cuuint64_t)n_tokens};
        cuuint64_t strides[2] = {(cuuint64_t)dim * 2, (cuuint64_t)q_stride * 2};
        cuuint32_t box[3] = {64, 1, (cuuint32_t)p.tok};
        if (int e = dt_encode(&mq, q, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "q")) return e;
    }
    for (int which = 0; which < 2; ++which) {
        const cuuint64_t size = which ? vdim : dim, heads = which ? n_kv_heads : 2 * n_kv_heads, row = size * 2;
        cuuint64_t dims[5] = {64, size / 64, (cuuint64_t)page_size, heads, (cuuint64_t)num_pages};
        cuuint64_t strides[4] = {128, row, row * page_size, row * page_size * heads};
        cuuint32_t box[5] = {64, 1, (cuuint32_t)p.kv_rows, 1, 1};
        // (pages with permuted chunks lie as the products want them; of others the copies permute)
        if (int e = dt_encode(which ? &mv : &mk, which ? v_pages : k_pages, 5, dims, strides, box,
                              (which ? v_swizzle : k_swizzle) ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, which ? "the value pages" : "the key pages")) return e;
    }
    return vdim == 64 ? dt_launch<1, 1>(mq, mk, mv, p, n_tiles, stream) : dt_launch<1, 2>(mq, mk, mv, p, n_tiles, stream);
}
