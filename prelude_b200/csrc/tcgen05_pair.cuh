// What kernels on paired blocks (tcgen05.mma.cta_group::2: two multiprocessors share one tile) add to tcgen05.cuh: the sizes of a
// stage, copies counted on the leading block's barrier, the paired product and its commits.
#pragma once
#include "tcgen05.cuh"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define GP_BM 128                   // rows of A per block (256 per pair)
#define GP_BN 256                   // columns of the pair's tile (each block loads 128 rows of B)
#define GP_HALF 128
#define GP_BK 64
#define GP_STAGES 6
#define GP_THREADS 320                  // eight epilogue warps, one that copies, one that issues the products
#define GP_EPI_WARPS 8
#define GP_A_BYTES (GP_BM * GP_BK * 2)              // a stage's tile of A in one block
#define GP_STAGE_BYTES (2 * GP_A_BYTES)             // and as much of B

__device__ __forceinline__ uint32_t gp_map_to_rank(uint32_t smem_addr, uint32_t rank) {   // the same variable in another block of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void gp_tmem_alloc2(uint32_t* holder, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(holder)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void gp_tmem_dealloc2(uint32_t taddr, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols) : "memory");
}
// a tile copy into this block's shared memory whose bytes are counted on a barrier of the LEADING block
// (`leader_bar`: a cluster-wide address); both blocks of the pair issue it, each for its own halves
__device__ __forceinline__ void gp_tma_load_2d(void* smem, const CUtensorMap* map, int c0, int c1, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(tc_smem(smem)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void gp_mma2(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, unsigned accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// one arrival on the barrier at this address in BOTH blocks when the products issued so far have finished
__device__ __forceinline__ void gp_commit_both(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(tc_smem(bar)), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void gp_arrive_cluster(uint32_t bar) {      // `bar`: a cluster-wide address
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// bfloat16 x bfloat16 -> float32, M = 256 over the pair, N = n columns (a multiple of 32, at most 256), both operands K-major
__device__ __forceinline__ uint32_t gp_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}

__device__ __forceinline__ void gp_bar_epilogue() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }
// 32 columns of this thread's row of the accumulator
__device__ __forceinline__ void gp_row_chunk(uint32_t taddr, float* v) {
    uint32_t r[32];
    tc_tmem_ld32(taddr, r);
    tc_tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

static inline int gp_make_map(CUtensorMap* map, const void* ptr, int rows, int K, long long ld, int box_rows = 128) {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {GP_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return pb_fail("gemm_pair: cuTensorMapEncodeTiled failed with code %d (rows=%d K=%d ld=%lld)", (int)r, rows, K, ld);
    return 0;
}

static inline int gp_max_pairs() {
    static int pairs = 0;
    if (pairs == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        pairs = sms > 1 ? sms / 2 : 74;
    }
    return pairs;
}
