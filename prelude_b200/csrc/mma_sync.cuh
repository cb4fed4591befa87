// Warp-level products (mma.sync m16n8k16, bfloat16 operands, float32 sums) for the kernels whose tiles are too small for
// tcgen05, and float32 operands for them: a float32 number is the sum of three bfloat16 ones to its last bit (3 x 8 bits of
// mantissa), so a product of a float32 matrix with a bfloat16 one is three products, exact but for the float32 sums.
#pragma once

#include "common.cuh"

__device__ __forceinline__ unsigned pb_smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void pb_ldmatrix_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pb_ldmatrix_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pb_ldmatrix_x2_trans(unsigned& r0, unsigned& r1, unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pb_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void pb_cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(pb_smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void pb_cp_async_wait() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void pb_named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }

// two float32 numbers as three pairs of bfloat16: a + b = sum of the parts, largest first
__device__ __forceinline__ void pb_split3(float a, float b, unsigned (&out)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        out[i] = *reinterpret_cast<const unsigned*>(&h);
        const float2 f = __bfloat1622float2(h);
        a -= f.x;
        b -= f.y;
    }
}

// A product of two operands in three parts each, of whose nine products the six that reach float32's last bit are taken: the largest
// into `big`, the other five into `small`.  a: three parts of an A operand; b[p]: the two registers of an n8 tile of B's part p.
__device__ __forceinline__ void pb_mma6(float (&big)[4], float (&small)[4], const unsigned (&a)[3][4], const unsigned (&b)[3][2]) {
    pb_mma(small, a[2], b[0][0], b[0][1]);
    pb_mma(small, a[1], b[1][0], b[1][1]);
    pb_mma(small, a[0], b[2][0], b[2][1]);
    pb_mma(small, a[1], b[0][0], b[0][1]);
    pb_mma(small, a[0], b[1][0], b[1][1]);
    pb_mma(big, a[0], b[0][0], b[0][1]);
}

// Addresses for ldmatrix.x4 of a lane, in elements of a row-major tile with row stride `ld`:
//   an A operand [16 rows m][16 columns k]; and two n8 tiles of a B operand stored [k][n], read transposed (n 0-7: r0, r1;
//   n 8-15: r2, r3)
__device__ __forceinline__ int pb_a_offset(int lane, int ld) { return (lane & 15) * ld + (lane >> 4) * 8; }
__device__ __forceinline__ int pb_bt_offset(int lane, int ld) { return (lane & 15) * ld + (lane >> 4) * 8; }
//   two n8 tiles of a B operand stored [n][k] (n 0-7: r0, r1; n 8-15: r2, r3)
__device__ __forceinline__ int pb_b_offset(int lane, int ld) { return ((lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 8; }
//   an A operand stored transposed, [k][m]
__device__ __forceinline__ int pb_at_offset(int lane, int ld) { return ((lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 8; }
