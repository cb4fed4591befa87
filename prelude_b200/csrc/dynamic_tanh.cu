// A squashing in a norm's place, fused with the residual add:
//
//   res += x ;  y = tanh(slope * res) * w + b          (all arithmetic in float32, one rounding at the store)
//
// Nothing is summed over a row, so the kernel is element by element: a thread owns 16 bytes of a row's output and waits for
// no other.  With `rows` (the gather form) row i of y is made from row rows[i] of x and res, and res is
// left alone.  The residual stream is float32 in every mode.
#include "common.cuh"

#include <math.h>

namespace {

// V consecutive elements in 16-byte accesses (4 of float32, or 4 or 8 of bfloat16), or one
template <int V>
__device__ __forceinline__ void dt_ld(const float* p, float (&o)[V]) {
    if constexpr (V >= 4) {
#pragma unroll
        for (int e = 0; e < V; e += 4) {
            const float4 f = *reinterpret_cast<const float4*>(p + e);
            o[e] = f.x; o[e + 1] = f.y; o[e + 2] = f.z; o[e + 3] = f.w;
        }
    } else {
        o[0] = p[0];
    }
}
template <int V>
__device__ __forceinline__ void dt_ld(const __nv_bfloat16* p, float (&o)[V]) {
    if constexpr (V == 8) {
        const uint4 raw = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
    } else {
#pragma unroll
        for (int e = 0; e < V; ++e) o[e] = __bfloat162float(p[e]);
    }
}
template <int V>
__device__ __forceinline__ void dt_st(float* p, const float (&v)[V]) {
    if constexpr (V >= 4) {
#pragma unroll
        for (int e = 0; e < V; e += 4) *reinterpret_cast<float4*>(p + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
    } else {
        p[0] = v[0];
    }
}
template <int V>
__device__ __forceinline__ void dt_st(__nv_bfloat16* p, const float (&v)[V]) {
    if constexpr (V == 8) {
        uint4 raw;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4*>(p) = raw;
    } else {
#pragma unroll
        for (int e = 0; e < V; ++e) p[e] = __float2bfloat16_rn(v[e]);
    }
}

// x: n_parts arrays, part_stride elements apart, whose sum (in ascending order) is added; a block has blockDim.x * V columns
// of one row
template <typename TX, typename TY, int V>
__global__ void __launch_bounds__(256) add_tanh_kernel(const TX* x, int n_parts, size_t part_stride, float* res,
                                                       const int32_t* rows, int n_rows_total, float slope,
                                                       const float* w, const float* b, TY* y, int width) {
    pb_grid_dep_launch();
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * V;
    if (c >= width) return;
    float g[V], s[V];                                        // written by no kernel: before the wait
    dt_ld<V>(w + c, g);
    dt_ld<V>(b + c, s);
    pb_grid_dep_wait();
    TY* out = y + (size_t)blockIdx.x * width + c;
    const int src = rows ? rows[blockIdx.x] : (int)blockIdx.x;
    float v[V];
    if (src < 0 || src >= n_rows_total) {
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = 0.f;
        dt_st<V>(out, v);
        return;
    }
    float* r = res + (size_t)src * width + c;
    dt_ld<V>(r, v);
    if (x != nullptr) {
        const TX* xr = x + (size_t)src * width + c;
        for (int p0 = 0; p0 < n_parts; p0 += 4) {            // up to four parts' loads in flight
            float a[4][V];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (p0 + u < n_parts) dt_ld<V>(xr + (size_t)(p0 + u) * part_stride, a[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (p0 + u < n_parts) {
#pragma unroll
                    for (int e = 0; e < V; ++e) v[e] += a[u][e];
                }
        }
        if (rows == nullptr) dt_st<V>(r, v);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = pb_squash(v[e], slope, g[e], s[e]);
    dt_st<V>(out, v);
}

template <typename TX, typename TY>
int launch_add_tanh(const void* x, int n_parts, size_t part_stride, float* res, const int32_t* rows, int n_out, int n_rows_total, float slope,
                    const float* w, const float* b, void* y, int width, cudaStream_t stream) {
    constexpr int V = sizeof(TY) == 2 ? 8 : 4;
    const bool vec = width % V == 0 && part_stride % V == 0 && pb_aligned(res, 16) && pb_aligned(w, 16) && pb_aligned(b, 16) && pb_aligned(y, 16) &&
                     (x == nullptr || pb_aligned(x, 16));
    const int pieces = vec ? width / V : width;
    int threads = 32;
    while (threads < 256 && threads < pieces) threads <<= 1;
    PB_REQUIRE((pieces + threads - 1) / threads < 65536, "add_tanh: rows of %d", width);
    const dim3 grid(n_out, (pieces + threads - 1) / threads);
    if (vec)
        pb_launch(add_tanh_kernel<TX, TY, V>, grid, dim3(threads), 0, stream, (const TX*)x, n_parts, part_stride, res, rows, n_rows_total, slope, w, b,
                  (TY*)y, width);
    else
        pb_launch(add_tanh_kernel<TX, TY, 1>, grid, dim3(threads), 0, stream, (const TX*)x, n_parts, part_stride, res, rows, n_rows_total, slope, w, b,
                  (TY*)y, width);
    return 0;
}

}  // namespace

// x null, or of type dtype, or (x_parts > 0) that many float32 arrays [n_rows_total, width], part_stride elements apart, to
// be added up; res float32 [n_rows_total, width]; rows null (every row, res updated) or int32 [n_out] (those rows, res
// untouched); w, b float32 [width]; y [n_out, width] of type dtype.
PB_API int pb_add_tanh(const void* x, int x_parts, long long part_stride, float* res, const int32_t* rows, int n_out, int n_rows_total,
                       float slope, const float* w, const float* b, void* y, int dtype, int width, cudaStream_t stream) {
    PB_REQUIRE(n_out >= 0 && n_rows_total >= 0 && width > 0, "add_tanh: bad sizes");
    PB_REQUIRE(res && w && b && y, "add_tanh: null pointer");
    PB_REQUIRE(rows != nullptr || n_out == n_rows_total, "add_tanh: without chosen rows every row is made");
    PB_REQUIRE(x_parts >= 0 && x_parts <= 64 && (x_parts == 0 || (x && part_stride >= (long long)n_rows_total * width)),
               "add_tanh: %d parts %lld apart", x_parts, part_stride);
    if (n_out == 0) return 0;
    int e = 0;
    if (x_parts > 0) {
        PB_DISPATCH_DTYPE(dtype, T, (e = launch_add_tanh<float, T>(x, x_parts, (size_t)part_stride, res, rows, n_out, n_rows_total, slope, w, b, y, width, stream)));
    } else {
        PB_DISPATCH_DTYPE(dtype, T, (e = launch_add_tanh<T, T>(x, 1, (size_t)0, res, rows, n_out, n_rows_total, slope, w, b, y, width, stream)));
    }
    if (e) return e;
    PB_CHECK_LAUNCH("add_tanh");
    return 0;
}
