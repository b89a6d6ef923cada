// Helpers of the recurrences whose state columns are independent of one another (gated_delta.cu, general_delta.cu): L neighbouring lanes own a
// column, lane part p holds the key channels {4 (i L + p) .. + 3} as NV float4, sums along a column meet by shuffles over the L lanes.
#pragma once
#include <cstdint>

namespace uzu {

__device__ __forceinline__ void gd_cp_async16(void* smem_ptr, const void* gmem_ptr) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_ptr)), "l"(gmem_ptr) : "memory");
}
__device__ __forceinline__ void gd_cp_async4(void* smem_ptr, const void* gmem_ptr) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_ptr)), "l"(gmem_ptr) : "memory");
}

template <int L>
__device__ __forceinline__ float gd_lane_sum(float v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// v[0] of lane part p <- the sum over the L lanes of a column of v[p / (L / U)]  (U values, U <= L, both powers of two)
template <int U, int L>
__device__ __forceinline__ void gd_transpose_sum(float (&v)[U], uint32_t part) {
    int n = U;
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = (part & o) != 0;
#pragma unroll
            for (int i = 0; i < U / 2; ++i) {
                if (i < n) {
                    const float keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
}

template <int NV>
__device__ __forceinline__ float gd_dot(const float4 (&a)[NV], const float4 (&b)[NV]) {
    float x = 0.0f, y = 0.0f, z = 0.0f, w = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        x = fmaf(a[i].x, b[i].x, x);
        y = fmaf(a[i].y, b[i].y, y);
        z = fmaf(a[i].z, b[i].z, z);
        w = fmaf(a[i].w, b[i].w, w);
    }
    return (x + y) + (z + w);
}

// S <- g S + k u on a lane's channels
template <int NV>
__device__ __forceinline__ void gd_update(float4 (&s)[NV], const float4 (&k)[NV], float g, float u) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        s[i].x = fmaf(k[i].x, u, g * s[i].x);
        s[i].y = fmaf(k[i].y, u, g * s[i].y);
        s[i].z = fmaf(k[i].z, u, g * s[i].z);
        s[i].w = fmaf(k[i].w, u, g * s[i].w);
    }
}

}  // namespace uzu
