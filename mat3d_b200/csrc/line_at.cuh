// line_at.cuh -- warp-split line transforms that exchange through the line's own
// unpadded storage, and tile accesses, shared by the fused passes
// (passes_plane.cuh, passes_zmid.cuh).
#pragma once
#include "passes_fast.cuh"

namespace m3d {

// line_fwd / line_inv (fft_reg.cuh) with the exchange through at(k1, u):
// element k1*T + u of the line's own storage, u = t ^ k1/Q: consecutive lanes
// stay within an aligned run of T elements when writing and spread over the
// banks when reading, so no padding is needed
template <typename C2, int E, int T, class At>
__device__ __forceinline__ void line_fwd_at(C2 (&v)[E], int t, const C2* tw, At at) {
    constexpr int N = E * T, Q = E / T;
    dft_reg<C2, E, N>(v, tw, -1);
#pragma unroll
    for (int k1 = 1; k1 < E; ++k1) v[k1] = cmul(v[k1], twid(tw, t * k1, -1));
    __syncwarp();  // every lane of the line has read its inputs
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) *at(k1, t ^ (k1 / Q)) = v[k1];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        C2 u[T];
#pragma unroll
        for (int t2 = 0; t2 < T; ++t2) u[t2] = *at(t * Q + q, t2 ^ t);
        dft_reg<C2, T, N>(u, tw, -1);
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) v[q * T + k2] = u[k2];
    }
    __syncwarp();
}
template <typename C2, int E, int T, class At>
__device__ __forceinline__ void line_inv_at(C2 (&v)[E], int t, const C2* tw, At at) {
    constexpr int N = E * T, Q = E / T;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        C2 u[T];
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) u[k2] = v[q * T + k2];
        dft_reg<C2, T, N>(u, tw, +1);
        const int k1 = t * Q + q;
#pragma unroll
        for (int t2 = 0; t2 < T; ++t2) *at(k1, t2 ^ t) = (t2 == 0) ? u[t2] : cmul(u[t2], twid(tw, t2 * k1, +1));
    }
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) v[k1] = *at(k1, t ^ (k1 / Q));
    __syncwarp();
    dft_reg<C2, E, N>(v, tw, +1);
}

__device__ __forceinline__ void cp_async_c(float2* d, const float2* s) { cp_async(d, s, 8, 8); }
__device__ __forceinline__ void cp_async_c(double2* d, const double2* s) { cp_async(d, s, 16, 16); }

// W consecutive complex elements of a tile row
__device__ __forceinline__ void tile_get(const float2* p, float2 (&u)[2]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    u[0] = make_float2(v.x, v.y);
    u[1] = make_float2(v.z, v.w);
}
__device__ __forceinline__ void tile_put(float2* p, const float2 (&u)[2]) {
    *reinterpret_cast<float4*>(p) = make_float4(u[0].x, u[0].y, u[1].x, u[1].y);
}
template <typename C2> __device__ __forceinline__ void tile_get(const C2* p, C2 (&u)[1]) { u[0] = *p; }
template <typename C2> __device__ __forceinline__ void tile_put(C2* p, const C2 (&u)[1]) { *p = u[0]; }

}  // namespace m3d
