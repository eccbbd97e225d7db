// LayerNorm rows by a warp, the rows in registers: what the norm's own kernel and the float32 product with a norm ahead share, so that
// both give the same bits (reference: include/model/ops.hpp:443-476).
#pragma once
#include "common.cuh"

namespace {
// RW rows of nv float4s (at most 32·NV) into v, their means and 1 / sqrt(variance + eps); all rows are under way together.
template <int NV, int RW>
__device__ __forceinline__ void layernorm_rows(const float* const (&src)[RW], int nv, int d, float eps, int lane, float4 (&v)[RW][NV], float (&mean)[RW],
                                               float (&inv)[RW]) {
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int i = j * 32 + lane;
            v[r][j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < nv)      // an explicit load: the values stay in registers for all three passes
                asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[r][j].x), "=f"(v[r][j].y), "=f"(v[r][j].z), "=f"(v[r][j].w) : "l"(src[r] + 4 * i));
        }
    float s[RW], q[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        s[r] = q[r] = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) s[r] += (v[r][j].x + v[r][j].y) + (v[r][j].z + v[r][j].w);
    }
    auto sums = [](float (&x)[RW]) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < RW; ++r) x[r] += __shfl_xor_sync(0xffffffffu, x[r], o);
    };
    sums(s);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        mean[r] = s[r] / (float)d;
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (j * 32 + lane < nv) {
                const float a = v[r][j].x - mean[r], b = v[r][j].y - mean[r], c = v[r][j].z - mean[r], e = v[r][j].w - mean[r];
                q[r] += (a * a + b * b) + (c * c + e * e);
            }
    }
    sums(q);
#pragma unroll
    for (int r = 0; r < RW; ++r) inv[r] = 1.f / sqrtf(q[r] / (float)d + eps);
}
__device__ __forceinline__ float4 layernorm_apply(const float4& x, float mean, float inv, const float4& gm, const float4& bt) {
    return make_float4((x.x - mean) * inv * gm.x + bt.x, (x.y - mean) * inv * gm.y + bt.y, (x.z - mean) * inv * gm.z + bt.z,
                       (x.w - mean) * inv * gm.w + bt.w);
}
}  // namespace
