// A LayerNorm row by a warp, the row in registers: what the norm's own kernel and the float32 product with a norm ahead share, so that
// both give the same bits (reference: include/model/ops.hpp:443-476).
#pragma once
#include "common.cuh"

namespace {
// Row `src` of nv float4s (at most 32·NV) into v, its mean and 1 / sqrt(variance + eps).
template <int NV>
__device__ __forceinline__ void layernorm_row(const float* src, int nv, int d, float eps, int lane, float4 (&v)[NV], float& mean, float& inv) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int i = j * 32 + lane;
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < nv)      // an explicit load: the values stay in registers for all three passes
            asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w) : "l"(src + 4 * i));
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
    mean = warp_sum(s) / (float)d;
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (j * 32 + lane < nv) {
            const float a = v[j].x - mean, b = v[j].y - mean, c = v[j].z - mean, e = v[j].w - mean;
            q += (a * a + b * b) + (c * c + e * e);
        }
    inv = 1.f / sqrtf(warp_sum(q) / (float)d + eps);
}
__device__ __forceinline__ float4 layernorm_apply(const float4& x, float mean, float inv, const float4& gm, const float4& bt) {
    return make_float4((x.x - mean) * inv * gm.x + bt.x, (x.y - mean) * inv * gm.y + bt.y, (x.z - mean) * inv * gm.z + bt.z,
                       (x.w - mean) * inv * gm.w + bt.w);
}
}  // namespace
