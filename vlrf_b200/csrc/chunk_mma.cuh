// What the chunked recurrences share: asynchronous copies, fragments for `mma.sync` on bfloat16, and float32 numbers as sums of
// bfloat16 ones.
#pragma once
#include "common.cuh"

__device__ __forceinline__ uint32_t fc_sm(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, or zeros where there is nothing
__device__ __forceinline__ void fc_cp16(void* dst, const void* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(fc_sm(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fc_ldsm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void fc_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void fc_ldsm_t2(uint32_t& r0, uint32_t& r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void fc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two numbers as the sum of two pairs of bfloat16
__device__ __forceinline__ void fc_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// … of three: all 24 bits of a float32 (the differences are exact)
__device__ __forceinline__ void fc_split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    x -= __low2float(h); y -= __high2float(h);
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(m), y - __high2float(m));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// c += a · b, a and b in three parts each: the six products of parts that reach 2^-24 of the whole, the smallest first, in a sum of
// their own.  (The tensor cores cut a sum's last bits off instead of rounding it: added to c one by one, six cuts at the size of c
// each time made the error of a result 1.7 times that of float32 FMAs; this way one is at the size of these 16 terms.)
__device__ __forceinline__ void fc_mma3(float (&c)[4], const uint32_t (&a)[3][4], uint32_t h0, uint32_t h1, uint32_t m0, uint32_t m1, uint32_t l0,
                                        uint32_t l1) {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    fc_mma(t, a[2], h0, h1);
    fc_mma(t, a[0], l0, l1);
    fc_mma(t, a[1], m0, m1);
    fc_mma(t, a[1], h0, h1);
    fc_mma(t, a[0], m0, m1);
    fc_mma(t, a[0], h0, h1);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += t[i];
}
