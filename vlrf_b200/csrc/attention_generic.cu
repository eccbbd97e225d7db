// Cache append and the general attention kernel over the paged cache.
//
// The cache of one layer is K and V of shape [block][kv_head][BT][head_dim]; a sequence's slot maps its
// positions to blocks through block_table[slot][pos / BT].  `kv_append` scatters the K and V columns of
// the fused projection into place (reference: include/model/kv_cache.hpp:215-251, before attention at
// include/model/attention.hpp:127-129).  `attn_generic` serves any mix of tokens: each (token, head) is
// one warp that walks the keys 0…pos of its slot in chunks of 32 with an online softmax in float32
// (reference: include/model/attention.hpp:207-309; scale :373-374; key visible iff k ≤ position
// :253-260).  It is the attention of the 32-bit path for prefill and decode, takes every head size that
// is a multiple of 16 up to 256 and any number of heads and groups, and is the fallback of the bfloat16
// path.  A window w > 0 hides keys at or before position − w.
#include "common.cuh"

namespace {

template <typename ET>
__global__ void kv_append_kernel(const ET* __restrict__ qkv, int ld, int k_off, int v_off,
                                 ET* __restrict__ Kc, ET* __restrict__ Vc,
                                 const int* __restrict__ block_table, int max_blocks,
                                 const int* __restrict__ tok_slot, const int* __restrict__ tok_pos,
                                 int Hkv, int dh, int BT, int* __restrict__ dev_err) {
    pdl_wait();                 // chained launch: nothing is read before the kernels ahead have finished
    pdl_launch_dependents();
    const int t = blockIdx.x;
    const int slot = tok_slot[t];
    if (slot < 0) return;  // padding row
    const int pos = tok_pos[t];
    const int bi = pos / BT;
    const int blk = (pos >= 0 && bi < max_blocks) ? block_table[(size_t)slot * max_blocks + bi] : -1;
    if (blk < 0) {
        if (threadIdx.x == 0) atomicOr(dev_err, VLRF_DEVERR_NO_BLOCK);
        return;
    }
    const int width = Hkv * dh;
    const ET* src = qkv + (size_t)t * ld;
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const int h = i / dh, c = i - h * dh;
        const size_t dst = (((size_t)blk * Hkv + h) * BT + (pos % BT)) * dh + c;
        Kc[dst] = src[k_off + i];
        Vc[dst] = src[v_off + i];
    }
}

// Loads that stay where they are written: left to itself the compiler sinks them to their uses, one wait each, to save registers.
__device__ __forceinline__ void load_now(const float* p, float (&v)[4]) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}
__device__ __forceinline__ void load_now(const __nv_bfloat16* p, uint4& v) {
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
}
__device__ __forceinline__ void load_now(const float* p, float& v) { asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p)); }
__device__ __forceinline__ void load_now(const __nv_bfloat16* p, float& v) {
    unsigned short u;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(u) : "l"(p));
    v = __uint_as_float((uint32_t)u << 16);
}
template <typename ET> struct Piece;                       // 16 bytes as they arrive
template <> struct Piece<float> {
    float v[4];
    __device__ __forceinline__ void load(const float* p) { load_now(p, v); }
    __device__ __forceinline__ float at(int i) const { return v[i]; }
};
template <> struct Piece<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { load_now(p, v); }
    __device__ __forceinline__ float at(int i) const {
        const uint32_t w = i < 2 ? v.x : i < 4 ? v.y : i < 6 ? v.z : v.w;
        return __uint_as_float((i & 1) ? w & 0xffff0000u : w << 16);
    }
};

constexpr int ATT_WARPS = 4;
constexpr int MAX_DH = 256;

// DH: the head size where it is known when compiling (0: the argument).  A key's row is asked for in runs of eight pieces of 16 bytes and the
// values of eight keys together, ahead of the sums that take them one after another: with a wait for every piece and every key 240 tokens of 12
// float32 heads of 64 took 67 us a layer, now 35 us.
template <typename ET, int DH>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attn_generic_kernel(const ET* __restrict__ qkv, int ld, int q_off, const ET* __restrict__ Kc,
                    const ET* __restrict__ Vc, const int* __restrict__ block_table, int max_blocks,
                    const int* __restrict__ tok_slot, const int* __restrict__ tok_pos,
                    ET* __restrict__ out, int ld_out, int H, int Hkv, int dh_arg, int BT, float scale,
                    int window, int* __restrict__ dev_err) {
    extern __shared__ __align__(16) float q_sm[];  // [ATT_WARPS][dh]
    constexpr int ND = DH > 0 ? (DH + 31) / 32 : MAX_DH / 32, N = 16 / (int)sizeof(ET);
    const int dh = DH > 0 ? DH : dh_arg;
    pdl_wait();                 // chained launch: nothing is read before the kernels ahead have finished
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int h = blockIdx.y * ATT_WARPS + warp;
    const int slot = tok_slot[t];
    if (h >= H || slot < 0) return;  // whole warp leaves together; no block-wide barrier below
    const int pos = tok_pos[t];
    const int hk = h / (H / Hkv);
    float* q = q_sm + warp * dh;
    const ET* qsrc = qkv + (size_t)t * ld + q_off + (size_t)h * dh;
    for (int i = lane; i < dh; i += 32) q[i] = ElemIO<ET>::load(qsrc + i) * scale;
    __syncwarp();

    float acc[ND];
#pragma unroll
    for (int i = 0; i < ND; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    const int first = (window > 0) ? max(0, pos - window + 1) : 0;
    const int* table = block_table + (size_t)slot * max_blocks;
    bool lost = false;

    for (int k0 = (first / 32) * 32; k0 <= pos; k0 += 32) {
        const int blk = table[k0 / BT];
        if (blk < 0) { lost = true; break; }
        const size_t base = (((size_t)blk * Hkv + hk) * BT + (k0 % BT)) * dh;
        const int key = k0 + lane;
        const bool valid = key >= first && key <= pos;
        float s = -INFINITY;
        if (valid) {
            const ET* krow = Kc + base + (size_t)lane * dh;
            float dot = 0.f;
            constexpr int RUN = 16 / N * 2;                     // pieces of 16 bytes that are asked for together (32 numbers)
#pragma unroll 2
            for (int c0 = 0; c0 < dh; c0 += RUN * N) {          // (head sizes are multiples of 16: the last run may be half)
                Piece<ET> kv[RUN];
#pragma unroll
                for (int i = 0; i < RUN; ++i)
                    if (c0 + i * N < dh) kv[i].load(krow + c0 + i * N);
#pragma unroll
                for (int i = 0; i < RUN; ++i)
                    if (c0 + i * N < dh) {
#pragma unroll
                        for (int j = 0; j < N; j += 4) {
                            const float4 qv = *reinterpret_cast<const float4*>(q + c0 + i * N + j);
                            dot = fmaf(qv.x, kv[i].at(j), dot);
                            dot = fmaf(qv.y, kv[i].at(j + 1), dot);
                            dot = fmaf(qv.z, kv[i].at(j + 2), dot);
                            dot = fmaf(qv.w, kv[i].at(j + 3), dot);
                        }
                    }
            }
            s = dot;
        }
        const float m_new = fmaxf(m, warp_max(s));      // at least one key of the chunk is valid
        const float p = valid ? expf(s - m_new) : 0.f;
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < ND; ++i) acc[i] *= corr;
        const int n_here = min(32, pos - k0 + 1);
        const ET* vbase = Vc + base;
        for (int j0 = 0; j0 < n_here; j0 += 8) {
            float v[8][ND];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < ND; ++i) {
                    const int c = i * 32 + lane;
                    v[j][i] = 0.f;
                    if (j0 + j < n_here && c < dh) load_now(vbase + (size_t)(j0 + j) * dh + c, v[j][i]);
                }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j0 + j);
                if (pj == 0.f) continue;                        // uniform across the warp (keys behind the last weigh nothing)
#pragma unroll
                for (int i = 0; i < ND; ++i) acc[i] = fmaf(pj, v[j][i], acc[i]);
            }
        }
        m = m_new;
    }
    if (lost && lane == 0) atomicOr(dev_err, VLRF_DEVERR_NO_BLOCK);
    const float inv = (l > 0.f) ? 1.f / l : 0.f;
    ET* dst = out + (size_t)t * ld_out + (size_t)h * dh;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        const int c = i * 32 + lane;
        if (c < dh) ElemIO<ET>::store(dst + c, acc[i] * inv);
    }
}
}  // namespace

extern "C" int vlrf_kv_append(const void* qkv, int dtype, int ld, int k_off, int v_off, void* Kc, void* Vc,
                              const int* block_table, int max_blocks, const int* tok_slot,
                              const int* tok_pos, int T, int Hkv, int dh, int BT, int* dev_err,
                              cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && Hkv > 0 && dh > 0 && BT > 0 && max_blocks > 0, "kv_append: bad sizes");
    VLRF_REQUIRE(dev_err != nullptr, "kv_append: needs the device error word");
    if (T == 0) return VLRF_OK;
    const int threads = (Hkv * dh >= 256) ? 256 : 128;
    if (dtype == VLRF_F32)
        launch_chained(kv_append_kernel<float>, dim3(T), dim3(threads), (size_t)0, stream, (const float*)qkv, ld, k_off, v_off, (float*)Kc,
                       (float*)Vc, block_table, max_blocks, tok_slot, tok_pos, Hkv, dh, BT, dev_err);
    else if (dtype == VLRF_BF16)
        launch_chained(kv_append_kernel<__nv_bfloat16>, dim3(T), dim3(threads), (size_t)0, stream, (const __nv_bfloat16*)qkv, ld, k_off, v_off,
                       (__nv_bfloat16*)Kc, (__nv_bfloat16*)Vc, block_table, max_blocks, tok_slot, tok_pos, Hkv, dh, BT, dev_err);
    else
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "kv_append: unknown dtype %d", dtype);
    return vlrf_check_launch("kv_append");
}

extern "C" int vlrf_attn_generic(const void* qkv, int dtype, int ld, int q_off, const void* Kc,
                                 const void* Vc, const int* block_table, int max_blocks,
                                 const int* tok_slot, const int* tok_pos, void* out, int ld_out, int T,
                                 int H, int Hkv, int dh, int BT, float scale, int window, int* dev_err,
                                 cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && H > 0 && Hkv > 0 && max_blocks > 0, "attention: bad sizes");
    VLRF_REQUIRE(H % Hkv == 0, "attention: %d heads cannot share %d key/value heads", H, Hkv);
    VLRF_REQUIRE(dh > 0 && dh % 16 == 0 && dh <= MAX_DH,
                 "attention: head size %d is not a multiple of 16 up to %d", dh, MAX_DH);
    VLRF_REQUIRE(BT % 32 == 0, "attention: cache blocks of %d tokens are not a multiple of 32", BT);
    VLRF_REQUIRE(window >= 0, "attention: negative window");
    VLRF_REQUIRE(dev_err != nullptr, "attention: needs the device error word");
    if (T == 0) return VLRF_OK;
    dim3 grid(T, (H + ATT_WARPS - 1) / ATT_WARPS);
    const size_t smem = (size_t)ATT_WARPS * dh * sizeof(float);
#define GO(ET, DHV) launch_chained(attn_generic_kernel<ET, DHV>, grid, dim3(ATT_WARPS * 32), smem, stream, (const ET*)qkv, ld, q_off, (const ET*)Kc, (const ET*)Vc, \
                                   block_table, max_blocks, tok_slot, tok_pos, (ET*)out, ld_out, H, Hkv, dh, BT, scale, window, dev_err)
    if (dtype == VLRF_F32) { if (dh == 64) GO(float, 64); else GO(float, 0); }
    else if (dtype == VLRF_BF16) { if (dh == 64) GO(__nv_bfloat16, 64); else GO(__nv_bfloat16, 0); }
    else
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "attention: unknown dtype %d", dtype);
#undef GO
    return vlrf_check_launch("attn_generic");
}
