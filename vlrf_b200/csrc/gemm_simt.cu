// Y[M,N] = act(X[M,K] · W[N,K]^T + bias[N]) (+ residual[M,N]) on the CUDA cores with float32 FMAs.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode of reduced precision
// is involved) and the fallback of the bfloat16 path for shapes that the tensor-core kernels
// refuse.  W is kept [out, in] with `in` contiguous, so the product is the reference's
// linear(x, W) = x · Wᵀ (include/model/compute.hpp:64-68) with bias (include/model/attention.hpp:103-105),
// activation (include/model/feedforward.hpp:54-76) and residual (include/model/transformer_block.hpp:153,158)
// applied in the epilogue.
//
// A row's result does not depend on how many rows share the call: every kernel for a type forms an element's sum in
// one order.  In float32 that order is: K in PARTS = 8 runs of equal length (`part_length`), each a chain of FMAs in the
// order of k, the eight sums added in their order.  The parts are what a few rows are spread over the GPU by (a chain of
// all K terms in one thread took 104 us a product at 4 rows, whatever its size):
//   up to 8 rows     gemm_f32_norm_kernel: the next, with a LayerNorm ahead and a cache write behind, where all its CTAs find room at once
//   up to 16 rows    gemm_f32_rows_kernel: a thread per (column, part); bound by streaming W once
//   more rows        gemm_f32_tile_kernel: 64 x 64 tiles, the eight parts of a tile one CTA each of a cluster; bound by FMAs
// bfloat16 operands take gemm_simt_kernel (shapes outside the tensor-core kernels' rules: rare and small).
#include "common.cuh"
#include "layernorm_row.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;

template <typename IT, typename OT>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(const IT* __restrict__ X, const IT* __restrict__ W, const float* __restrict__ bias,
                 const float* residual, OT* Y, int M, int N, int K, int ldx, int ldy, int act) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lr = tid >> 2;         // 0..63: row of the tile this thread loads
    const int lk = (tid & 3) * 4;    // 0,4,8,12: first of its 4 k's
    const int ty = tid >> 4, tx = tid & 15;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            const int gm = m0 + lr, gn = n0 + lr;
            As[lk + j][lr] = (gm < M && k < K) ? ElemIO<IT>::load(X + (size_t)gm * ldx + k) : 0.f;
            Bs[lk + j][lr] = (gn < N && k < K) ? ElemIO<IT>::load(W + (size_t)gn * K + k) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            v = apply_act_rt(v, act);
            if (residual) v += residual[(size_t)m * ldy + n];
            ElemIO<OT>::store(Y + (size_t)m * ldy + n, v);
        }
    }
}
// ---- float32 ------------------------------------------------------------------------------------------------------------

constexpr int PARTS = 8;
constexpr int KB = 32;                 // numbers of k a stage of a ring holds, per part
constexpr int KPITCH = KB + 4;         // … and their pitch in shared memory: neighbours start one 16-byte bank group apart

__host__ __device__ inline int part_length(int K) { return ((K + PARTS - 1) / PARTS + 3) & ~3; }

template <int BYTES> __device__ __forceinline__ void cp_async_zfill(float* dst, const float* src, bool take) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = take ? BYTES : 0;    // (nothing is read where n is 0; the rest of the destination becomes zero)
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// KB numbers of row `row` from column k0 on into dst, zeros from column `end` on and for rows that are not there.  VEC: the
// rows begin on 16 bytes and k0, end are multiples of 4.  `lane` of the `lanes` threads that share the work.
template <bool VEC> __device__ __forceinline__ void stage_piece(float* dst, const float* base, size_t ld, int row, int rows, int k0, int end, int piece) {
    constexpr int W = VEC ? 4 : 1;
    const int k = k0 + piece * W;
    const bool take = row < rows && k < end;
    cp_async_zfill<W * 4>(dst + piece * W, take ? base + (size_t)row * ld + k : base, take);
}

__device__ __forceinline__ float fma4(const float4& a, const float4& b, float acc) {
    acc = fmaf(a.x, b.x, acc);
    acc = fmaf(a.y, b.y, acc);
    acc = fmaf(a.z, b.z, acc);
    return fmaf(a.w, b.w, acc);
}

__device__ __forceinline__ void f32_finish(float v, const float* bias, const float* residual, float* Y, int m, int n, int ldy, int act) {
    if (bias) v += bias[n];
    v = apply_act_rt(v, act);
    if (residual) v += residual[(size_t)m * ldy + n];
    Y[(size_t)m * ldy + n] = v;
}

// Up to R rows.  A CTA owns C columns; thread (part p, column c) runs the chain of its part for all rows.  W and x arrive
// through a ring of STAGES stages of KB numbers of every part (`cp.async`, coalesced along k); the first stages of W are
// asked for before the kernel ahead has ended.  A warp holds several columns of few parts, so that its reads of x are one
// wavefront each; R and C trade reads of x for CTAs.  N x K at 4 rows, weights from memory (one chain a thread before): 2,304 x 768
// 58 -> 4.1 us, 768 x 3,072 232 -> 7.3 us, 50,257 x 768 201 -> 33 us (4.7 TB/s); at 1 row the last is 25 us (6.2 TB/s); at 16 rows
// 59 -> 6.2, 235 -> 19 and 205 -> 63 us.
template <int R, int C> __host__ __device__ constexpr int rows_stage_floats() { return PARTS * C * KPITCH + PARTS * (R * KPITCH + 4); }

template <int R, int C, int STAGES, bool VEC>
__global__ void __launch_bounds__(C * PARTS)
gemm_f32_rows_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias, const float* residual,
                     float* Y, int M, int N, int K, int ldx, int ldy, int act) {
    extern __shared__ __align__(16) float ring[];
    constexpr int STAGE = rows_stage_floats<R, C>(), THREADS_R = C * PARTS, PIECES = VEC ? KB / 4 : KB;
    pdl_launch_dependents();
    const int tid = threadIdx.x, c = tid % C, p = tid / C, n0 = blockIdx.x * C;
    const int len = part_length(K), n_chunks = (min(len, K) + KB - 1) / KB;
    auto load_w = [&](int chunk) {
        float* at = ring + (chunk % STAGES) * STAGE;
        for (int i = tid; i < PARTS * C * PIECES; i += THREADS_R) {
            const int piece = i % PIECES, cc = i / PIECES % C, pp = i / (PIECES * C);
            stage_piece<VEC>(at + (pp * C + cc) * KPITCH, W, K, n0 + cc, N, pp * len + chunk * KB, min(K, (pp + 1) * len), piece);
        }
    };
    auto load_x = [&](int chunk) {
        float* at = ring + (chunk % STAGES) * STAGE + PARTS * C * KPITCH;
        for (int i = tid; i < PARTS * R * PIECES; i += THREADS_R) {
            const int piece = i % PIECES, r = i / PIECES % R, pp = i / (PIECES * R);
            stage_piece<VEC>(at + pp * (R * KPITCH + 4) + r * KPITCH, X, ldx, r, M, pp * len + chunk * KB, min(K, (pp + 1) * len), piece);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < n_chunks) load_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < n_chunks) load_x(s);
        cp_async_commit();
    }
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                   // the stage is here, and the one before it has been read by everyone
        if (chunk + STAGES - 1 < n_chunks) {
            load_w(chunk + STAGES - 1);
            load_x(chunk + STAGES - 1);
        }
        cp_async_commit();
        const float* at = ring + (chunk % STAGES) * STAGE;
        const float4* w4 = (const float4*)(at + (p * C + c) * KPITCH);
        const float4* x4 = (const float4*)(at + PARTS * C * KPITCH + p * (R * KPITCH + 4));
#pragma unroll
        for (int k = 0; k < KB / 4; ++k) {
            const float4 w = w4[k];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fma4(x4[r * (KPITCH / 4) + k], w, acc[r]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    float* sums = ring;                                    // [part][row][column]
#pragma unroll
    for (int r = 0; r < R; ++r) sums[(p * R + r) * C + c] = acc[r];
    __syncthreads();
    for (int i = tid; i < R * C; i += THREADS_R) {
        const int r = i / C, n = n0 + i % C;
        if (r >= M || n >= N) continue;
        float v = sums[i];
#pragma unroll
        for (int pp = 1; pp < PARTS; ++pp) v += sums[pp * R * C + i];
        f32_finish(v, bias, residual, Y, r, n, ldy, act);
    }
}

// Up to R rows with a LayerNorm ahead (vlrf_gemm_f32_norm_gains says where that pays) and, for a q/k/v projection, the write of its k and v columns into one layer's paged cache behind:
// the norm's kernel and the append's are launches of their own otherwise, 2.5 us each inside a decode step for rows that every CTA here
// has read and normed in 1.  The sums are those of gemm_f32_rows_kernel, the norm is that of embed_norm.cu (a warp a row, the row in
// registers), so the same bits come out.  The whole rows lie in shared memory, each part's run 16 bytes further than its place
// asks for, which keeps a warp's reads of several parts on banks of their own.
struct F32Scatter {
    float* Kc; float* Vc;                                  // [block][kv_head][BT][dh]; Kc == nullptr: none
    const int* block_table; const int* tok_slot; const int* tok_pos;
    int max_blocks, k_off, v_off, width, dh, Hkv, BT;      // width = Hkv·dh
};
constexpr int NORM_MAX_K = 1024, NORM_NV = NORM_MAX_K / 128, NORM_STAGES = 4;
template <int R, int C, int STAGES> __host__ __device__ constexpr size_t norm_smem(int K) {
    return ((size_t)STAGES * PARTS * C * KPITCH + (size_t)R * (K + 4 * PARTS) + 2 * (size_t)K) * 4;
}

template <int R, int C, int STAGES>
__global__ void __launch_bounds__(C * PARTS)
gemm_f32_norm_kernel(const float* __restrict__ X, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                     const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ Y, int M, int N, int K, int act,
                     F32Scatter kv, int* __restrict__ dev_err) {
    extern __shared__ __align__(16) float ring[];
    __shared__ int s_blk[R], s_row[R];                     // where each row's token lies in the cache
    constexpr int STAGE = PARTS * C * KPITCH, THREADS_R = C * PARTS, PIECES = KB / 4;
    pdl_launch_dependents();
    const int tid = threadIdx.x, c = tid % C, p = tid / C, n0 = blockIdx.x * C, warp = tid >> 5, lane = tid & 31;
    const int len = part_length(K), n_chunks = (min(len, K) + KB - 1) / KB, pitch = K + 4 * PARTS, nv = K >> 2;
    float* rows = ring + STAGES * STAGE;                   // [R][K + 4·PARTS]
    auto load_w = [&](int chunk) {
        float* at = ring + (chunk % STAGES) * STAGE;
        for (int i = tid; i < PARTS * C * PIECES; i += THREADS_R) {
            const int piece = i % PIECES, cc = i / PIECES % C, pp = i / (PIECES * C);
            stage_piece<true>(at + (pp * C + cc) * KPITCH, W, K, n0 + cc, N, pp * len + chunk * KB, min(K, (pp + 1) * len), piece);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < n_chunks) load_w(s);
        cp_async_commit();
    }
    float4* const gm = reinterpret_cast<float4*>(rows + R * pitch);      // the norm's weight and bias
    float4* const bt = gm + nv;
    for (int i = tid; i < nv; i += THREADS_R) {
        gm[i] = reinterpret_cast<const float4*>(gamma)[i];
        bt[i] = reinterpret_cast<const float4*>(beta)[i];
    }
    __syncthreads();
    pdl_wait();
    if (kv.Kc != nullptr && tid < R) {
        int blk = -1, row = 0;
        const int slot = tid < M ? kv.tok_slot[tid] : -1;
        if (slot >= 0) {
            const int pos = kv.tok_pos[tid], bi = pos / kv.BT;
            blk = pos >= 0 && bi < kv.max_blocks ? kv.block_table[(size_t)slot * kv.max_blocks + bi] : -1;
            row = pos % kv.BT;
            if (blk < 0 && blockIdx.x == 0) atomicOr(dev_err, VLRF_DEVERR_NO_BLOCK);
        }
        s_blk[tid] = blk;
        s_row[tid] = row;
    }
    constexpr int WARPS = THREADS_R / 32, RW = R / WARPS >= 2 ? 2 : 1;   // two of a warp's rows at a time
    for (int r = warp * RW; r < R; r += WARPS * RW) {
        float4 v[RW][NORM_NV];
        float mean[RW], inv[RW];
        const float* src[RW];
#pragma unroll
        for (int e = 0; e < RW; ++e) src[e] = X + (size_t)min(r + e, M - 1) * K;
        layernorm_rows<NORM_NV, RW>(src, nv, K, eps, lane, v, mean, inv);
#pragma unroll
        for (int j = 0; j < NORM_NV; ++j) {
            const int i = j * 32 + lane;
            if (i < nv) {
                const float4 g4 = gm[i], b4 = bt[i];
                const int at = 4 * i + 4 * (4 * i / len);
#pragma unroll
                for (int e = 0; e < RW; ++e) *reinterpret_cast<float4*>(rows + (size_t)(r + e) * pitch + at) = layernorm_apply(v[e][j], mean[e], inv[e], g4, b4);
            }
        }
    }
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                   // the stage (and the rows) are here, and the stage before it has been read by everyone
        if (chunk + STAGES - 1 < n_chunks) load_w(chunk + STAGES - 1);
        cp_async_commit();
        const float4* w4 = (const float4*)(ring + (chunk % STAGES) * STAGE + (p * C + c) * KPITCH);
        const int k0 = p * len + chunk * KB, k1 = min(K, (p + 1) * len);
        const float* x0 = rows + k0 + 4 * p;
#pragma unroll
        for (int k = 0; k < KB / 4; ++k) {
            if (k0 + 4 * k >= k1) break;                   // (the weights behind the part's end are zeros, the rows there another part's)
            const float4 w = w4[k];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fma4(*reinterpret_cast<const float4*>(x0 + (size_t)r * pitch + 4 * k), w, acc[r]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    float* sums = ring;                                    // [part][row][column]
#pragma unroll
    for (int r = 0; r < R; ++r) sums[(p * R + r) * C + c] = acc[r];
    __syncthreads();
    for (int i = tid; i < R * C; i += THREADS_R) {
        const int r = i / C, n = n0 + i % C;
        if (r >= M || n >= N) continue;
        float v = sums[i];
#pragma unroll
        for (int pp = 1; pp < PARTS; ++pp) v += sums[pp * R * C + i];
        if (bias) v += bias[n];
        v = apply_act_rt(v, act);
        Y[(size_t)r * N + n] = v;
        if (kv.Kc != nullptr && n >= kv.k_off && s_blk[r] >= 0) {
            const bool is_v = n >= kv.v_off;
            const int col = n - (is_v ? kv.v_off : kv.k_off);
            if (col < kv.width) (is_v ? kv.Vc : kv.Kc)[(((size_t)s_blk[r] * kv.Hkv + col / kv.dh) * kv.BT + s_row[r]) * kv.dh + col % kv.dh] = v;
        }
    }
}

// Many rows.  The PARTS CTAs of a cluster multiply one 64 x 64 tile, each over its part of K (128 threads, 8 x 4 elements a
// thread read four k at a time: 12 shared-memory wavefronts for 128 FMA instructions of a warp, so the FMAs bound it); then
// each adds the eight sums of 8 of the tile's rows out of its neighbours' shared memory, in the order of the parts.  N x K at 64, 240
// and 1,000 rows (tiles of 64 x 64 over all of K, 4 x 4 elements a thread, before): 768 x 3,072 242, 222, 324 -> 25, 51, 146 us;
// 2,304 x 768 62, 57, 149 -> 16, 34, 116 us; 50,257 x 768 230, 793, 3,053 -> 156, 609, 2,422 us (32 TFLOP/s).
constexpr int TILE = 64, TILE_STAGES = 3, TILE_THREADS = 128, TILE_STAGE = 2 * TILE * KPITCH, SUM_PITCH = TILE + 4;
constexpr int TILE_SMEM = TILE_STAGES * TILE_STAGE * 4;
static_assert(TILE * SUM_PITCH * 4 <= TILE_SMEM, "a tile of sums takes the ring's place");

template <bool VEC>
__global__ void __launch_bounds__(TILE_THREADS)
gemm_f32_tile_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias, const float* residual,
                     float* Y, int M, int N, int K, int ldx, int ldy, int act) {
    extern __shared__ __align__(16) float ring[];
    constexpr int PIECES = VEC ? KB / 4 : KB;
    pdl_launch_dependents();
    const int tid = threadIdx.x, part = blockIdx.x % PARTS;
    const int n0 = blockIdx.x / PARTS * TILE, m0 = blockIdx.y * TILE;
    // warps 2 (rows) x 2 (columns); a thread's rows are mg + 8 i, its columns ng + 16 j: a warp's reads then fall on
    // neighbouring rows, one bank group apart
    const int lane = tid & 31, warp = tid >> 5;
    const int mg = (warp >> 1) * 4 + (lane >> 3), ng = (warp & 1) * 8 + (lane & 7);
    const int len = part_length(K), first = part * len, end = min(K, first + len);
    const int n_chunks = max(0, (end - first + KB - 1) / KB);
    auto load = [&](int chunk, bool weights) {
        float* at = ring + (chunk % TILE_STAGES) * TILE_STAGE + (weights ? TILE * KPITCH : 0);
        for (int i = tid; i < TILE * PIECES; i += TILE_THREADS) {
            const int piece = i % PIECES, r = i / PIECES;
            if (weights) stage_piece<VEC>(at + r * KPITCH, W, K, n0 + r, N, first + chunk * KB, end, piece);
            else stage_piece<VEC>(at + r * KPITCH, X, ldx, m0 + r, M, first + chunk * KB, end, piece);
        }
    };
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s)
        if (s < n_chunks) load(s, true);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < n_chunks) load(s, false);
        cp_async_commit();
    }
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        cp_async_wait<TILE_STAGES - 2>();
        __syncthreads();
        if (chunk + TILE_STAGES - 1 < n_chunks) {
            load(chunk + TILE_STAGES - 1, true);
            load(chunk + TILE_STAGES - 1, false);
        }
        cp_async_commit();
        const float* at = ring + (chunk % TILE_STAGES) * TILE_STAGE;
        const float4* a4 = (const float4*)(at + mg * KPITCH);
        const float4* b4 = (const float4*)(at + TILE * KPITCH + ng * KPITCH);
#pragma unroll
        for (int k = 0; k < KB / 4; ++k) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = b4[j * 16 * (KPITCH / 4) + k];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 a = a4[i * 8 * (KPITCH / 4) + k];
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma4(a, b[j], acc[i][j]);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    float* sums = ring;                                    // [row][column] of this part
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[(mg + 8 * i) * SUM_PITCH + ng + 16 * j] = acc[i][j];
    cluster_sync_all();
    {
        const int r = part * (TILE / PARTS) + tid / 16, col = tid % 16 * 4;      // 8 rows of 16 pieces of 4: one a thread
        const uint32_t own = (uint32_t)__cvta_generic_to_shared(sums + r * SUM_PITCH + col);
        float4 v = ld_cluster_f32x4(own, 0);
#pragma unroll
        for (int pp = 1; pp < PARTS; ++pp) {
            const float4 u = ld_cluster_f32x4(own, pp);
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        const int m = m0 + r, n = n0 + col;
        if (m < M) {
            if (n < N) f32_finish(v.x, bias, residual, Y, m, n, ldy, act);
            if (n + 1 < N) f32_finish(v.y, bias, residual, Y, m, n + 1, ldy, act);
            if (n + 2 < N) f32_finish(v.z, bias, residual, Y, m, n + 2, ldy, act);
            if (n + 3 < N) f32_finish(v.w, bias, residual, Y, m, n + 3, ldy, act);
        }
    }
    cluster_sync_relaxed();                                // nobody leaves while a neighbour still reads its sums
}

template <int R, int C, int STAGES, bool VEC>
int launch_f32_rows(const float* X, const float* W, const float* bias, const float* residual, float* Y, int M, int N, int K, int ldx, int ldy,
                    int act, cudaStream_t stream) {
    constexpr size_t smem = (size_t)STAGES * rows_stage_floats<R, C>() * 4;
    static_assert(smem <= 227 * 1024 && STAGES * rows_stage_floats<R, C>() >= PARTS * R * C, "shared memory");
    auto kern = gemm_f32_rows_kernel<R, C, STAGES, VEC>;
    static DeviceMarks marks;
    const cudaError_t e = allow_shared_memory(marks, kern, smem);
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "gemm: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    launch_chained(kern, dim3((N + C - 1) / C), dim3(C * PARTS), smem, stream, X, W, bias, residual, Y, M, N, K, ldx, ldy, act);
    return vlrf_check_launch("gemm_f32_rows");
}

template <int R, int C>
int launch_f32_norm(const float* X, const float* gamma, const float* beta, float eps, const float* W, const float* bias, float* Y, int M, int N, int K,
                    int act, const F32Scatter& kv, int* dev_err, cudaStream_t stream) {
    constexpr int STAGES = NORM_STAGES;
    static_assert((size_t)STAGES * C * KPITCH >= (size_t)R * C, "the sums take the ring's place");
    const size_t smem = norm_smem<R, C, STAGES>(K);
    auto kern = gemm_f32_norm_kernel<R, C, STAGES>;
    static DeviceMarks marks;
    const cudaError_t e = allow_shared_memory(marks, kern, norm_smem<R, C, STAGES>(NORM_MAX_K));
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "gemm: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    launch_chained(kern, dim3((N + C - 1) / C), dim3(C * PARTS), smem, stream, X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err);
    return vlrf_check_launch("gemm_f32_norm");
}
template <int R>
int launch_f32_norm_for(const float* X, const float* gamma, const float* beta, float eps, const float* W, const float* bias, float* Y, int M, int N,
                        int K, int act, const F32Scatter& kv, int* dev_err, cudaStream_t stream) {
    if (N < 8 * vlrf_sm_count()) return launch_f32_norm<R, 4>(X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err, stream);
    return launch_f32_norm<R, 8>(X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err, stream);
}

// Columns a CTA: as few as leave every SM a CTA (4 where 8 would not), 32 where even those make two waves (a head over
// a vocabulary), so that x is read from L2 less often.
template <int R, bool VEC>
int launch_f32_rows_for(const float* X, const float* W, const float* bias, const float* residual, float* Y, int M, int N, int K, int ldx, int ldy,
                        int act, cudaStream_t stream) {
    constexpr int S = R <= 8 ? 5 : 4;
    const int sms = vlrf_sm_count();
    if (N < 8 * sms) return launch_f32_rows<R, 4, S, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    if (N < 2 * 32 * sms) return launch_f32_rows<R, 8, S, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    return launch_f32_rows<R, 32, 2, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
}

// Rows a thread: the next instantiation up.  Tiles from 17 rows on: at 16 the rows kernel wins at every shape above (6.2 against 15.5
// us at 64 rows of 2,304 x 768, which is what a tile costs at 17 rows too), and its registers hold 16 sums.
template <bool VEC>
int launch_f32(const float* X, const float* W, const float* bias, const float* residual, float* Y, int M, int N, int K, int ldx, int ldy, int act,
               cudaStream_t stream) {
    if (M == 1) return launch_f32_rows_for<1, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    if (M <= 4) return launch_f32_rows_for<4, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    if (M <= 8) return launch_f32_rows_for<8, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    if (M <= 16) return launch_f32_rows_for<16, VEC>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, stream);
    auto kern = gemm_f32_tile_kernel<VEC>;
    static DeviceMarks marks;
    const cudaError_t e = allow_shared_memory(marks, kern, TILE_SMEM);
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "gemm: %d bytes of shared memory: %s", TILE_SMEM, cudaGetErrorString(e));
    const dim3 grid((unsigned)((N + TILE - 1) / TILE * PARTS), (unsigned)((M + TILE - 1) / TILE));
    launch_chained_cluster(kern, grid, dim3(TILE_THREADS), TILE_SMEM, dim3(PARTS), stream, X, W, bias, residual, Y, M, N, K, ldx, ldy, act);
    return vlrf_check_launch("gemm_f32_tile");
}
}  // namespace

extern "C" int vlrf_gemm_simt(const void* X, const void* W, const float* bias, const float* residual,
                              void* Y, int M, int N, int K, int ldx, int ldy, int in_dtype, int out_dtype,
                              int act, cudaStream_t stream) {
    VLRF_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    VLRF_REQUIRE(ldx >= K && ldy >= N, "gemm: leading sizes ldx=%d ldy=%d are smaller than K=%d N=%d", ldx, ldy, K, N);
    VLRF_REQUIRE(act >= 0 && act <= VLRF_ACT_LAST_FUSED, "gemm: unknown activation %d", act);
    if (M == 0) return VLRF_OK;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    VLRF_REQUIRE(grid.y <= 65535, "gemm: M=%d needs more than 65535 row tiles", M);
#define LAUNCH(IT, OT)                                                                                  \
    gemm_simt_kernel<IT, OT><<<grid, THREADS, 0, stream>>>((const IT*)X, (const IT*)W, bias, residual, \
                                                           (OT*)Y, M, N, K, ldx, ldy, act)
    if (in_dtype == VLRF_F32 && out_dtype == VLRF_F32) {
        const bool vec = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)X | (uintptr_t)W) % 16 == 0;
        return vec ? launch_f32<true>((const float*)X, (const float*)W, bias, residual, (float*)Y, M, N, K, ldx, ldy, act, stream)
                   : launch_f32<false>((const float*)X, (const float*)W, bias, residual, (float*)Y, M, N, K, ldx, ldy, act, stream);
    }
    if (in_dtype == VLRF_BF16 && out_dtype == VLRF_F32) LAUNCH(__nv_bfloat16, float);
    else if (in_dtype == VLRF_BF16 && out_dtype == VLRF_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16);
    else return vlrf_fail(VLRF_ERR_INVALID_ARG, "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
#undef LAUNCH
    return vlrf_check_launch("gemm_simt");
}

// Whether the product with a LayerNorm ahead takes these rows: up to 8, as many columns as the norm keeps in registers.  (With rows for 16 a
// launch took 1.15 to 1.8 times what norm, product and append take one after the other: 9 rows of 768 x 2,304 11.8, 13.5 us, of 768 x 3,072 13.6, 24.4.
// With registers for 1,664 columns GPT-2's sizes were 3 to 10 % slower, and of those with 1,280 and 1,600 columns half gained, half lost.)
extern "C" int vlrf_gemm_f32_norm_takes(int M, int K) { return M >= 1 && M <= 8 && K >= 4 && K % 4 == 0 && K <= NORM_MAX_K ? 1 : 0; }

// Whether it also gains: where all its CTAs find room on the GPU at once, by their shared memory (the rows, the norm's weight and bias and the ring).  A
// CTA of a second round norms all rows again, behind what it could have hidden that behind.  Norm and product apart (with the append for q/k/v) against
// together, us: 1 row of 768 x 2,304 7.6, 5.7, of 1,024 x 4,096 7.1, 5.9; 4 rows of 768 x 3,072 7.3, 6.1, of 1,024 x 3,072 11.9, 7.9, of 1,024 x 4,096
// (512 CTAs, room for 444) 12.1, 12.2; 8 rows of 768 x 3,072 (384 CTAs, room for 444) 10.2, 8.8, of 1,024 x 3,072 (384, 296) 15.4, 19.0, of 1,024 x 4,096 13.0, 17.2.
extern "C" int vlrf_gemm_f32_norm_gains(int M, int N, int K, int sms) {
    if (!vlrf_gemm_f32_norm_takes(M, K)) return 0;
    const bool wide = N >= 8 * sms;                        // (as launch_f32_norm_for)
    const size_t smem = wide ? (M == 1 ? norm_smem<1, 8, NORM_STAGES>(K) : M <= 4 ? norm_smem<4, 8, NORM_STAGES>(K) : norm_smem<8, 8, NORM_STAGES>(K))
                             : (M == 1 ? norm_smem<1, 4, NORM_STAGES>(K) : M <= 4 ? norm_smem<4, 4, NORM_STAGES>(K) : norm_smem<8, 4, NORM_STAGES>(K));
    const int ctas = wide ? (N + 7) / 8 : (N + 3) / 4;
    return ctas <= (int)(228 * 1024 / (smem + 1024)) * sms ? 1 : 0;      // (an SM's 228 KiB; a CTA has 1 KiB beside what it asks for)
}

// Y = act(LayerNorm(X) · Wᵀ + bias) in float32, X [M][K], Y [M][N]; Kc != null: columns k_off … and v_off … also into the cache.
extern "C" int vlrf_gemm_f32_norm(const float* X, const float* gamma, const float* beta, float eps, const float* W, const float* bias, float* Y,
                                  int M, int N, int K, int act, float* Kc, float* Vc, const int* block_table, int max_blocks,
                                  const int* tok_slot, const int* tok_pos, int k_off, int v_off, int Hkv, int dh, int BT, int* dev_err,
                                  cudaStream_t stream) {
    VLRF_REQUIRE(vlrf_gemm_f32_norm_takes(M, K) && N > 0, "gemm_f32_norm: %d rows of %d columns are not taken", M, K);
    VLRF_REQUIRE((((uintptr_t)X | (uintptr_t)W | (uintptr_t)gamma | (uintptr_t)beta) & 15) == 0, "gemm_f32_norm: rows must begin on 16 bytes");
    VLRF_REQUIRE(act >= 0 && act <= VLRF_ACT_LAST_FUSED && dev_err != nullptr, "gemm_f32_norm: bad arguments");
    F32Scatter kv{};
    if (Kc != nullptr) {
        VLRF_REQUIRE(Vc && block_table && tok_slot && tok_pos && Hkv > 0 && dh > 0 && BT > 0 && max_blocks > 0 && k_off >= 0 && v_off >= k_off + Hkv * dh,
                     "gemm_f32_norm: incomplete cache scatter arguments");
        kv = F32Scatter{Kc, Vc, block_table, tok_slot, tok_pos, max_blocks, k_off, v_off, Hkv * dh, dh, Hkv, BT};
    }
    if (M == 1) return launch_f32_norm_for<1>(X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err, stream);
    if (M <= 4) return launch_f32_norm_for<4>(X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err, stream);
    return launch_f32_norm_for<8>(X, gamma, beta, eps, W, bias, Y, M, N, K, act, kv, dev_err, stream);
}
