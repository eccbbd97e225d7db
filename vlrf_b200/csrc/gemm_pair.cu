// Y[M,N] = act(X[M,K] · W[N,K]^T + bias) (+ residual) for the many rows of a prompt step, by pairs of SMs: a cluster of two
// CTAs computes 256 columns of Y by `bn` rows as one tcgen05 product of `cta_group::2`.  bfloat16 operands, float32
// accumulation in tensor memory.
//
// W is the 256-row operand and the rows of X the other one, so the accumulator holds Yᵀ: a lane of tensor memory is a
// column of Y, CTA 0 has the first 128 of the tile's columns and CTA 1 the rest.  Each CTA brings its own 128 rows of W and
// half of the tile's rows of X (TMA, 128-byte swizzle); the tensor cores of both SMs read both halves.  A stage of the
// ring is therefore 16 KiB + 64·bn bytes a CTA where a CTA of its own that computes 128 × bn needs 16 KiB + 128·bn: the
// products of a prompt step were bound by what their stages pull through L2.  And a warp's store is 32 consecutive
// columns of a row, whole lines, where a lane that has a row touches a line a lane.
//
// Ten warps a CTA, as in gemm_tcgen05.cu: warp 8 requests the CTA's loads, warp 9 of CTA 0 issues the MMAs of both, warps 0-7
// are the epilogue (two share 32 lanes of the accumulator and take half of its columns, the tile's rows, each).
//   full[s]       in CTA 0: the bytes of both CTAs' loads of a stage (both request with this barrier)
//   empty[s]      in both: the MMAs have read the stage (one commit signals both)
//   acc_full[b]   in both: the accumulator is complete
//   acc_empty[b]  in CTA 0: the 16 epilogue warps of both have read it
// CTAs are persistent: a pair takes the tiles (pair number), + number of pairs, …; the rows that are left behind whole tiles
// make tiles of their own, as wide as they need, which come last.  Two accumulators alternate, so a tile's
// epilogue overlaps the next tile's MMAs.  Every wait is bounded; a wait that gives up, whichever role's, calls off the work of both CTAs and
// sets a bit of the device error word.  Both CTAs meet at the end on every path; where the work was called off, what either has
// requested and the MMAs issued are waited for then (bounded too), since they write, read and signal the shared memory of
// both, and both meet once more.  Only then is tensor memory given back.
//
// The product is the reference's linear(x, W) = x · Wᵀ (include/model/compute.hpp:64-68), its epilogues those of
// include/model/feedforward.hpp:54-76 and include/model/transformer_block.hpp:153,158, its scatter include/model/kv_cache.hpp:215-251.
#include <type_traits>
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int PR_BM = 128;               // rows of W a CTA
constexpr int PR_BK = 64;                // elements of K a stage: one 128-byte swizzle atom
constexpr int PR_THREADS = 320;
constexpr int PR_MAX_STAGES = 8;
constexpr int PR_A_BYTES = PR_BM * PR_BK * 2;
constexpr int PR_SMEM = 200 * 1024;      // for the ring

struct PrKvScatter {
    void* Kc; void* Vc;                  // [block][kv_head][BT][dh], bf16; Kc == nullptr: no scatter
    const int* block_table; const int* tok_slot; const int* tok_pos;
    int max_blocks, k_off, v_off, width, dh, Hkv, BT;   // width = Hkv*dh
};

// the address of `own` (in this CTA's shared memory) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t pr_map(uint32_t own, uint32_t rank) {
    uint32_t there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(own), "r"(rank));
    return there;
}
// a tiled load into this CTA's shared memory that counts on a barrier of either CTA of the pair
__device__ __forceinline__ void pr_load(uint32_t dst, const CUtensorMap* tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pr_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives at the barrier at this address in both CTAs once all MMAs issued so far are complete
__device__ __forceinline__ void pr_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(tsm(bar)), "h"((uint16_t)3) : "memory");
}
// takes bytes off what a barrier of this CTA still expects
__device__ __forceinline__ void pr_take_off(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(tsm(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pr_arrive_at(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// What a pair whose work was called off waits for (bounded): the MMAs issued, and the last use of each stage by either CTA.  A function of its own, which
// keeps the kernel's registers as they are without it (inlined, steps of 2,048 prompt tokens of GPT-2 took 885 us instead of 881).
__device__ __noinline__ void pr_drain(int warp, uint32_t rank, int pair, int n_pairs, int n_kb, int whole, int bn, int rest, int ka, int stages,
                                      uint64_t* full, uint64_t* drained, int* s_issued, int* s_never) {
    if (warp == 9) {
        if (rank == 0 && elect_one()) pr_commit(drained);           // arrives in both CTAs behind the MMAs issued so far
        __syncwarp();
        tbar_wait_warp(drained, 0, s_never);
    } else if (warp == 8 && rank == 0 && elect_one()) {
        // CTA 0 announces the bytes of both, so a use that only it has requested lacks the other's half, and one that only CTA 1 has
        // requested is not announced yet
        int theirs;
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(theirs) : "r"(pr_map(tsm(s_issued), 1)) : "memory");
        const int mine = *s_issued, most = max(mine, theirs);
        for (int t = max(0, most - stages); t < most; ++t) {
            const uint32_t half = ka * (PR_A_BYTES + (pair + t / n_kb * n_pairs < whole ? bn : rest) * PR_BK);
            if (t >= mine) tbar_expect_tx(&full[t % stages], half);
            else if (t >= theirs) pr_take_off(&full[t % stages], half);
            tbar_wait_or_abort(&full[t % stages], (uint32_t)((t / stages) & 1), s_never);
        }
    }
    __syncwarp();
    cluster_sync_all();
}

// LIMITED: waits give up after `limit` polls (tests of a pair whose work is called off; the limit as an argument costs the MMAs' lane a per cent)
template <typename OT, bool LIMITED>
__global__ void __launch_bounds__(PR_THREADS)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                 const __grid_constant__ CUtensorMap tmap_rest, const float* __restrict__ bias, const float* residual, OT* Y, int M,
                 int N, int K, int ldy, int act, int bn, int stages, int ka, uint32_t limit, PrKvScatter kv, int* __restrict__ dev_err, long long* trace) {
    extern __shared__ unsigned char pr_raw[];
    const uint32_t polls = LIMITED ? limit : TC_WAIT_LIMIT;
    __shared__ uint64_t bars[2 * PR_MAX_STAGES + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort, s_never, s_issued;                       // s_issued: stages that this CTA has requested, over all tiles
    if (threadIdx.x == 0) VLRF_TRACE(trace, 3, (int)blockIdx.x, 0);
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pr_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t b_bytes = (uint32_t)bn * PR_BK;                   // half of a whole tile's rows, 128 bytes each
    const uint32_t a_stage = ka * PR_A_BYTES, b_stage = ka * b_bytes;                      // a stage holds ka atoms of K
    unsigned char* a_tiles = smem;                                   // [stages][ka][128][128 B]
    unsigned char* b_tiles = smem + (size_t)stages * a_stage;        // [stages][ka][bn/2][128 B]
    uint64_t* full = bars;
    uint64_t* empty = bars + PR_MAX_STAGES;
    uint64_t* acc_full = bars + 2 * PR_MAX_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drained = acc_empty + 2;                               // in both: no MMA is under way (only where the work was called off)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_kb = (K + ka * PR_BK - 1) / (ka * PR_BK);           // stages of K (atoms behind K's end are read as zeros)
    // whole tiles of bn rows, a tile of W's rows with all of X's one after another; then those with the rows that are left
    const int whole_x = M / bn, rest = (M - whole_x * bn + 31) & ~31, tiles_w = (N + 2 * PR_BM - 1) / (2 * PR_BM);
    const int whole = whole_x * tiles_w, n_tiles = whole + (rest > 0 ? tiles_w : 0);
    auto place = [&](int tile, int& w_tile, int& row, int& rows) {
        if (tile < whole) { w_tile = tile / whole_x; row = (tile - w_tile * whole_x) * bn; rows = bn; }
        else { w_tile = tile - whole; row = whole_x * bn; rows = rest; }
    };
    const uint32_t acc_stride = bn <= 128 ? 128 : 256, tmem_cols = 2 * acc_stride;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { tbar_init(&full[s], 1); tbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { tbar_init(&acc_full[b], 1); tbar_init(&acc_empty[b], 16); }
        tbar_init(drained, 1);
        s_abort = 0;
        s_never = 0;
        s_issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (warp == 8 && lane == 0) { tma_prefetch_descriptor(&tmap_w); tma_prefetch_descriptor(&tmap_x); tma_prefetch_descriptor(&tmap_rest); }
    if (warp == 9) {                               // (while the other CTA arrives)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tsm(&tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // both CTAs' barriers exist before either's loads signal them
    const uint32_t full0 = pr_map(tsm(full), 0);
    auto call_off = [&]() {                        // both CTAs stop
        atomicExch(&s_abort, 1);
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(pr_map(tsm(&s_abort), rank ^ 1u)), "r"(1u) : "memory");
    };
    // the weights do not depend on the kernel ahead: the first tile's are requested before the wait
    const int early = pair < n_tiles ? min(stages, n_kb) : 0;
    if (warp == 8 && early > 0 && elect_one()) {
        int w_tile, row, rows;
        place(pair, w_tile, row, rows);
        const int w_row = w_tile * (2 * PR_BM) + (int)rank * PR_BM;
        for (int kb = 0; kb < early; ++kb) {
            if (rank == 0) tbar_expect_tx(&full[kb], 2u * ka * (PR_A_BYTES + rows * PR_BK));
            for (int a = 0; a < ka; ++a)
                pr_load(tsm(a_tiles + (size_t)kb * a_stage + a * PR_A_BYTES), &tmap_w, (kb * ka + a) * PR_BK, w_row, full0 + 8u * kb);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                               // (where tensor memory begins)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    pdl_launch_dependents();
    pdl_wait();                                    // X (and the residual) come from the kernel before
    if (threadIdx.x == 0) VLRF_TRACE(trace, 3, (int)blockIdx.x, 1);

    if (warp == 8) {
        if (elect_one()) {
            int s = 0, n_issued = 0;
            uint32_t use = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                int w_tile, row, rows;
                place(tile, w_tile, row, rows);
                const int w_row = w_tile * (2 * PR_BM) + (int)rank * PR_BM, x_row = row + (int)rank * (rows >> 1);
                const CUtensorMap* map_x = tile < whole ? &tmap_x : &tmap_rest;
                for (int kb = 0; kb < n_kb; ++kb) {
                    if (n_issued >= early) {
                        if (use >= 1 && !tbar_wait_or_abort(&empty[s], (use - 1) & 1, &s_abort, polls)) { ok = false; break; }
                        if (rank == 0) tbar_expect_tx(&full[s], 2u * ka * (PR_A_BYTES + rows * PR_BK));
                        for (int a = 0; a < ka; ++a)
                            pr_load(tsm(a_tiles + (size_t)s * a_stage + a * PR_A_BYTES), &tmap_w, (kb * ka + a) * PR_BK, w_row, full0 + 8u * s);
                    }
                    for (int a = 0; a < ka; ++a)
                        pr_load(tsm(b_tiles + (size_t)s * b_stage + a * b_bytes), map_x, (kb * ka + a) * PR_BK, x_row, full0 + 8u * s);
                    ++n_issued;
                    if (++s == stages) { s = 0; ++use; }
                }
            }
            s_issued = n_issued;
            if (!ok) call_off();
        }
    } else if (warp == 9) {
        if (rank == 0 && elect_one()) {
            const uint64_t da0 = umma_desc_k128(a_tiles), db0 = umma_desc_k128(b_tiles);
            uint32_t s = 0, phase = 0, tc = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
                const uint32_t b = tc & 1, use = tc >> 1;
                if (use >= 1 && !tbar_wait_or_abort(&acc_empty[b], (use - 1) & 1, &s_abort, polls)) { ok = false; break; }
                const uint32_t tmem_d = tmem_base + b * acc_stride, idesc = umma_idesc_bf16(2 * PR_BM, tile < whole ? bn : rest);
                for (int kb = 0; kb < n_kb; ++kb) {
                    if (!tbar_wait_or_abort(&full[s], phase, &s_abort, polls)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint64_t da = da0 + (uint64_t)(s * (a_stage >> 4)), db = db0 + (uint64_t)(s * (b_stage >> 4));
#pragma unroll
                    for (int k = 0; k < PR_BK / 16; ++k)          // 16 elements = 32 bytes = 2 descriptor units along K
                        pr_mma(tmem_d, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    if (ka == 2) {
                        da += PR_A_BYTES >> 4;
                        db += b_bytes >> 4;
#pragma unroll
                        for (int k = 0; k < PR_BK / 16; ++k) pr_mma(tmem_d, da + 2 * k, db + 2 * k, idesc, 1u);
                    }
                    pr_commit(&empty[s]);
                    if (kb + 1 == n_kb) pr_commit(&acc_full[b]);
                    if (++s == (uint32_t)stages) { s = 0; phase ^= 1; }
                }
            }
            if (!ok) call_off();
        }
    } else {
        // epilogue: warps q and q+4 share accumulator lanes 32q … 32q+31, 32 columns of Y, and take half of the rows each
        const int q = warp & 3, half = warp >> 2;
        const uint32_t acc_empty0 = pr_map(tsm(acc_empty), 0);
        uint32_t tc = 0;
        for (int tile = pair; tile < n_tiles; tile += n_pairs, ++tc) {
            const uint32_t b = tc & 1;
            int w_tile, r0, rows;                                     // r0: the tile's first row
            place(tile, w_tile, r0, rows);
            const int c_begin = half ? rows >> 5 : 0, c_end = half ? rows >> 4 : rows >> 5;      // in chunks of 16 rows of Y
            const int n = w_tile * (2 * PR_BM) + (int)rank * PR_BM + q * 32 + lane;              // this thread's column of Y
            const bool live = n < N;
            const float bv = (bias != nullptr && live) ? bias[n] : 0.f;
            // Chunks whose 16 rows and 32 columns all exist go without a branch a row (with one a chunk took 2,200 cycles, most of a product of
            // small K).  The residual of a chunk is asked for a chunk ahead, that of the first while the MMAs still run.
            const bool all_cols = n - lane + 32 <= N, pairs_ok = ldy % 2 == 0 && (reinterpret_cast<uintptr_t>(Y) & 3) == 0;
            float res[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) res[j] = 0.f;
            auto fetch = [&](int c) {
                if (residual == nullptr || c >= c_end) return;
                const float* from = residual + (size_t)(r0 + c * 16) * ldy + n;
                if (all_cols && r0 + c * 16 + 16 <= M) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) res[j] = from[(size_t)j * ldy];
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (live && r0 + c * 16 + j < M) res[j] = from[(size_t)j * ldy];
                }
            };
            fetch(c_begin);
            // where this thread's column lies in the cache: the pointer to its place in a block's first row
            __nv_bfloat16* to = nullptr;
            if (kv.Kc != nullptr && live && n >= kv.k_off) {
                const bool is_v = n >= kv.v_off;
                const int col = n - (is_v ? kv.v_off : kv.k_off);
                if (col < kv.width)
                    to = reinterpret_cast<__nv_bfloat16*>(is_v ? kv.Vc : kv.Kc) + (size_t)(col / kv.dh) * kv.BT * kv.dh + col % kv.dh;
            }
            const bool scatters = __any_sync(0xffffffffu, to != nullptr);
            if (!tbar_wait_warp(&acc_full[b], (tc >> 1) & 1, &s_abort, polls)) { if (lane == 0) call_off(); break; }
            if (threadIdx.x == 0) { if (tc == 0) VLRF_TRACE(trace, 3, (int)blockIdx.x, 2); VLRF_TRACE(trace, 3, (int)blockIdx.x, 3); }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + b * acc_stride + ((uint32_t)(q * 32) << 16);
            auto chunks = [&](auto act_c) {                           // the activation as a compile-time constant
                constexpr int ACT = decltype(act_c)::value;
                uint32_t r[16];
                auto ask = [&](int c) {                              // 16 rows of the accumulator, a chunk ahead
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                        : "r"(tmem_d + (uint32_t)(c * 16)));
                };
                if (c_begin < c_end) ask(c_begin);
#pragma unroll 1
                for (int c = c_begin; c < c_end; ++c) {
                    // the cache row of each of the chunk's tokens, a lane a token
                    int blk = -2, row = 0;
                    if (scatters && lane < 16 && r0 + c * 16 + lane < M) {
                        const int m = r0 + c * 16 + lane, slot = kv.tok_slot[m];
                        if (slot >= 0) {
                            const int pos = kv.tok_pos[m];
                            blk = kv.block_table[(size_t)slot * kv.max_blocks + pos / kv.BT];
                            row = pos % kv.BT;
                            if (blk < 0) atomicOr(dev_err, VLRF_DEVERR_NO_BLOCK);
                        }
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = apply_act_const<OT, ACT>(__uint_as_float(r[j]) + bv) + res[j];
                    if (c + 1 < c_end) ask(c + 1);
                    fetch(c + 1);
                    OT* y = Y + (size_t)(r0 + c * 16) * ldy + n;
                    if (all_cols && r0 + c * 16 + 16 <= M && (sizeof(OT) == 4 || pairs_ok)) {
                        if (sizeof(OT) == 4) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) ElemIO<OT>::store(y + (size_t)j * ldy, v[j]);
                        } else {
                            // two lanes exchange a number, then the even one has two columns of an even row, the other two of the next
                            uint32_t* at = reinterpret_cast<uint32_t*>(Y + (size_t)(r0 + c * 16 + (lane & 1)) * ldy + (n & ~1));
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? v[j] : v[j + 1], 1);
                                at[(size_t)j * (ldy >> 1)] = lane & 1 ? pack2(got, v[j + 1]) : pack2(v[j], got);
                            }
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (live && r0 + c * 16 + j < M) ElemIO<OT>::store(y + (size_t)j * ldy, v[j]);
                    }
                    if (scatters) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int bj = __shfl_sync(0xffffffffu, blk, j), rj = __shfl_sync(0xffffffffu, row, j);
                            if (to != nullptr && bj >= 0) to[((size_t)bj * kv.Hkv * kv.BT + rj) * kv.dh] = __float2bfloat16_rn(v[j]);
                        }
                    }
                }
            };
            if (act == VLRF_ACT_NONE) chunks(std::integral_constant<int, VLRF_ACT_NONE>{});
            else if (act == VLRF_ACT_GELU_TANH) chunks(std::integral_constant<int, VLRF_ACT_GELU_TANH>{});
            else if (act == VLRF_ACT_RELU2) chunks(std::integral_constant<int, VLRF_ACT_RELU2>{});
            else if (act == VLRF_ACT_SILU) chunks(std::integral_constant<int, VLRF_ACT_SILU>{});
            else chunks(std::integral_constant<int, VLRF_ACT_GELU_ERF>{});
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) pr_arrive_at(acc_empty0 + 8u * b);        // this warp has read its part of the accumulator
        }
    }
    if (threadIdx.x == 0) VLRF_TRACE(trace, 3, (int)blockIdx.x, 6);
    // both CTAs meet here on every path; then the allocating warps give the tensor memory back
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (s_abort)                                   // (the same in both CTAs: who calls off tells the other before they meet)
        pr_drain(warp, rank, pair, n_pairs, n_kb, whole, bn, rest, ka, stages, full, drained, &s_issued, &s_never);
    if (warp == 9)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    if (threadIdx.x == 0 && s_abort) atomicOr(dev_err, VLRF_DEVERR_WAIT_TIMEOUT);
}

thread_local int g_polls = -1;

template <typename OT, bool LIMITED>
int launch_pair_as(const void* X, const void* W, const float* bias, const float* residual, void* Y, int M, int N, int K, int ldx,
                int ldy, int act, int bn, const PrKvScatter& kv, int* dev_err, cudaStream_t stream) {
    CUtensorMap tw, tx, tr;
    int st = vlrf_make_tmap_bf16(W, N, K, K, PR_BM, PR_BK, &tw);
    if (st != VLRF_OK) return st;
    st = vlrf_make_tmap_bf16(X, M, K, ldx, bn / 2, PR_BK, &tx);
    if (st != VLRF_OK) return st;
    const int rest = (M % bn + 31) & ~31;
    tr = tx;
    if (rest > 0 && rest != bn) st = vlrf_make_tmap_bf16(X, M, K, ldx, rest / 2, PR_BK, &tr);
    if (st != VLRF_OK) return st;
    const int ka = bn <= 128 && K > PR_BK ? 2 : 1, stage = ka * (PR_A_BYTES + bn * PR_BK);
    const int stages = PR_SMEM / stage < PR_MAX_STAGES ? PR_SMEM / stage : PR_MAX_STAGES;
    const size_t smem = 1024 + (size_t)stages * stage;
    static DeviceMarks marks;
    auto kern = gemm_pair_kernel<OT, LIMITED>;
    cudaError_t e = allow_shared_memory(marks, kern, 1024 + PR_SMEM);
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "gemm_pair: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    const long long tiles = (long long)((M + bn - 1) / bn) * ((N + 2 * PR_BM - 1) / (2 * PR_BM));
    const int pairs = vlrf_sm_count() / 2;
    dim3 grid(2u * (unsigned)(tiles < pairs ? tiles : pairs));
    e = launch_chained_cluster(kern, grid, dim3(PR_THREADS), smem, dim3(2), stream, tw, tx, tr, bias, residual, (OT*)Y, M, N, K, ldy,
                               act, bn, stages, ka, (uint32_t)g_polls, kv, dev_err, vlrf_trace_buffer());
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "gemm_pair: %s", cudaGetErrorString(e));
    return vlrf_check_launch("gemm_pair");
}
template <typename OT>
int launch_pair(const void* X, const void* W, const float* bias, const float* residual, void* Y, int M, int N, int K, int ldx,
                int ldy, int act, int bn, const PrKvScatter& kv, int* dev_err, cudaStream_t stream) {
    return g_polls < 0 ? launch_pair_as<OT, false>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, bn, kv, dev_err, stream)
                       : launch_pair_as<OT, true>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, bn, kv, dev_err, stream);
}
}  // namespace

// Rows of a tile: those with which the pair that has most to do has least, a tile counting its rows and 96 more (what it costs to begin and
// end, and the tensor cores' least time for an MMA, which tiles below 128 rows do not fill).  float32 results of M x N x K, time by rows (us): 2,048 x 768
// x 768 96: 7.0, 128: 7.3, 64: 8.0; 2,048 x 3,072 x 768 192: 14.8, 128: 15.2, 256: 16.8; 2,050 x 1,600 x 6,400 224: 40.6, 256: 40.7, 192 (a second
// round for 3 tiles of 77): 67.9; 1,928 x 11,264 x 2,048 256: 81, 224: 85, 128: 88.
extern "C" int vlrf_gemm_pair_rows(int M, int N, int sms) {
    const int pairs = sms / 2 > 0 ? sms / 2 : 1;
    const long long tiles_w = ((long long)N + 2 * PR_BM - 1) / (2 * PR_BM);
    long long best = -1;
    int rows = 64;
    for (int bn = 256; bn >= 64; bn -= 32) {
        const long long whole = M / bn * tiles_w, left = (M % bn + 31) & ~31;
        // whole tiles first, tile t to pair t mod pairs; then a tile of the rows that are left for each of W's.  The first pair has no fewer than any
        // of either, and a whole tile costs no less than one of what is left: it has most to do.
        const long long mine = (whole + pairs - 1) / pairs, tiles = (whole + (left ? tiles_w : 0) + pairs - 1) / pairs;
        const long long most = mine * (bn + 96) + (tiles - mine) * (left + 96);
        if (best < 0 || most < best) { best = most; rows = bn; }
    }
    return rows;
}

// How often a wait of the calling thread's next launches polls its barrier before it gives up (negative: as ever), but for those that follow on
// giving up.  For tests of a pair whose work is called off.
extern "C" int vlrf_gemm_pair_wait_polls(int polls) { g_polls = polls; return VLRF_OK; }

// bn: rows of a tile (a multiple of 32 up to 256)
extern "C" int vlrf_gemm_pair(const void* X, const void* W, const float* bias, const float* residual, void* Y, int M, int N, int K,
                              int ldx, int ldy, int out_dtype, int act, int bn, void* Kc, void* Vc, const int* block_table,
                              int max_blocks, const int* tok_slot, const int* tok_pos, int k_off, int v_off, int Hkv, int dh, int BT,
                              int* dev_err, cudaStream_t stream) {
    VLRF_REQUIRE(M >= 1 && N >= 1 && K >= 8 && K % 8 == 0 && ldx % 8 == 0 && ldx >= K && ldy >= N, "gemm_pair: M=%d N=%d K=%d ldx=%d ldy=%d", M, N, K, ldx, ldy);
    VLRF_REQUIRE(bn >= 32 && bn <= 256 && bn % 32 == 0, "gemm_pair: no tiles of %d rows", bn);
    VLRF_REQUIRE(act >= 0 && (act <= VLRF_ACT_LAST_FUSED || act == VLRF_ACT_SILU) && dev_err != nullptr, "gemm_pair: bad arguments");
    VLRF_REQUIRE(out_dtype == VLRF_BF16 || out_dtype == VLRF_F32, "gemm_pair: unknown output dtype %d", out_dtype);
    PrKvScatter kv{};
    if (Kc != nullptr) {
        VLRF_REQUIRE(Vc && block_table && tok_slot && tok_pos && Hkv > 0 && dh > 0 && BT > 0 && max_blocks > 0,
                     "gemm_pair: incomplete cache scatter arguments");
        VLRF_REQUIRE(out_dtype == VLRF_BF16, "gemm_pair: the cache scatter writes bfloat16");
        kv = PrKvScatter{Kc, Vc, block_table, tok_slot, tok_pos, max_blocks, k_off, v_off, Hkv * dh, dh, Hkv, BT};
    }
    return out_dtype == VLRF_BF16 ? launch_pair<__nv_bfloat16>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, bn, kv, dev_err, stream)
                                  : launch_pair<float>(X, W, bias, residual, Y, M, N, K, ldx, ldy, act, bn, kv, dev_err, stream);
}
