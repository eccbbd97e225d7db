// Prompt-step attention on the tcgen05 tensor cores: ragged, causal, over the paged cache (bfloat16, head
// size 64).
//
// A CTA takes 128 consecutive new tokens of one sequence and one head, and walks the sequence's keys in
// blocks of 128 (two cache blocks) up to the diagonal (reference include/model/attention.hpp:233; visibility
// k ≤ past + q :253-260; scale :373-374; softmax :265-307).  Its ten warps have fixed jobs:
//   warp 8  producer: the query tile once, then key and value tiles in turn through a ring of four
//           shared-memory slots (tiled TMA loads, 128-byte swizzle, one load per 64-token cache block);
//   warp 9  issues the MMAs: S = Q·Kᵀ (128 × 128, four k steps) into tensor memory, and, once the
//           probabilities are there too, O += P·V (128 × 64, eight k steps; P is the operand in tensor memory, V is
//           read as it lies in the cache, head dimension contiguous, through an MN-major descriptor);
//   warps 0-7  softmax: a query row is one lane of tensor memory, and two threads, of warps q and q + 4, have a half of a block's
//           keys each; they exchange the row's maximum through shared memory.  A thread takes its 64 scores of a block into
//           registers at once, which frees S for the next block's scores, and writes P as bfloat16 into tensor memory.  Blocks on
//           the diagonal, and with a window all blocks, are masked: their scores are read a chunk at a time, twice, and chunks of 32 keys that
//           lie behind all of a warp's rows are left out (4,096 tokens of 16 heads with a window of 2,048 75 us, without one 64).
//           O stays in tensor memory until the CTA's last block; where a row's maximum grew, its O is read back, scaled and
//           written again once P is on its way.  (Scaling only where the maximum has grown by much would save that mostly, but
//           then the largest P is not 1, which bfloat16 holds exactly, and peaked rows lose: 1.42e-3 -> 1.54e-3 off 64 bits.)
// A thread a row (its 128 scores read twice, P through shared memory, O added up in registers) took 20.1 us for 2 x 1,024 tokens of 12 heads,
// 30.6 for 4 x 1,024 of 16, now 17.7 and 23.1; sixteen softmax warps an SM instead of eight keep the exponentials' unit and the issue slots busier.  (Waits
// with one answer for all lanes of a warp cost 1 % of that, 3 where 200 tokens stand behind 3,000: 34.6 -> 35.7 us.)
// A CTA's blocks are a chain (scores, softmax, output product, one after the other), so a step with few
// tiles is bound by its longest tile, not by the SMs' throughput.  The keys of a long tile can therefore be
// dealt to up to `n_parts` CTAs: each leaves its rows' maximum, sum and outputs in global scratch, and the
// one that finishes last (a counter per tile says which) merges all of them in a fixed order, so the result
// does not depend on which CTA that is.  Long tiles come first in the grid.
// Two CTAs fit an SM (82 KiB of shared memory, 256 columns of tensor memory each): while one waits for its
// MMAs the other computes exponentials.  Rows of the last cache block behind the sequence's end hold
// whatever was there before; their scores are masked by assignment and their rows of V are cleared before
// the MMA reads them (0 · NaN would not be 0).  Every wait is bounded; a CTA that gives up sets the device
// error word, waits (bounded) for its copies in flight, frees its tensor memory and leaves.
#include <type_traits>
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int FT_BQ = 128, FT_BK = 128, FT_DH = 64, FT_CB = 64;   // queries / keys per block, head size, tokens per cache block
constexpr int FT_THREADS = 320;
constexpr int FT_TILE = FT_BK * FT_DH * 2;                         // bytes of a K or V tile (and of the Q tile)
constexpr int FT_SLOTS = 4;
constexpr int FT_TMEM_COLS = 256;                                  // S: columns 0-127, O: 128-191, P (two bfloat16 a column): 192-255
constexpr int FT_MIN_PART = 2;                                     // key blocks a part holds at least (what the host plans with)
constexpr int FT_PART_BLOCKS = 3;                                  // key blocks a part holds at most, while the tile has parts left
constexpr int FT_MAX_PARTS = 8;
constexpr int FT_PART_FLOATS = FT_DH * FT_BQ + 2 * FT_BQ;          // a part's scratch: outputs [64][128], maxima, sums

// Shared-memory matrix descriptor of an MN-major tile [k][64 elements] whose rows are 128 bytes written by TMA
// with the 128-byte swizzle: the 64 elements of a row are the operand's N, rows are its K; groups of 8 rows
// are 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_mn128(const void* tile) {
    uint64_t d = 0;
    d |= (uint64_t)((tsm(tile) >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;                               // leading byte offset (one 64-wide chunk of N only): unused
    d |= (uint64_t)(1024 >> 4) << 32;                     // stride byte offset: 8 rows of K
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;                               // SWIZZLE_128B
    return d;
}
// D float32, A bfloat16 K-major, B bfloat16 MN-major
__host__ __device__ constexpr uint32_t umma_idesc_bf16_bmn(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// 2^x for x ≤ 0 or so, in one instruction (−inf gives 0; results below the normal range are flushed to 0)
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// D += A · B with A (bfloat16, two of a row's elements a column) in tensor memory
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}

// What a CTA whose work was called off, whichever role gave up, waits for (bounded): the copies requested, which land in its shared memory, and the
// MMAs issued, which read it.
__device__ __noinline__ void ft_drain(int warp, uint64_t* q_full, uint64_t* full, uint64_t* drained, int n_issued, int* s_never) {
    if (warp == 9) {
        if (elect_one()) umma_commit(drained);
        __syncwarp();
        tbar_wait_warp(drained, 0, s_never);
    } else if (warp == 8 && elect_one()) {
        tbar_wait_or_abort(q_full, 0, s_never);
        for (int t = max(0, n_issued - FT_SLOTS); t < n_issued; ++t)
            tbar_wait_or_abort(&full[t % FT_SLOTS], (uint32_t)((t / FT_SLOTS) & 1), s_never);
    }
    __syncthreads();
}

// LIMITED: waits give up after `limit` polls (tests of a CTA whose work is called off)
template <bool LIMITED>
__global__ void __launch_bounds__(FT_THREADS, 2)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, int q_off, const int* __restrict__ block_table,
                       int max_blocks, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                       const int* __restrict__ seq_pos0, __nv_bfloat16* __restrict__ out, int ld_out, int H, int Hkv,
                       float scale, int window, int n_parts, float* __restrict__ partials, int* __restrict__ counters,
                       int n_tiles, int listed, uint32_t limit, int* __restrict__ dev_err, long long* trace) {
    const uint32_t polls = LIMITED ? limit : TC_WAIT_LIMIT;
    extern __shared__ unsigned char ft_raw[];
    // (stations of the time stamps, kind 4: 0 the CTA begins, 1 the kernel ahead has finished, 6 the CTA is done)
    const int tcta = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    if (threadIdx.x == 0) VLRF_TRACE(trace, 4, tcta, 0);
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_tile = smem;                                    // [128][128 B]
    unsigned char* kv_tiles = smem + FT_TILE;                        // [FT_SLOTS][128][128 B]: K_0, V_0, K_1, V_1, … in turn
    float* s_part = reinterpret_cast<float*>(kv_tiles + FT_SLOTS * FT_TILE);      // [2][2][128]: the halves' maxima of a block (by its parity); sums at the end
    uint64_t* q_full = reinterpret_cast<uint64_t*>(s_part + 4 * FT_BQ);
    uint64_t* full = q_full + 1;                                     // [FT_SLOTS]
    uint64_t* empty = full + FT_SLOTS;                               // [FT_SLOTS]
    uint64_t* s_full = empty + FT_SLOTS;
    uint64_t* s_read = s_full + 1;                                   // the scores are in registers: S may be written again
    uint64_t* p_full = s_read + 1;
    uint64_t* o_full = p_full + 1;
    uint64_t* drained = o_full + 1;                                  // no MMA is under way (only where the work was called off)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    int* s_never = s_abort + 1;                                      // stays 0: for waits that nothing calls off
    int* s_last = s_never + 1;                                       // whether this CTA merges its tile's parts
    int* s_issued = s_last + 1;                                      // tiles requested: 2j is K of block j, 2j+1 its V

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // z is the slowest index of the order in which CTAs are started: first parts before second parts, so that the
    // CTAs without work (short tiles have fewer parts) come last, and within a part long tiles first.  n_tiles: of the longest sequence.
    // listed: y counts the tiles that exist, the last tiles of all sequences first, where a place for every tile that the longest sequence
    // has would leave most CTAs without work (a CTA that only sets itself up and leaves takes a place on an SM for some 3 us).
    int part = blockIdx.z / n_tiles, qt = n_tiles - 1 - blockIdx.z % n_tiles, seq = blockIdx.y;
    const int h = blockIdx.x;

    // set-up that reads nothing of the kernel ahead
    if (threadIdx.x == 0) {
        tbar_init(q_full, 1);
        for (int i = 0; i < FT_SLOTS; ++i) { tbar_init(&full[i], 1); tbar_init(&empty[i], 1); }
        tbar_init(s_full, 1);
        tbar_init(s_read, 8);
        tbar_init(p_full, 8);
        tbar_init(o_full, 1);
        tbar_init(drained, 1);
        *s_abort = 0;
        *s_never = 0;
        *s_last = 1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        if (lane == 0) { tma_prefetch_descriptor(&tmap_q); tma_prefetch_descriptor(&tmap_k); tma_prefetch_descriptor(&tmap_v); }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tsm(tmem_slot)), "r"((uint32_t)FT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    if (threadIdx.x == 0) VLRF_TRACE(trace, 4, tcta, 1);
    pdl_launch_dependents();
    int row0, row_end, slot, pos0;
    bool exists = true;
    if (listed > 0) {                                // (at most 32 sequences: a lane each, every warp for itself)
        part = blockIdx.z;
        const bool there = lane < listed;
        row0 = there ? seq_start[lane] : 0;
        row_end = there ? seq_start[lane + 1] : 0;
        slot = there ? seq_slot[lane] : -1;
        pos0 = there ? seq_pos0[lane] : 0;
        const int mine = slot >= 0 ? (row_end - row0 + FT_BQ - 1) / FT_BQ : 0;
        int left = blockIdx.y;
        seq = -1;
        for (qt = n_tiles - 1; qt >= 0; --qt) {
            const unsigned has = __ballot_sync(0xffffffffu, mine > qt);
            const int n = __popc(has);
            if (left < n) {
                seq = __ffs(__ballot_sync(0xffffffffu, mine > qt && __popc(has & ((1u << lane) - 1u)) == left)) - 1;
                break;
            }
            left -= n;
        }
        exists = seq >= 0;                           // (fewer tiles than places)
        seq = max(seq, 0);
        qt = max(qt, 0);
        row0 = __shfl_sync(0xffffffffu, row0, seq);
        row_end = __shfl_sync(0xffffffffu, row_end, seq);
        slot = __shfl_sync(0xffffffffu, slot, seq);
        pos0 = __shfl_sync(0xffffffffu, pos0, seq);
    } else {
        row0 = seq_start[seq];
        row_end = seq_start[seq + 1];
        slot = seq_slot[seq];
        pos0 = seq_pos0[seq];
    }
    const int n_new = row_end - row0;
    const int hk = h / (H / Hkv);
    const int q_first = pos0 + qt * FT_BQ;                           // absolute position of the tile's first query
    const int q_last = min(pos0 + n_new, q_first + FT_BQ) - 1;       // … and of its last
    const int kb_last = q_last / FT_BK;
    const int kb_first = (window > 0) ? max(0, q_first - window + 1) / FT_BK : 0;
    const int n_kb = kb_last - kb_first + 1;
    // the tile's key blocks are dealt to tile_parts CTAs; the others of its n_parts have nothing to do
    const int tile_parts = max(1, min(n_parts, (n_kb + FT_PART_BLOCKS - 1) / FT_PART_BLOCKS));
    const bool active = exists && qt * FT_BQ < n_new && slot >= 0 && part < tile_parts;     // uniform over the CTA
    const int my_first = kb_first + part * n_kb / tile_parts;
    const int my_n = active ? kb_first + (part + 1) * n_kb / tile_parts - my_first : 0;
    const int cb_last = q_last / FT_CB;                              // last cache block that holds a visible key
    const int* table = block_table + (size_t)max(slot, 0) * max_blocks;
    const int tile_id = (seq * H + h) * n_tiles + qt;

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_s = *tmem_slot, tmem_o = tmem_s + 128, tmem_p = tmem_s + 192;

    if (warp == 8) {
        if (my_n > 0 && elect_one()) {
            tbar_expect_tx(q_full, FT_TILE);
            tma_load_2d(q_tile, &tmap_q, q_off + h * FT_DH, row0 + qt * FT_BQ, q_full);
            int n_issued = 0;
            bool ok = true;
            for (int t = 0; t < 2 * my_n && ok; ++t) {
                const int sl = t % FT_SLOTS, use = t / FT_SLOTS;
                if (use >= 1 && !tbar_wait_or_abort(&empty[sl], (uint32_t)((use - 1) & 1), s_abort, polls)) { ok = false; break; }
                const int cb0 = (my_first + (t >> 1)) * 2;            // the block's two cache blocks
                const int n_cb = (cb0 + 1 <= cb_last) ? 2 : 1;
                int blk[2];
                for (int i = 0; i < n_cb; ++i) {
                    blk[i] = table[cb0 + i];
                    if (blk[i] < 0) { atomicOr(dev_err, VLRF_DEVERR_NO_BLOCK); ok = false; }
                }
                if (!ok) break;
                tbar_expect_tx(&full[sl], n_cb * (FT_TILE / 2));
                for (int i = 0; i < n_cb; ++i)
                    tma_load_2d(kv_tiles + (size_t)sl * FT_TILE + i * (FT_TILE / 2), (t & 1) ? &tmap_v : &tmap_k, 0,
                                (blk[i] * Hkv + hk) * FT_CB, &full[sl]);
                ++n_issued;
            }
            *s_issued = n_issued;
            if (!ok) atomicExch(s_abort, 1);
        }
    } else if (warp == 9) {
        if (my_n > 0) {                              // (the whole warp waits, with one answer, and elects a lane for every issue: 1 % less time here than a lane alone)
            constexpr uint32_t idesc_s = umma_idesc_bf16(FT_BQ, FT_BK);
            constexpr uint32_t idesc_o = umma_idesc_bf16_bmn(FT_BQ, FT_DH);
            bool ok = tbar_wait_warp(q_full, 0, s_abort, polls);
            const uint64_t dq = umma_desc_k128(q_tile), dk0 = umma_desc_k128(kv_tiles), dv0 = umma_desc_mn128(kv_tiles);
            // S_j = Q · K_jᵀ into tensor memory, four k steps
            auto issue_s = [&](int j) -> bool {
                const uint32_t tk = 2u * j, sl = tk % FT_SLOTS;
                if (!tbar_wait_warp(&full[sl], (tk / FT_SLOTS) & 1u, s_abort, polls)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint64_t dk = dk0 + (uint64_t)(sl * (FT_TILE >> 4));
#pragma unroll
                    for (int k = 0; k < FT_DH / 16; ++k) umma_bf16(tmem_s, dq + 2 * k, dk + 2 * k, idesc_s, k > 0 ? 1u : 0u);
                    umma_commit(s_full);
                    umma_commit(&empty[sl]);
                }
                __syncwarp();
                return true;
            };
            ok = ok && issue_s(0);
            for (int j = 0; j < my_n && ok; ++j) {
                // S_{j+1} as soon as the softmax warps hold S_j in registers, O += P_j · V_j once they have written P_j
                if (j + 1 < my_n && !(tbar_wait_warp(s_read, (uint32_t)(j & 1), s_abort, polls) && issue_s(j + 1))) { ok = false; break; }
                const uint32_t tv = 2u * j + 1, sl = tv % FT_SLOTS;
                if (!tbar_wait_warp(&full[sl], (tv / FT_SLOTS) & 1u, s_abort, polls)) { ok = false; break; }
                if (!tbar_wait_warp(p_full, (uint32_t)(j & 1), s_abort, polls)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint64_t dv = dv0 + (uint64_t)(sl * (FT_TILE >> 4));
#pragma unroll
                    for (int k = 0; k < FT_BK / 16; ++k)      // 16 keys a step: 8 columns of P, 16 rows of V
                        umma_bf16_ta(tmem_o, tmem_p + 8u * k, dv + (uint64_t)(k * 16 * 128 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                    umma_commit(o_full);
                    umma_commit(&empty[sl]);
                }
                __syncwarp();
            }
            if (!ok) atomicExch(s_abort, 1);
        }
    } else if (active) {
        // ---- softmax warps: a lane of tensor memory is a query row; warps q and q + 4 have a half of a block's keys each
        const int q = warp & 3, half = warp >> 2, r = q * 32 + lane;
        const int q_pos = q_first + r;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        const float sl2 = scale * 1.4426950408889634f;               // scores in units of log2(e)
        const unsigned win_eff = window > 0 ? (unsigned)window : 0x7fffffffu;   // key visible: 0 ≤ q_pos − key < win_eff
        float m_run = -INFINITY, l_run = 0.f;                        // the row's maximum; the sum of this half
        bool ok = true;
        // one block; MASKED: some key of it is hidden from some row
        auto block = [&](int j, auto masked_c) {
            constexpr bool MASKED = decltype(masked_c)::value;
            const int k0 = (my_first + j) * FT_BK + half * 64;        // the half's first key
            // chunks of 32 keys of which a row of this warp sees any (those behind lie above the diagonal)
            const int q_top = q_first + q * 32 + 31;
            const int n_live = MASKED ? (q_top < k0 ? 0 : min(2, ((q_top - k0) >> 5) + 1)) : 2;
            // (a warp that has given up goes on meeting its neighbour, who may not have)
            if (!ok || !tbar_wait_warp(s_full, (uint32_t)(j & 1), s_abort, polls)) {
                ok = false;
                asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
                return;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the row's maximum over this block (of the raw scores: the scale is positive).  Blocks without a mask keep the scores in
            // registers; a mask's blocks, one in a tile's row of them, read a chunk at a time, twice.
            const uint32_t s_at = tmem_s + lane_addr + (uint32_t)(half * 64);
            uint32_t sv[2][32];
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (!MASKED) {
                tmem_ld32(s_at, sv[0]);
                tmem_ld32(s_at + 32u, sv[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tbar_arrive(s_read);
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(sv[c][i]));
            } else {
#pragma unroll 1
                for (int c = 0; c < n_live; ++c) {
                    tmem_ld32(s_at + (uint32_t)(c * 32), sv[0]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const int d0 = q_pos - (k0 + c * 32);             // q_pos − key for i = 0
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], (unsigned)(d0 - i) < win_eff ? __uint_as_float(sv[0][i]) : -INFINITY);
                }
            }
            const float m_half = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            s_part[((j & 1) * 2 + half) * FT_BQ + r] = m_half;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
            const float m_new = fmaxf(m_run, fmaxf(m_half, s_part[((j & 1) * 2 + (half ^ 1)) * FT_BQ + r]) * sl2);
            const float corr = m_run == -INFINITY ? 1.f : fast_exp2(m_run - m_new);      // (from −inf on the row's sums are 0 so far)
            l_run *= corr;
            m_run = m_new;
            const float m_use = (m_run == -INFINITY) ? 0.f : m_run;   // a row that sees nothing yet: every p is 0
            if (j > 0) {                                              // O holds the blocks before, and P may be written again
                if (!tbar_wait_warp(o_full, (uint32_t)((j - 1) & 1), s_abort, polls)) { ok = false; return; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            // exponentials, their sum, P as bfloat16 into tensor memory
            float sm4[4] = {0.f, 0.f, 0.f, 0.f};
            auto chunk = [&](int c, const uint32_t (&x)[32]) {
                uint32_t pk[16];
                const int d0 = q_pos - (k0 + c * 32);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float p0 = fast_exp2(fmaf(__uint_as_float(x[i]), sl2, -m_use)), p1 = fast_exp2(fmaf(__uint_as_float(x[i + 1]), sl2, -m_use));
                    if (MASKED) {
                        p0 = (unsigned)(d0 - i) < win_eff ? p0 : 0.f;
                        p1 = (unsigned)(d0 - i - 1) < win_eff ? p1 : 0.f;
                    }
                    sm4[i & 3] += p0;
                    sm4[(i + 1) & 3] += p1;
                    pk[i >> 1] = pack2(p0, p1);
                }
                tmem_st16(tmem_p + lane_addr + (uint32_t)(half * 32 + c * 16), pk);
            };
            if (!MASKED) {
                chunk(0, sv[0]);
                chunk(1, sv[1]);
            } else {
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                    if (c < n_live) {
                        tmem_ld32(s_at + (uint32_t)(c * 32), sv[0]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        chunk(c, sv[0]);
                    } else {
                        uint32_t none[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) none[i] = 0u;
                        tmem_st16(tmem_p + lane_addr + (uint32_t)(half * 32 + c * 16), none);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tbar_arrive(s_read);
            }
            l_run += (sm4[0] + sm4[1]) + (sm4[2] + sm4[3]);
            if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {      // a row's maximum grew: its O (a half of the columns here) follows
                uint32_t ov[32];
                tmem_ld32(tmem_o + lane_addr + (uint32_t)half * 32u, ov);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
                tmem_st32(tmem_o + lane_addr + (uint32_t)half * 32u, ov);
            }
            // rows of V that this CTA did not load, or that lie behind the sequence's last token, hold whatever was there before: clear them
            const int there = min(pos0 + n_new - (my_first + j) * FT_BK, ((my_first + j) * 2 + 1 <= cb_last ? 2 : 1) * FT_CB);
            if (there < FT_BK) {
                const int tv = 2 * j + 1;
                if (!tbar_wait_warp(&full[tv % FT_SLOTS], (uint32_t)((tv / FT_SLOTS) & 1), s_abort, polls)) { ok = false; return; }
                unsigned char* vt = kv_tiles + (size_t)(tv % FT_SLOTS) * FT_TILE;
                const int first_row = max(there, 0);
                for (int idx = warp * 32 + lane; idx < (FT_BK - first_row) * 8; idx += 256)
                    *reinterpret_cast<uint4*>(vt + (first_row + (idx >> 3)) * 128 + ((idx & 7) << 4)) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads them
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tbar_arrive(p_full);
        };
        for (int j = 0; j < my_n; ++j) {
            if (window > 0 || (my_first + j) * FT_BK + FT_BK - 1 > q_first) block(j, std::true_type{});      // (uniform over the CTA)
            else block(j, std::false_type{});
        }
        // the row's result of this half's columns, and the sum of both halves of the keys
        constexpr int HD = FT_DH / 2;
        float o_acc[HD];
#pragma unroll
        for (int d = 0; d < HD; ++d) o_acc[d] = 0.f;
        if (my_n > 0) {
            if (ok && tbar_wait_warp(o_full, (uint32_t)((my_n - 1) & 1), s_abort, polls)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t ov[HD];
                tmem_ld32(tmem_o + lane_addr + (uint32_t)(half * HD), ov);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < HD; ++i) o_acc[i] = __uint_as_float(ov[i]);
            } else {
                ok = false;
                atomicExch(s_abort, 1);
            }
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");               // (also behind the last block's maxima)
        s_part[half * FT_BQ + r] = l_run;
        asm volatile("bar.sync 5, 256;" ::: "memory");
        l_run = s_part[r] + s_part[FT_BQ + r];
        bool writes_out = true;
        if (tile_parts > 1) {
            // leave this part's result in scratch ([d][row], so that a warp writes whole lines), then see
            // whether the tile's other parts are all there
            float* mine = partials + ((size_t)tile_id * n_parts + part) * FT_PART_FLOATS;
#pragma unroll
            for (int d = 0; d < HD; ++d) mine[(half * HD + d) * FT_BQ + r] = o_acc[d];
            if (half == 0) {
                mine[FT_DH * FT_BQ + r] = m_run;
                mine[FT_DH * FT_BQ + FT_BQ + r] = l_run;
            }
            __threadfence();
            asm volatile("bar.sync 5, 256;" ::: "memory");
            if (threadIdx.x == 0) {
                const int before = atomicAdd(&counters[tile_id], 1);
                *s_last = (before == tile_parts - 1) ? 1 : 0;
                if (before == tile_parts - 1) counters[tile_id] = 0;          // left as it was found
            }
            asm volatile("bar.sync 5, 256;" ::: "memory");
            writes_out = *s_last != 0;
            if (writes_out) {
                __threadfence();
                // every part in turn, this CTA's own included: the sum does not depend on who came last
                m_run = -INFINITY; l_run = 0.f;
#pragma unroll
                for (int d = 0; d < HD; ++d) o_acc[d] = 0.f;
                for (int p = 0; p < tile_parts; ++p) {
                    const float* theirs = partials + ((size_t)tile_id * n_parts + p) * FT_PART_FLOATS;
                    const float m_p = __ldcg(theirs + FT_DH * FT_BQ + r), l_p = __ldcg(theirs + FT_DH * FT_BQ + FT_BQ + r);
                    const float m_new = fmaxf(m_run, m_p);
                    const float a = (m_run == -INFINITY) ? 0.f : fast_exp2(m_run - m_new);
                    const float b = (m_p == -INFINITY) ? 0.f : fast_exp2(m_p - m_new);
                    l_run = fmaf(l_run, a, l_p * b);
                    m_run = m_new;
#pragma unroll
                    for (int d0 = 0; d0 < HD; d0 += 16) {
                        float v[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __ldcg(theirs + (half * HD + d0 + i) * FT_BQ + r);
#pragma unroll
                        for (int i = 0; i < 16; ++i) o_acc[d0 + i] = fmaf(o_acc[d0 + i], a, v[i] * b);
                    }
                }
            }
        }
        if (writes_out) {
            // the row as bfloat16 into shared memory (Q's tile: no MMA reads it any more), then each warp
            // writes 16 rows four at a time, so that a store instruction fills whole lines
            const float inv = (l_run > 0.f) ? 1.f / l_run : 0.f;
            unsigned char* stage = q_tile;                            // [128][128 B], 16-byte pieces swizzled by row
            if (ok) {
#pragma unroll
                for (int d = 0; d < HD; d += 8) {
                    uint4 pk;
                    pk.x = pack2(o_acc[d] * inv, o_acc[d + 1] * inv); pk.y = pack2(o_acc[d + 2] * inv, o_acc[d + 3] * inv);
                    pk.z = pack2(o_acc[d + 4] * inv, o_acc[d + 5] * inv); pk.w = pack2(o_acc[d + 6] * inv, o_acc[d + 7] * inv);
                    *reinterpret_cast<uint4*>(stage + r * 128 + (((half * HD + d) >> 3 ^ (r & 7)) << 4)) = pk;
                }
            }
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
            if (ok) {
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int rr = q * 32 + half * 16 + it * 4 + (lane >> 3), piece = lane & 7;
                    const int q_local = qt * FT_BQ + rr;
                    if (q_local < n_new) {
                        const uint4 pk = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((piece ^ (rr & 7)) << 4));
                        *reinterpret_cast<uint4*>(out + (size_t)(row0 + q_local) * ld_out + (size_t)h * FT_DH + piece * 8) = pk;
                    }
                }
            }
        }
    }
    // everyone meets here on every path; then the allocating warp gives the tensor memory back
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (*s_abort) ft_drain(warp, q_full, full, drained, *s_issued, s_never);
    if (warp == 8) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"((uint32_t)FT_TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0) VLRF_TRACE(trace, 4, tcta, 6);
    if (threadIdx.x == 0 && *s_abort) atomicOr(dev_err, VLRF_DEVERR_WAIT_TIMEOUT);
}
thread_local int g_polls = -1;
}  // namespace

// Whether the tcgen05 prompt attention takes these sizes (bfloat16 only): head size 64, cache blocks of 64
// tokens, rows of the output and of the fused q/k/v buffer on 16-byte boundaries.
extern "C" int vlrf_attn_prefill_tc_takes(int dh, int BT, int ld, int q_off, int ld_out) {
    return (dh == FT_DH && BT == FT_CB && ld % 8 == 0 && q_off % 8 == 0 && ld_out % 8 == 0) ? 1 : 0;
}

// Scratch of one part of a tile, in floats; the most parts a tile is dealt to; key blocks (of 128) a part holds
// at least; queries of a tile.
extern "C" int vlrf_attn_prefill_tc_part_floats() { return FT_PART_FLOATS; }
extern "C" int vlrf_attn_prefill_tc_max_parts() { return FT_MAX_PARTS; }
extern "C" int vlrf_attn_prefill_tc_min_part_blocks() { return FT_MIN_PART; }
extern "C" int vlrf_attn_prefill_tc_tile() { return FT_BQ; }

// Whether the tiles that exist are listed, instead of a place for each that the longest sequence has: where they alone take the two places of
// every SM, and as many CTAs without work again would come and go between them (five prompts of 1,013 to 31 tokens and three single tokens,
// 25 heads, 600 of 1,600 CTAs: 42.8 -> 33.1 us; that step of GPT-2 XL 9,610 -> 9,343).  With fewer tiles than places the kernels behind, which may
// begin once the last CTA has, begin while SMs idle and crowd onto those: whole prompt steps of GPT-2 with 216 of 660 and of 864 CTAs listed 818 ->
// 841 and 915 -> 946 us, GPT-2 medium 272 of 880 1,816 -> 1,878; with 300 of 560 (large) 3,950 -> 4,007, with 320 of 880 3,069 -> 3,000.
extern "C" int vlrf_attn_prefill_tc_lists(int n_tokens, int n_seqs, int max_new, int H, int n_parts, int sms) {
    if (n_seqs < 2 || n_seqs > 32 || max_new > 64 * FT_BQ) return 0;          // (a lane of a warp per sequence)
    const long long all = (long long)((max_new + FT_BQ - 1) / FT_BQ) * n_seqs, exist = (long long)n_tokens / FT_BQ + n_seqs;
    const long long each = (long long)H * n_parts, full = 2ll * sms;
    return exist * each >= full && (all - exist) * each >= full ? 1 : 0;
}

// How often a wait of the calling thread's next launches polls its barrier before it gives up (negative: as ever), but for those that follow on
// giving up.  For tests of a CTA whose work is called off.
extern "C" int vlrf_attn_prefill_tc_wait_polls(int polls) { g_polls = polls; return VLRF_OK; }

// n_parts > 1 wants `partials` ([sequences × heads × tiles × n_parts] × part_floats) and `counters`
// ([sequences × heads × tiles], zero; left zero).
extern "C" int vlrf_attn_prefill_tc(const void* qkv, int ld, int q_off, const void* Kc, const void* Vc, int n_blocks,
                                    const int* block_table, int max_blocks, const int* seq_slot, const int* seq_start,
                                    const int* seq_pos0, void* out, int ld_out, int n_tokens, int n_seqs, int max_new,
                                    int H, int Hkv, int dh, int BT, float scale, int window, int n_parts, float* partials,
                                    int* counters, int* dev_err, cudaStream_t stream) {
    VLRF_REQUIRE(vlrf_attn_prefill_tc_takes(dh, BT, ld, q_off, ld_out), "attn_prefill_tc: head size %d / block %d / row strides %d, %d are not taken", dh, BT, ld, ld_out);
    VLRF_REQUIRE(n_tokens > 0 && n_seqs > 0 && max_new > 0 && H > 0 && Hkv > 0 && H % Hkv == 0 && max_blocks > 0, "attn_prefill_tc: bad sizes");
    VLRF_REQUIRE(n_seqs <= 65535, "attn_prefill_tc: too many sequences for one launch");
    VLRF_REQUIRE(window >= 0 && dev_err != nullptr, "attn_prefill_tc: bad arguments");
    VLRF_REQUIRE(n_parts >= 1 && n_parts <= FT_MAX_PARTS && (n_parts == 1 || (partials != nullptr && counters != nullptr)),
                 "attn_prefill_tc: %d parts (1 to %d; more than one wants scratch)", n_parts, FT_MAX_PARTS);
    const long long kv_rows = (long long)n_blocks * Hkv * BT;
    CUtensorMap tq, tk, tv;
    int st = vlrf_make_tmap_bf16(qkv, n_tokens, ld, ld, FT_BQ, 64, &tq);
    if (st != VLRF_OK) return st;
    st = vlrf_make_tmap_bf16(Kc, kv_rows, dh, dh, FT_CB, 64, &tk);
    if (st != VLRF_OK) return st;
    st = vlrf_make_tmap_bf16(Vc, kv_rows, dh, dh, FT_CB, 64, &tv);
    if (st != VLRF_OK) return st;
    const size_t smem = 1024 + (size_t)(1 + FT_SLOTS) * FT_TILE + 4 * FT_BQ * 4 + 24 * 8;
    static DeviceMarks marks[2];
    auto kern = g_polls < 0 ? attn_prefill_tc_kernel<false> : attn_prefill_tc_kernel<true>;
    cudaError_t e = allow_shared_memory(marks[g_polls < 0 ? 0 : 1], kern, smem);
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "attn_prefill_tc: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    const long long tiles = (max_new + FT_BQ - 1) / FT_BQ;
    VLRF_REQUIRE(tiles * n_parts <= 65535, "attn_prefill_tc: %lld tiles of %d parts are too many for one launch", tiles, n_parts);
    const long long places = (long long)n_tokens / FT_BQ + n_seqs;      // the tiles that exist are at most so many
    const int listed = vlrf_attn_prefill_tc_lists(n_tokens, n_seqs, max_new, H, n_parts, vlrf_sm_count()) ? n_seqs : 0;
    dim3 grid(H, listed ? (unsigned)places : n_seqs, (unsigned)(listed ? n_parts : tiles * n_parts));
    e = launch_chained(kern, grid, dim3(FT_THREADS), smem, stream, tq, tk, tv, q_off, block_table, max_blocks, seq_slot, seq_start, seq_pos0,
                       (__nv_bfloat16*)out, ld_out, H, Hkv, scale, window, n_parts, partials, counters, (int)tiles, listed, (uint32_t)g_polls,
                       dev_err, vlrf_trace_buffer());
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "attn_prefill_tc: %s", cudaGetErrorString(e));
    return vlrf_check_launch("attn_prefill_tc");
}
