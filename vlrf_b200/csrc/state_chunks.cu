// Recurrences with a matrix state per head and one decay per head and token, over prompts, 64 tokens at a time on the tensor cores
// (`mma.sync`) at the precision of float32.
//
// A head keeps a matrix S of K rows by V columns.  Token i brings q_i, k_i (K numbers, shared by the H / G heads of a group), v_i (V
// numbers), the logarithm f_i ≤ 0 of a decay and a gain.  With F_i = f_1 + … + f_i inside a chunk and S_c the state ahead of it,
//     o_i     = e^(F_i) S_cᵀ q_i + Σ_(j ≤ i) e^(F_i − F_j) gain_j (q_i · k_j) v_j,        S_(c+1) = e^(F_L) S_c + U_c,
//     U_c     = Σ_j e^(F_L − F_j) gain_j k_j v_jᵀ
// so three kernels do it, each with every chunk at the same time but for the short sum in the middle:
//   state_chunk_writes   U_c of every chunk
//   state_chunk_states   a thread per four numbers of a state walks its sequence's chunks: S_c takes U_c's place, the last one is kept
//   state_chunk_outputs  the products of o; the scores q · k of a chunk are formed once for all heads and columns that share them
//
// Kind STATE_SPACE (ssd.cu): q = C, k = B, v = x, f = −exp(a_log) dt, gain = dt = softplus(·); o gets D · x added.
//
// Token by token (ssd.cu) a prompt of 1,024 tokens is 1,024 dependent steps of about 330 cycles, in as many CTAs as there are heads
// and column blocks, whatever idles beside them.  In chunks the dependent steps are 16, and the arithmetic is products: 2 x 1,024 tokens, 32 heads of
// 64 x 64 in 4 groups, 137 -> 69 us, 32 heads of 128 x 128 in 8 groups 343 -> 283 us.  The outputs keep the tensor pipe busy for 25 % of
// their cycles (23 % at 128 x 128): with 8 or 16 warps an SM a scheduler issues in 0.27 (0.19) of its cycles, and a warp waits in turn for memory, fixed
// latencies, instructions, barriers and the tensor pipe, none of them much above a fifth; two chains of products beside each other changed nothing.
// Its error against 64 bits is 0.9e-7 where token by token's is 1.2e-7.
//
// Precision.  Everything that was float32 enters the products whole: each operand as the sum of three bfloat16 numbers (24 bits) and
// each product as the six partial ones that reach 2^-24 of it (fc_mma3), summed in float32.  Exponents are sums of
// logarithms of one sign, over 16 tokens at most and whole blocks of 16; where one is the difference of two such sums (inside a block)
// these are kept to 48 bits; no weight is above 1
// before its gain.  The 32-bit engine keeps to the FMA kernels.
//
// Range.  A product of a zero weight and an infinity is not zero, and an infinity has no three parts: a token's infinity would reach the
// tokens of its block that come before it.  So the writes look at every number that enters: where one of a head's in a tile of columns
// (its rows, step sizes, decays, the state it starts from) is not finite or beyond RC_LIMIT, below which no product of this file
// overflows, `wild` says so, the states leave that tile as it was, and a fourth kernel does it again, token by token.
//
// Layouts: q, k, v float32 rows of any stride (multiples of 4 numbers, on 16 bytes); scratch per chunk and head K·V float32, laid
// out as the state is, the chunks of sequence s beginning at seq_start[s] / 64 + s; aux a number per chunk and head; wild an int per
// chunk, head and tile of 64 columns.  Heads are independent: where the scratch that a caller has does not hold every head's states, the three
// kernels run over a range of groups at a time (a pass), one range after another in the same scratch.
#include "common.cuh"
#include "chunk_mma.cuh"

namespace {
constexpr int RC = 64;                 // tokens of a chunk
constexpr int RT = 64;                 // columns of V that a CTA works on at a time (an item: a head and such a tile)
constexpr int RX = RT + 8;             // … and their pitch in shared memory (16 bytes of padding keep ldmatrix off bank conflicts)
constexpr int R_THREADS = 256;
constexpr int R_ITEMS = 4;             // items a CTA works through with one set of q and k
// Rows and gains: weights stay below 2^28, scores of 128 products below 2^63, what 64 tokens write or read below 2^125.  States: read below
// 2^28 · 2^90 · 128.
constexpr float RC_LIMIT = 268435456.f, RC_STATE_LIMIT = 1.2379400392853803e27f;      // 2^28, 2^90

struct StateChunks {
    const float *q, *k, *v;
    int ldq, ldk, ldv;
    const float *s0, *dt_bias, *a_log, *skip;
    int ld_s0;
    float* scratch;
    float* aux;                        // F_L
    int* wild;
    float* state;
    int state_row;
    const int *seq_slot, *seq_start, *seq_pos0;
    float* y;
    int ldy, H, G, V;
    int least;                         // tokens of the runs that are taken here
    int g0, groups;                    // the groups of this pass; scratch and aux hold their heads only
    __host__ __device__ int per_group() const { return H / G; }
    __host__ __device__ int heads() const { return groups * per_group(); }
};

// What a head's tokens of a chunk weigh.  Lp + Lo: the log decays of a token's block of 16 up to and with it, in two floats, for the
// differences of two of them; Ls: those of its block
// behind it; before, after: of the blocks ahead of and behind a block; block: of a whole block.
struct HeadScalars {
    float Lp[RC], Lo[RC], Ls[RC], gain[RC], before[4], after[4], block[4];
};

// A warp: the numbers of head h for the L tokens from `first` on (tokens 2·lane and 2·lane + 1 a lane).  Returns whether they are what the
// products take.
__device__ __forceinline__ bool head_scalars(const StateChunks& A, int h, int first, int L, int lane, HeadScalars& out) {
    const float a = -expf(A.a_log[h]), bias = A.dt_bias[h];
    float f[2], gain[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        const float raw = t < L ? A.s0[(size_t)(first + t) * A.ld_s0 + h] : 0.f;
        gain[e] = t < L ? softplus_f(raw + bias) : 0.f;
        f[e] = a * gain[e];
    }
    const int in_block = lane & 7;
    double up = (double)f[0] + f[1];
    float down = f[0] + f[1];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, up, o, 8);
        const float d = __shfl_down_sync(0xffffffffu, down, o, 8);
        if (in_block >= o) up += u;
        if (in_block + o < 8) down += d;
    }
    double ahead = __shfl_up_sync(0xffffffffu, up, 1, 8);
    float behind = __shfl_down_sync(0xffffffffu, down, 1, 8);
    if (in_block == 0) ahead = 0.0;
    if (in_block == 7) behind = 0.f;
    ahead += f[0];
    out.Lp[2 * lane] = (float)ahead;
    out.Lo[2 * lane] = (float)(ahead - (float)ahead);
    out.Lp[2 * lane + 1] = (float)up;
    out.Lo[2 * lane + 1] = (float)(up - (float)up);
    out.Ls[2 * lane] = behind + f[1];
    out.Ls[2 * lane + 1] = behind;
    out.gain[2 * lane] = gain[0];
    out.gain[2 * lane + 1] = gain[1];
    const float whole = (float)up, t0 = __shfl_sync(0xffffffffu, whole, 7), t1 = __shfl_sync(0xffffffffu, whole, 15),
                t2 = __shfl_sync(0xffffffffu, whole, 23), t3 = __shfl_sync(0xffffffffu, whole, 31);
    if (lane == 0) {
        out.before[0] = 0.f; out.before[1] = t0; out.before[2] = t0 + t1; out.before[3] = t0 + t1 + t2;
        out.block[0] = t0; out.block[1] = t1; out.block[2] = t2; out.block[3] = t3;
        out.after[3] = 0.f; out.after[2] = t3; out.after[1] = t3 + t2; out.after[0] = t3 + t2 + t1;
    }
    // (written so that a NaN fails; a sum of logarithms of one sign is finite only if each of them is)
    return __all_sync(0xffffffffu, gain[0] < RC_LIMIT && gain[1] < RC_LIMIT) && t0 + t1 + t2 + t3 > -3e38f;
}
__device__ __forceinline__ bool tame(const float4& x, float limit) {
    return (fabsf(x.x) < limit) & (fabsf(x.y) < limit) & (fabsf(x.z) < limit) & (fabsf(x.w) < limit);
}

// Four numbers into the three planes of a tile, `plane` elements apart.
__device__ __forceinline__ void store_planes(__nv_bfloat16* at, int plane, const float4& x) {
    uint32_t h[2], m[2], l[2];
    fc_split3(x.x, x.y, h[0], m[0], l[0]);
    fc_split3(x.z, x.w, h[1], m[1], l[1]);
    *reinterpret_cast<uint2*>(at) = make_uint2(h[0], h[1]);
    *reinterpret_cast<uint2*>(at + plane) = make_uint2(m[0], m[1]);
    *reinterpret_cast<uint2*>(at + 2 * plane) = make_uint2(l[0], l[1]);
}
__device__ __forceinline__ float4 quad_or_zero(const float* p, bool there) { return there ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f); }

// The K numbers of the chunk's tokens (rows of stride ld) into planes [3][RC][K + 8].  Returns whether this thread's are what the products take.
template <int K>
__device__ __forceinline__ bool load_rows(__nv_bfloat16* planes, const float* rows, int ld, int L, int tid) {
    constexpr int QUADS = RC * K / 4, EACH = (QUADS + R_THREADS - 1) / R_THREADS;
    float4 x[EACH];
#pragma unroll
    for (int e = 0; e < EACH; ++e) {
        const int i = tid + e * R_THREADS, r = i / (K / 4), c = (i - r * (K / 4)) * 4;
        x[e] = quad_or_zero(rows + (size_t)r * ld + c, i < QUADS && r < L);
    }
#pragma unroll
    for (int e = 0; e < EACH; ++e) {
        const int i = tid + e * R_THREADS, r = i / (K / 4), c = (i - r * (K / 4)) * 4;
        if (i < QUADS) store_planes(planes + r * (K + 8) + c, RC * (K + 8), x[e]);
    }
    bool fine = true;
#pragma unroll
    for (int e = 0; e < EACH; ++e) fine &= tame(x[e], RC_LIMIT);
    return fine;
}

template <int K> constexpr int writes_smem() { return (3 * RC * (K + 8) + 3 * RC * RX) * 2 + R_ITEMS * (int)sizeof(HeadScalars) + R_ITEMS * RC * 4; }

// grid (chunks of the longest run, groups · parts of a group's items, sequences)
template <int K>
__global__ void __launch_bounds__(R_THREADS)
state_chunk_writes_kernel(const StateChunks A, int v_tiles, int parts) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char rc_raw[];
    constexpr int KS = K + 8;
    __nv_bfloat16* ks = reinterpret_cast<__nv_bfloat16*>(rc_raw);        // [3][64][KS]
    __nv_bfloat16* xs = ks + 3 * RC * KS;                                // [3][64][RX]
    HeadScalars* sc = reinterpret_cast<HeadScalars*>(xs + 3 * RC * RX);
    float* weight = reinterpret_cast<float*>(sc + R_ITEMS);              // [items][64]
    __shared__ bool item_fine[R_ITEMS];
    const int s = blockIdx.z, c0 = blockIdx.x * RC;
    const int start = A.seq_start[s], n = A.seq_start[s + 1] - start;
    if (c0 >= n || n < A.least || A.seq_slot[s] < 0) return;
    const int L = min(RC, n - c0), first = start + c0;
    const int part = blockIdx.y % parts, g = A.g0 + blockIdx.y / parts, per_group = A.per_group(), i0 = part * R_ITEMS, items = min(R_ITEMS, per_group * v_tiles - i0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, heads = A.heads(), h_first = A.g0 * per_group;
    const size_t chunk = (size_t)(start / RC + s + blockIdx.x);
    float4 x[4];                                                         // the next item's values, a quarter of a token's tile a thread
    auto ask = [&](int item) {
        const int h = g * per_group + (i0 + item) / v_tiles, v0 = (i0 + item) % v_tiles * RT;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = tid / 16 + 16 * e, c = tid % 16 * 4;
            x[e] = quad_or_zero(A.v + (size_t)(first + r) * A.ldv + (size_t)h * A.V + v0 + c, r < L && v0 + c < A.V);
        }
    };
    ask(0);
    // the queries enter here only to be looked at (the outputs load them again); no `&&`, which would ask for one behind the other
    bool rows_fine = true;
#pragma unroll
    for (int e = 0; e < RC * K / 4 / R_THREADS; ++e) {
        const int i = tid + e * R_THREADS, r = i / (K / 4), c = (i - r * (K / 4)) * 4;
        rows_fine &= tame(quad_or_zero(A.q + (size_t)(first + r) * A.ldq + (size_t)g * K + c, r < L), RC_LIMIT);
    }
    if (warp < items) {
        const int h = g * per_group + (i0 + warp) / v_tiles;
        const bool fine = head_scalars(A, h, first, L, lane, sc[warp]);
        if (lane == 0) item_fine[warp] = fine;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = lane + 32 * e;
            weight[warp * RC + t] = expf(sc[warp].Ls[t] + sc[warp].after[t >> 4]) * sc[warp].gain[t];
        }
        if (lane == 0 && (i0 + warp) % v_tiles == 0) A.aux[chunk * heads + h - h_first] = sc[warp].before[3] + sc[warp].Lp[RC - 1];
    }
    rows_fine &= load_rows<K>(ks, A.k + (size_t)first * A.ldk + (size_t)g * K, A.ldk, L, tid);
    rows_fine = __syncthreads_and(rows_fine);
    const float* from = A.state + ((size_t)A.seq_slot[s] * 2 + (A.seq_pos0[s] & 1)) * A.state_row;
    const int chunks = (n + RC - 1) / RC;
    for (int item = 0; item < items; ++item) {
        const int h = g * per_group + (i0 + item) / v_tiles, v0 = (i0 + item) % v_tiles * RT;
        bool fine = rows_fine && item_fine[item];
        // the state that the sequence starts from: its chunks look at a share each
        for (int i = blockIdx.x * R_THREADS + tid; i < K * RT / 4; i += chunks * R_THREADS) {
            const int r = i / (RT / 4), c = v0 + i % (RT / 4) * 4;
            fine &= tame(quad_or_zero(from + ((size_t)h * K + r) * A.V + c, c < A.V), RC_STATE_LIMIT);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = tid / 16 + 16 * e, c = tid % 16 * 4;
            const float w = weight[item * RC + r];
            fine &= tame(x[e], RC_LIMIT);
            store_planes(xs + r * RX + c, RC * RX, make_float4(w * x[e].x, w * x[e].y, w * x[e].z, w * x[e].w));
        }
        if (item + 1 < items) ask(item + 1);
        fine = __syncthreads_and(fine);
        if (tid == 0) A.wild[(chunk * A.H + h) * v_tiles + v0 / RT] = fine ? 0 : 1;
        // 16 rows of the state by 32 columns at a time
        float* U = A.scratch + (chunk * heads + h - h_first) * (size_t)K * A.V;
        for (int unit = warp; unit < K / 8; unit += R_THREADS / 32) {
            const int r0 = (unit >> 1) * 16, cc = (unit & 1) * 32;
            float acc[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll
            for (int kk = 0; kk < RC / 16; ++kk) {
                uint32_t a[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    fc_ldsm_t(a[p], fc_sm(ks + p * RC * KS + (kk * 16 + (lane & 7) + 8 * (lane >> 4)) * KS + r0 + 8 * ((lane >> 3) & 1)));
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    uint32_t b[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        fc_ldsm_t(b[p], fc_sm(xs + p * RC * RX + (kk * 16 + (lane & 15)) * RX + cc + (j + (lane >> 4)) * 8));
                    fc_mma3(acc[j], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
                    fc_mma3(acc[j + 1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = r0 + (lane >> 2) + 8 * r, col = v0 + cc + j * 8 + 2 * (lane & 3);
                    if (col < A.V) *reinterpret_cast<float2*>(U + (size_t)row * A.V + col) = make_float2(acc[j][2 * r], acc[j][2 * r + 1]);
                }
        }
        __syncthreads();
    }
}

// grid (quads of a sequence's states / 128, sequences)
__global__ void __launch_bounds__(128)
state_chunk_states_kernel(const StateChunks A, int per_head, int v_tiles) {
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.y, slot = A.seq_slot[s];
    if (slot < 0) return;
    const int start = A.seq_start[s], n = A.seq_start[s + 1] - start, pos0 = A.seq_pos0[s];
    const int heads = A.heads(), h_first = A.g0 * A.per_group();
    const size_t all = (size_t)per_head * heads, i = 4 * ((size_t)blockIdx.x * 128 + threadIdx.x);
    if (i >= all || n < A.least) return;
    const float* from = A.state + ((size_t)slot * 2 + (pos0 & 1)) * A.state_row + (size_t)h_first * per_head;
    float* to = A.state + ((size_t)slot * 2 + ((pos0 + n) & 1)) * A.state_row + (size_t)h_first * per_head;
    const int chunks = (n + RC - 1) / RC, hl = (int)(i / per_head);
    float4 S = *reinterpret_cast<const float4*>(from + i);
    const size_t slot0 = (size_t)(start / RC + s);
    float* u = A.scratch + slot0 * all + i;
    const float* aux = A.aux + slot0 * heads + hl;
    const int* wild = A.wild + (slot0 * A.H + h_first + hl) * v_tiles + (int)(i % A.V) / RT;
    int any_wild = 0;
    constexpr int AHEAD = 8;                        // chunks asked for together
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 U[AHEAD];
        float F[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            U[j] = quad_or_zero(u + (size_t)(c0 + j) * all, c0 + j < chunks);
            F[j] = c0 + j < chunks ? aux[(size_t)(c0 + j) * heads] : 0.f;
            any_wild |= c0 + j < chunks ? wild[(size_t)(c0 + j) * A.H * v_tiles] : 0;
        }
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            if (c0 + j < chunks) {
                *reinterpret_cast<float4*>(u + (size_t)(c0 + j) * all) = S;
                const float f = expf(F[j]);
                S.x = fmaf(f, S.x, U[j].x); S.y = fmaf(f, S.y, U[j].y); S.z = fmaf(f, S.z, U[j].z); S.w = fmaf(f, S.w, U[j].w);
            }
        }
    }
    if (!any_wild) *reinterpret_cast<float4*>(to + i) = S;      // (else it stays what token by token begins with: `to` may be `from`)
}

template <int K> constexpr int keys_or_state() { return 3 * (RC * (K + 8) > K * RX ? RC * (K + 8) : K * RX); }
template <int K> constexpr int outputs_smem() {
    return (3 * RC * (K + 8) + keys_or_state<K>() + 3 * RC * RX) * 2 + R_ITEMS * (int)sizeof(HeadScalars) + R_THREADS / 32 * RC * 4;
}

// grid as for the writes.  Warp w takes rows 16 (w / 2) … + 15 of the chunk and columns 32 (w mod 2) … + 31 of a tile; the scores of
// its rows stay in its registers for all items.
template <int K>
__global__ void __launch_bounds__(R_THREADS, K <= 64 ? 2 : 1)
state_chunk_outputs_kernel(const StateChunks A, int v_tiles, int parts) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char rc_raw[];
    constexpr int KS = K + 8, QS = K * RT / 4, SE = (QS + R_THREADS - 1) / R_THREADS;
    __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(rc_raw);        // [3][64][KS]
    __nv_bfloat16* ks = qs + 3 * RC * KS;                                // [3][64][KS], then the state's tile [3][K][RX]
    __nv_bfloat16* ss = ks;
    __nv_bfloat16* xs = ks + keys_or_state<K>();                         // [3][64][RX]
    HeadScalars* sc = reinterpret_cast<HeadScalars*>(xs + 3 * RC * RX);
    float* col_all = reinterpret_cast<float*>(sc + R_ITEMS);             // [warps][64]
    const int s = blockIdx.z, c0 = blockIdx.x * RC;
    const int start = A.seq_start[s], n = A.seq_start[s + 1] - start;
    if (c0 >= n || n < A.least || A.seq_slot[s] < 0) return;
    const int L = min(RC, n - c0), first = start + c0;
    const int part = blockIdx.y % parts, grp = A.g0 + blockIdx.y / parts, per_group = A.per_group(), i0 = part * R_ITEMS,
              items = min(R_ITEMS, per_group * v_tiles - i0);
    const int heads = A.heads(), h_first = A.g0 * per_group;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rb = warp >> 1, cc = (warp & 1) * 32, row0 = rb * 16;
    const size_t chunk = (size_t)(start / RC + s + blockIdx.x);
    float* colf = col_all + warp * RC;
    float4 x[4], S[SE];
    auto ask = [&](int item) {
        const int h = grp * per_group + (i0 + item) / v_tiles, v0 = (i0 + item) % v_tiles * RT;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = tid / 16 + 16 * e, c = tid % 16 * 4;
            x[e] = quad_or_zero(A.v + (size_t)(first + r) * A.ldv + (size_t)h * A.V + v0 + c, r < L && v0 + c < A.V);
        }
        const float* from = A.scratch + (chunk * heads + h - h_first) * (size_t)K * A.V + v0;
#pragma unroll
        for (int e = 0; e < SE; ++e) {
            const int i = tid + e * R_THREADS, r = i / 16, c = i % 16 * 4;
            S[e] = quad_or_zero(from + (size_t)r * A.V + c, i < QS && v0 + c < A.V);
        }
    };
    if (warp < items) head_scalars(A, grp * per_group + (i0 + warp) / v_tiles, first, L, lane, sc[warp]);
    load_rows<K>(qs, A.q + (size_t)first * A.ldq + (size_t)grp * K, A.ldq, L, tid);
    load_rows<K>(ks, A.k + (size_t)first * A.ldk + (size_t)grp * K, A.ldk, L, tid);
    ask(0);
    __syncthreads();
    float score[8][4];                              // rows row0 …, keys 8 j …: those up to the rows' own block
#pragma unroll
    for (int j = 0; j < 8; ++j) score[j][0] = score[j][1] = score[j][2] = score[j][3] = 0.f;
#pragma unroll 2
    for (int kk = 0; kk < K / 16; ++kk) {
        uint32_t a[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) fc_ldsm(a[p], fc_sm(qs + p * RC * KS + (row0 + (lane & 15)) * KS + kk * 16 + (lane >> 4) * 8));
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            if (j <= 2 * rb + 1) {
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    fc_ldsm(b[p], fc_sm(ks + p * RC * KS + (j * 8 + (lane & 7) + 8 * (lane >> 4)) * KS + kk * 16 + 8 * ((lane >> 3) & 1)));
                fc_mma3(score[j], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
                fc_mma3(score[j + 1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
            }
        }
    }
    for (int item = 0; item < items; ++item) {
        const int h = grp * per_group + (i0 + item) / v_tiles, v0 = (i0 + item) % v_tiles * RT;
        const HeadScalars& w = sc[item];
        __syncthreads();                            // everyone is done with the keys, or with the item before
#pragma unroll
        for (int e = 0; e < 4; ++e) store_planes(xs + (tid / 16 + 16 * e) * RX + tid % 16 * 4, RC * RX, x[e]);
#pragma unroll
        for (int e = 0; e < SE; ++e) {
            const int i = tid + e * R_THREADS;
            if (i < QS) store_planes(ss + (i / 16) * RX + i % 16 * 4, K * RX, S[e]);
        }
        if (item + 1 < items) ask(item + 1);
        // what the keys ahead of the warp's rows weigh at the end of the block before them
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = lane + 32 * e, jb = j >> 4;
            if (j < row0) colf[j] = expf(w.Ls[j] + ((jb + 1 < rb ? w.block[jb + 1] : 0.f) + (jb + 2 < rb ? w.block[jb + 2] : 0.f))) * w.gain[j];
        }
        __syncthreads();
        float acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
        // the state's share
#pragma unroll 2
        for (int kk = 0; kk < K / 16; ++kk) {
            uint32_t a[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) fc_ldsm(a[p], fc_sm(qs + p * RC * KS + (row0 + (lane & 15)) * KS + kk * 16 + (lane >> 4) * 8));
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) fc_ldsm_t(b[p], fc_sm(ss + p * K * RX + (kk * 16 + (lane & 15)) * RX + cc + (j + (lane >> 4)) * 8));
                fc_mma3(acc[j], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
                fc_mma3(acc[j + 1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
            }
        }
        const float Lp0 = w.Lp[row0 + g], Lp1 = w.Lp[row0 + g + 8], Lo0 = w.Lo[row0 + g], Lo1 = w.Lo[row0 + g + 8], in0 = expf(w.before[rb] + Lp0), in1 = expf(w.before[rb] + Lp1);
        const float at0 = expf(Lp0), at1 = expf(Lp1);
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[j][0] *= in0; acc[j][1] *= in0; acc[j][2] *= in1; acc[j][3] *= in1; }
        // the chunk's own tokens up to the warp's rows, a block of 16 at a time
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk > rb) continue;
            float m[2][4];                          // keys 16 kk + 8 u + 2 t, + 1 of rows g and g + 8
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int key = kk * 16 + u * 8 + 2 * t;
                if (kk < rb) {
                    const float w0 = colf[key], w1 = colf[key + 1];
                    m[u][0] = score[2 * kk + u][0] * (at0 * w0); m[u][1] = score[2 * kk + u][1] * (at0 * w1);
                    m[u][2] = score[2 * kk + u][2] * (at1 * w0); m[u][3] = score[2 * kk + u][3] * (at1 * w1);
                } else {
                    const int d = u * 8 + 2 * t;    // the keys' places in the block, the rows' being g and g + 8
                    const float L0 = w.Lp[key], L1 = w.Lp[key + 1], l0 = w.Lo[key], l1 = w.Lo[key + 1], g0 = w.gain[key], g1 = w.gain[key + 1];
                    m[u][0] = d <= g ? score[2 * kk + u][0] * (expf((Lp0 - L0) + (Lo0 - l0)) * g0) : 0.f;
                    m[u][1] = d + 1 <= g ? score[2 * kk + u][1] * (expf((Lp0 - L1) + (Lo0 - l1)) * g1) : 0.f;
                    m[u][2] = d <= g + 8 ? score[2 * kk + u][2] * (expf((Lp1 - L0) + (Lo1 - l0)) * g0) : 0.f;
                    m[u][3] = d + 1 <= g + 8 ? score[2 * kk + u][3] * (expf((Lp1 - L1) + (Lo1 - l1)) * g1) : 0.f;
                }
            }
            uint32_t a[3][4];
            fc_split3(m[0][0], m[0][1], a[0][0], a[1][0], a[2][0]);
            fc_split3(m[0][2], m[0][3], a[0][1], a[1][1], a[2][1]);
            fc_split3(m[1][0], m[1][1], a[0][2], a[1][2], a[2][2]);
            fc_split3(m[1][2], m[1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) fc_ldsm_t(b[p], fc_sm(xs + p * RC * RX + (kk * 16 + (lane & 15)) * RX + cc + (j + (lane >> 4)) * 8));
                fc_mma3(acc[j], a, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
                fc_mma3(acc[j + 1], a, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
            }
        }
        const float skip = A.skip[h];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int i = row0 + g + 8 * r;
            if (i >= L) continue;
            const float* vr = A.v + (size_t)(first + i) * A.ldv + (size_t)h * A.V;
            float* dst = A.y + (size_t)(first + i) * A.ldy + (size_t)h * A.V;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = v0 + cc + j * 8 + 2 * t;
                if (col < A.V) {
                    const float2 own = *reinterpret_cast<const float2*>(vr + col);
                    *reinterpret_cast<float2*>(dst + col) = make_float2(fmaf(skip, own.x, acc[j][2 * r]), fmaf(skip, own.y, acc[j][2 * r + 1]));
                }
            }
        }
    }
}

// The tiles that the chunks could not do, token by token: a CTA looks at R_REDO of a sequence's, a warp each, and does those in turn; thread (row group,
// column).  Nothing to do, as nearly always, costs a launch of few CTAs (the same inside the outputs made these slower: 1,164 against 1,184 us for a
// prompt step of two runs of 1,024 over four layers of 32 heads of 64 x 64).
constexpr int R_REDO = 8;
template <int K>
__global__ void __launch_bounds__(R_THREADS)
state_chunk_redo_kernel(const StateChunks A, int v_tiles) {
    constexpr int ROWS = K / 4;
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float sums[2 * 4 * RT];              // the row groups' sums of a token, [2][4][RT]
    __shared__ bool todo[R_REDO];
    const int s = blockIdx.y, start = A.seq_start[s], n = A.seq_start[s + 1] - start;
    if (n < A.least || A.seq_slot[s] < 0) return;
    const int tid = threadIdx.x, col = tid % RT, rg = tid / RT, item0 = A.g0 * A.per_group() * v_tiles + blockIdx.x * R_REDO,
              item_end = (A.g0 + A.groups) * A.per_group() * v_tiles;
    {
        const int item = item0 + (tid >> 5);
        int any = 0;
        if (item < item_end)
            for (int c = tid & 31; c < (n + RC - 1) / RC; c += 32) any |= A.wild[(size_t)(start / RC + s + c) * A.H * v_tiles + item];
        any = __any_sync(0xffffffffu, any);
        if ((tid & 31) == 0) todo[tid >> 5] = any != 0;
        if (!__syncthreads_or(any)) return;
    }
    const int pos0 = A.seq_pos0[s];
    for (int i = 0; i < R_REDO; ++i) {
        if (!todo[i]) continue;
        const int h = (item0 + i) / v_tiles, v0 = (item0 + i) % v_tiles * RT;
        const int v = v0 + col, g = h / A.per_group();
        const bool there = v < A.V;
        const size_t at = ((size_t)h * K + rg * ROWS) * A.V + v, slot = (size_t)A.seq_slot[s] * 2;
        const float* from = A.state + (slot + (pos0 & 1)) * A.state_row + at;
        float* to = A.state + (slot + ((pos0 + n) & 1)) * A.state_row + at;
        float S[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) S[r] = there ? from[(size_t)r * A.V] : 0.f;
        const float a = -expf(A.a_log[h]), bias = A.dt_bias[h], skip = A.skip[h];
        for (int t = 0; t < n; ++t) {
            const size_t row = (size_t)start + t;
            const float dt = softplus_f(A.s0[row * A.ld_s0 + h] + bias), decay = expf(a * dt);
            const float x = there ? A.v[row * A.ldv + (size_t)h * A.V + v] : 0.f, dx = dt * x;
            const float* k = A.k + row * A.ldk + g * K + rg * ROWS;
            const float* q = A.q + row * A.ldq + g * K + rg * ROWS;
            float part = 0.f;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                S[r] = fmaf(decay, S[r], k[r] * dx);
                part = fmaf(S[r], q[r], part);
            }
            float* mine = sums + (t & 1) * 4 * RT;
            mine[rg * RT + col] = part;
            __syncthreads();                            // (the other copy is written before anyone can come back to this one)
            if (rg == 0 && there) A.y[row * A.ldy + (size_t)h * A.V + v] = fmaf(skip, x, ((mine[col] + mine[RT + col]) + mine[2 * RT + col]) + mine[3 * RT + col]);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
            if (there) to[(size_t)r * A.V] = S[r];
        __syncthreads();                            // the sums' buffers are free again
    }
}

template <int K> int launch_state_chunks(const StateChunks& A, int n_seqs, int max_new, cudaStream_t stream) {
    static DeviceMarks writes_marks, outputs_marks;
    cudaError_t e = allow_shared_memory(writes_marks, state_chunk_writes_kernel<K>, writes_smem<K>());
    if (e == cudaSuccess) e = allow_shared_memory(outputs_marks, state_chunk_outputs_kernel<K>, outputs_smem<K>());
    if (e != cudaSuccess) return vlrf_fail(VLRF_ERR_CUDA, "state_chunks: %d bytes of shared memory: %s", outputs_smem<K>(), cudaGetErrorString(e));
    const int chunks = (max_new + RC - 1) / RC, v_tiles = (A.V + RT - 1) / RT, parts = (A.H / A.G * v_tiles + R_ITEMS - 1) / R_ITEMS;
    VLRF_REQUIRE((long long)A.groups * parts <= 65535, "state_chunks: too many heads");
    const dim3 grid(chunks, A.groups * parts, n_seqs);
    launch_chained(state_chunk_writes_kernel<K>, grid, dim3(R_THREADS), (size_t)writes_smem<K>(), stream, A, v_tiles, parts);
    int st = vlrf_check_launch("state_chunks: writes");
    if (st != VLRF_OK) return st;
    const long long quads = (long long)A.heads() * K * A.V / 4;
    launch_chained(state_chunk_states_kernel, dim3((unsigned)((quads + 127) / 128), n_seqs), dim3(128), (size_t)0, stream, A, K * A.V, v_tiles);
    st = vlrf_check_launch("state_chunks: states");
    if (st != VLRF_OK) return st;
    launch_chained(state_chunk_outputs_kernel<K>, grid, dim3(R_THREADS), (size_t)outputs_smem<K>(), stream, A, v_tiles, parts);
    st = vlrf_check_launch("state_chunks: outputs");
    if (st != VLRF_OK) return st;
    launch_chained(state_chunk_redo_kernel<K>, dim3((A.heads() * v_tiles + R_REDO - 1) / R_REDO, n_seqs), dim3(R_THREADS), (size_t)0, stream, A, v_tiles);
    return vlrf_check_launch("state_chunks: redo");
}
bool sc_on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
}  // namespace

// Whether the chunked kernels take a state-space recurrence of these sizes: states of 16, 32, 64 or 128 rows, everything on 16 bytes.
extern "C" int vlrf_ssd_chunks_takes(int H, int G, int N, int P, int channels, int state_row) {
    return (H > 0 && G > 0 && H % G == 0 && (N == 16 || N == 32 || N == 64 || N == 128) && P > 0 && P % 4 == 0 && channels % 4 == 0 &&
            state_row % 4 == 0 && channels == H * P + 2 * G * N) ? 1 : 0;
}

// How the groups of a step of T tokens in n_seqs sequences share scratch of at most `limit` numbers: how many a pass takes (0: not even
// one fits), as evenly as passes allow.  Per chunk: a state and a number for every head of a pass, and the marks of all heads' tiles.
static int chunk_groups(int T, int n_seqs, int H, int G, int N, int P, long long limit, long long* floats) {
    const long long slots = (long long)T / RC + n_seqs, marks = slots * H * ((P + RT - 1) / RT), group = slots * (H / G) * ((long long)N * P + 1);
    long long most = limit < marks ? 0 : (limit - marks) / group;
    if (most > G) most = G;
    if (most < 1) { *floats = 0; return 0; }
    const int passes = (int)((G + most - 1) / most), groups = (G + passes - 1) / passes;
    *floats = groups * group + marks;
    return groups;
}

// float32 numbers of scratch that a step of T tokens in n_seqs sequences takes where it may have `limit`; 0: it cannot run in so little
extern "C" int vlrf_ssd_chunks_scratch(int T, int n_seqs, int H, int G, int N, int P, long long limit, long long* floats) {
    VLRF_REQUIRE(T >= 0 && n_seqs > 0 && H > 0 && G > 0 && H % G == 0 && N > 0 && P > 0 && floats != nullptr, "ssd_chunks_scratch: bad arguments");
    chunk_groups(T, n_seqs, H, G, N, P, limit, floats);
    return VLRF_OK;
}

extern "C" int vlrf_ssd_chunks(const float* xbc, int channels, const float* proj, int ld, int dt_off, const float* dt_bias, const float* a_log,
                               const float* D, float* scratch, long long scratch_floats, float* state, int state_row, const int* seq_slot, const int* seq_start,
                               const int* seq_pos0, float* y, int n_tokens, int n_seqs, int max_new, int chunked, int H, int G, int N, int P,
                               cudaStream_t stream) {
    VLRF_REQUIRE(vlrf_ssd_chunks_takes(H, G, N, P, channels, state_row), "ssd_chunks: a state of %d by %d or the rows' strides are not taken", N, P);
    VLRF_REQUIRE(n_tokens >= 0 && n_seqs >= 0 && n_seqs <= 65535 && max_new >= 0 && scratch != nullptr && dt_off + H <= ld && chunked >= 1,
                 "ssd_chunks: bad arguments");
    VLRF_REQUIRE((size_t)H * N * P <= (size_t)state_row, "ssd_chunks: the state row does not hold the states");
    VLRF_REQUIRE(sc_on16(xbc) && sc_on16(scratch) && sc_on16(state) && sc_on16(y), "ssd_chunks: misaligned rows");
    if (n_seqs == 0 || max_new == 0) return VLRF_OK;
    StateChunks A;
    A.v = xbc; A.k = xbc + (size_t)H * P; A.q = A.k + (size_t)G * N;
    A.ldq = A.ldk = A.ldv = channels;
    A.s0 = proj + dt_off; A.ld_s0 = ld; A.dt_bias = dt_bias; A.a_log = a_log; A.skip = D;
    A.state = state; A.state_row = state_row; A.seq_slot = seq_slot; A.seq_start = seq_start; A.seq_pos0 = seq_pos0;
    A.least = chunked;
    A.y = y; A.ldy = H * P; A.H = H; A.G = G; A.V = P;
    long long floats = 0;
    const int groups = chunk_groups(n_tokens, n_seqs, H, G, N, P, scratch_floats, &floats);
    VLRF_REQUIRE(groups > 0, "ssd_chunks: %lld numbers of scratch do not hold a group's chunks", scratch_floats);
    const size_t slots = ((size_t)n_tokens / RC + n_seqs) * groups * (H / G);          // (chunk, head of a pass)
    A.scratch = scratch;
    A.aux = scratch + slots * (size_t)N * P;
    A.wild = reinterpret_cast<int*>(A.aux + slots);
    for (A.g0 = 0; A.g0 < G; A.g0 += groups) {
        A.groups = G - A.g0 < groups ? G - A.g0 : groups;
        const int st = N == 16   ? launch_state_chunks<16>(A, n_seqs, max_new, stream)
                       : N == 32 ? launch_state_chunks<32>(A, n_seqs, max_new, stream)
                       : N == 64 ? launch_state_chunks<64>(A, n_seqs, max_new, stream)
                                 : launch_state_chunks<128>(A, n_seqs, max_new, stream);
        if (st != VLRF_OK) return st;
    }
    return VLRF_OK;
}
