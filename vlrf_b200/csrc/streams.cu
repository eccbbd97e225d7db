// A residual carried in several streams, and the small row-wise kernels of models that use one.
//
// The residual of a token is S rows of d float32 numbers, [T][S][d].  A sublayer reads one row, a weighted sum of the
// streams, through its norm; its result y is then written back into every stream together with a mix of the old
// streams:
//     read:   u = Σ_s a[s] · x[s]            h = u / sqrt(mean(u²) + eps) · w        (one kernel, sums in float32)
//     write:  x'[j] = Σ_s m[s][j] · x[s] + b[j] · y      for every j at once, from the old streams
// With a = null every coefficient is 1 (the sum of the streams: what the model's last norm reads), and `rows` gathers
// the tokens whose logits are wanted.  S = 1 with a = null is the plain RMS norm of a row.
//
// A write that is followed by the next sublayer's read is one kernel (write_read): one pass over the streams.
//
// embed_streams: x[t][s] = table[token[t]] · scale for every stream s (scale 1 and one stream: a plain lookup).
// embed_bigram: x[t] = table[token[t]] · scale + pairs[row], one stream; row = (token before · mul_prev + token · mul_cur)
//   mod buckets, and row `buckets` (the table's last) for a sequence's first token.  The token before is the row above
//   where the step brings it, else the sequence's kept token: an int32 state [slot][2] holds each sequence's last token
//   twice, a step reading the copy of the parity of the position it begins at and writing the copy of the parity of the
//   position it ends at, so a step of one token leaves what it read and may run twice.  The CTA of a sequence's first
//   token of the step also keeps the sequence's last token of the step, after its own read of the kept one.
// embed_sinusoid: x[t] = table[token[t]] · scale + the position in sinusoids (entry 2i the sine, entry 2i + 1 the cosine of
//   position · freq[i]), one stream.
// softcap: v ← cap · tanh(v / cap) over float32 rows (logits).  scale_values: v ← v · factor.
#include "common.cuh"

namespace {
constexpr int ST_THREADS = 128;
constexpr int ST_MAX_STREAMS = 16;

template <typename WT>
__global__ void __launch_bounds__(ST_THREADS)
embed_streams_kernel(const WT* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int d, int V,
                     int S, float scale, int* __restrict__ dev_err) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    int id = tokens[t];
    if (id < 0 || id >= V) {
        if (threadIdx.x == 0) atomicOr(dev_err, VLRF_DEVERR_TOKEN_RANGE);
        id = min(max(id, 0), V - 1);
    }
    const WT* row = table + (size_t)id * d;
    float* out = x + (size_t)t * S * d;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) {
        const float v = ElemIO<WT>::load(row + i) * scale;
        for (int s = 0; s < S; ++s) out[(size_t)s * d + i] = v;
    }
}

// The angle is formed in 64-bit and brought into −π … π before the 32-bit sine and cosine, so that a far position loses nothing.
template <typename WT>
__global__ void __launch_bounds__(ST_THREADS)
embed_sinusoid_kernel(const WT* __restrict__ table, const int* __restrict__ tokens, const int* __restrict__ tok_slot,
                      const int* __restrict__ tok_pos, const double* __restrict__ freq, float* __restrict__ x, int d, int V, float scale,
                      int* __restrict__ dev_err) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    if (tok_slot[t] < 0) return;              // padding row (the whole CTA leaves)
    int id = tokens[t];
    if (id < 0 || id >= V) {
        if (threadIdx.x == 0) atomicOr(dev_err, VLRF_DEVERR_TOKEN_RANGE);
        id = min(max(id, 0), V - 1);
    }
    const WT* row = table + (size_t)id * d;
    float* out = x + (size_t)t * d;
    const double pos = (double)tok_pos[t], turn = 6.283185307179586476925;
    for (int i = threadIdx.x; 2 * i < d; i += ST_THREADS) {
        const double a = pos * freq[i];
        float sn, cn;
        sincosf((float)(a - rint(a / turn) * turn), &sn, &cn);
        out[2 * i] = fmaf(ElemIO<WT>::load(row + 2 * i), scale, sn);
        if (2 * i + 1 < d) out[2 * i + 1] = fmaf(ElemIO<WT>::load(row + 2 * i + 1), scale, cn);
    }
}

template <typename WT>
__global__ void __launch_bounds__(ST_THREADS)
embed_bigram_kernel(const WT* __restrict__ table, const WT* __restrict__ pairs, const int* __restrict__ tokens,
                    const int* __restrict__ tok_slot, const int* __restrict__ tok_pos, const int* __restrict__ seq_start, int n_seqs,
                    int* __restrict__ kept, float* __restrict__ x, int T, int d, int V, int buckets, int mul_prev, int mul_cur,
                    float scale, __nv_bfloat16* __restrict__ also, int* __restrict__ dev_err) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ int row_sm;
    const int t = blockIdx.x;
    const int slot = tok_slot[t];
    if (slot < 0) return;                     // padding row (the whole CTA leaves)
    int id = tokens[t];
    if (id < 0 || id >= V) {
        if (threadIdx.x == 0) atomicOr(dev_err, VLRF_DEVERR_TOKEN_RANGE);
        id = min(max(id, 0), V - 1);
    }
    if (threadIdx.x == 0) {
        const int pos = tok_pos[t];
        const bool above = t > 0 && tok_slot[t - 1] == slot && tok_pos[t - 1] == pos - 1;   // the step brings the token before
        int prev = -1;
        if (above) prev = tokens[t - 1];
        else {
            if (pos > 0) prev = kept[(size_t)slot * 2 + (pos & 1)];
            // this row begins its sequence's tokens of the step: find where they end and keep the last one
            int lo = 0, hi = n_seqs - 1;
            while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (seq_start[mid] <= t) lo = mid; else hi = mid - 1; }
            const int last = seq_start[lo + 1] - 1;
            if (last >= t && last < T) kept[(size_t)slot * 2 + ((pos + (last - t) + 1) & 1)] = tokens[last];
        }
        int row = buckets;
        if (pos > 0) {
            prev = min(max(prev, 0), V - 1);
            row = (int)(((long long)prev * mul_prev + (long long)id * mul_cur) % buckets);
            if (row < 0) row += buckets;
        }
        row_sm = row;
    }
    __syncthreads();
    const WT* er = table + (size_t)id * d;
    const WT* br = pairs + (size_t)row_sm * d;
    float* out = x + (size_t)t * d;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) {
        const float v = fmaf(ElemIO<WT>::load(er + i), scale, ElemIO<WT>::load(br + i));
        out[i] = v;
        if (also != nullptr) also[(size_t)t * d + i] = __float2bfloat16_rn(v);     // what the first sublayer reads of the row
    }
}

__global__ void scale_values_kernel(float* __restrict__ v, long long n, float factor) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] *= factor;
}

template <typename OT>
__global__ void __launch_bounds__(ST_THREADS)
streams_read_norm_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ a,
                         const float* __restrict__ w, OT* __restrict__ out, int d, int S, float eps) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float u_sm[];          // [d]
    __shared__ float red[ST_THREADS / 32];
    __shared__ float coef[ST_MAX_STREAMS];
    const int r = blockIdx.x;
    const float* xr = x + (size_t)(rows ? rows[r] : r) * S * d;
    if (threadIdx.x < S) coef[threadIdx.x] = a ? a[threadIdx.x] : 1.f;
    __syncthreads();
    float ss = 0.f;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) {
        float u = 0.f;
        for (int s = 0; s < S; ++s) u = fmaf(coef[s], xr[(size_t)s * d + i], u);
        u_sm[i] = u;
        ss = fmaf(u, u, ss);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < ST_THREADS / 32; ++i) total += red[i];
    const float inv = 1.f / sqrtf(total / (float)d + eps);
    OT* o = out + (size_t)r * d;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) ElemIO<OT>::store(o + i, u_sm[i] * inv * w[i]);
}

template <int SMAX>
__global__ void __launch_bounds__(ST_THREADS)
streams_write_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ b,
                     const float* __restrict__ y, int d, int S) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float m_sm[ST_MAX_STREAMS * ST_MAX_STREAMS];
    __shared__ float b_sm[ST_MAX_STREAMS];
    for (int i = threadIdx.x; i < S * S; i += ST_THREADS) m_sm[i] = mix[i];
    if (threadIdx.x < S) b_sm[threadIdx.x] = b[threadIdx.x];
    __syncthreads();
    const int t = blockIdx.x;
    float* xr = x + (size_t)t * S * d;
    const float* yr = y + (size_t)t * d;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) {
        float old[SMAX];
#pragma unroll
        for (int s = 0; s < SMAX; ++s) old[s] = s < S ? xr[(size_t)s * d + i] : 0.f;
        const float yv = yr[i];
#pragma unroll
        for (int j = 0; j < SMAX; ++j) {
            if (j < S) {
                float v = b_sm[j] * yv;
#pragma unroll
                for (int s = 0; s < SMAX; ++s)
                    if (s < S) v = fmaf(m_sm[s * S + j], old[s], v);
                xr[(size_t)j * d + i] = v;
            }
        }
    }
}

// The write of one sublayer and the read of the next in one pass over the streams: x' as in the write kernel, then
// h = RMSnorm(Σ_j a[j] · x'[j]) · w.  The row's u stays in shared memory between the two.
template <int SMAX, typename OT>
__global__ void __launch_bounds__(ST_THREADS)
streams_write_read_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ b,
                          const float* __restrict__ y, const float* __restrict__ a, const float* __restrict__ w,
                          OT* __restrict__ out, int d, int S, float eps) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float u_sm[];          // [d]
    __shared__ float m_sm[ST_MAX_STREAMS * ST_MAX_STREAMS];
    __shared__ float b_sm[ST_MAX_STREAMS], a_sm[ST_MAX_STREAMS];
    __shared__ float red[ST_THREADS / 32];
    for (int i = threadIdx.x; i < S * S; i += ST_THREADS) m_sm[i] = mix[i];
    if (threadIdx.x < S) { b_sm[threadIdx.x] = b[threadIdx.x]; a_sm[threadIdx.x] = a[threadIdx.x]; }
    __syncthreads();
    const int t = blockIdx.x;
    float* xr = x + (size_t)t * S * d;
    const float* yr = y + (size_t)t * d;
    float ss = 0.f;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) {
        float old[SMAX];
#pragma unroll
        for (int s = 0; s < SMAX; ++s) old[s] = s < S ? xr[(size_t)s * d + i] : 0.f;
        const float yv = yr[i];
        float u = 0.f;
#pragma unroll
        for (int j = 0; j < SMAX; ++j) {
            if (j < S) {
                float v = b_sm[j] * yv;
#pragma unroll
                for (int s = 0; s < SMAX; ++s)
                    if (s < S) v = fmaf(m_sm[s * S + j], old[s], v);
                xr[(size_t)j * d + i] = v;
                u = fmaf(a_sm[j], v, u);
            }
        }
        u_sm[i] = u;
        ss = fmaf(u, u, ss);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < ST_THREADS / 32; ++i) total += red[i];
    const float inv = 1.f / sqrtf(total / (float)d + eps);
    OT* o = out + (size_t)t * d;
    for (int i = threadIdx.x; i < d; i += ST_THREADS) ElemIO<OT>::store(o + i, u_sm[i] * inv * w[i]);
}

// The two kernels that read a row through a norm, and the embedding, with a row's quads in registers, one a thread: for rows of up
// to 4,096 numbers (a multiple of 4) on 16-byte boundaries and up to 8 streams.  All of a thread's loads are under way at once, the
// coefficients' and the weight's ahead of the wait; walking a row 128 numbers at a time, a round trip after another, took 15 us
// for 8 rows of 4 x 2,048 inside a decode step, and the time did not depend on the number of rows.
constexpr int STQ_MAX_STREAMS = 8, STQ_MAX_D = 4096;

__device__ __forceinline__ float4 fma4(float a, const float4& x, const float4& c) {
    return make_float4(fmaf(a, x.x, c.x), fmaf(a, x.y, c.y), fmaf(a, x.z, c.z), fmaf(a, x.w, c.w));
}
// h = u / sqrt(mean(u²) + eps) · w for a row whose quads the threads hold (zeros where there is none)
template <typename OT>
__device__ __forceinline__ void finish_quad_row(const float4& u, const float4& w, OT* o, int q, int d4, float eps, float (&red)[32]) {
    float ss = u.x * u.x;
    ss = fmaf(u.y, u.y, ss); ss = fmaf(u.z, u.z, ss); ss = fmaf(u.w, u.w, ss);
    ss = warp_sum(ss);
    if ((q & 31) == 0) red[q >> 5] = ss;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < (int)blockDim.x >> 5; ++i) total += red[i];
    const float inv = 1.f / sqrtf(total / (float)(4 * d4) + eps);
    if (q >= d4) return;
    const float4 h = make_float4(u.x * inv * w.x, u.y * inv * w.y, u.z * inv * w.z, u.w * inv * w.w);
    if constexpr (sizeof(OT) == 4) reinterpret_cast<float4*>(o)[q] = h;
    else {
        __nv_bfloat162 p[2] = {__floats2bfloat162_rn(h.x, h.y), __floats2bfloat162_rn(h.z, h.w)};
        reinterpret_cast<uint2*>(o)[q] = *reinterpret_cast<const uint2*>(p);
    }
}

template <int SMAX, typename OT>
__global__ void __launch_bounds__(STQ_MAX_D / 4)
streams_write_read_quads_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ b,
                                const float* __restrict__ y, const float* __restrict__ a, const float* __restrict__ w,
                                OT* __restrict__ out, int d4, int S, float eps) {
    __shared__ float m_sm[SMAX * SMAX], b_sm[SMAX], a_sm[SMAX], red[32];
    const int q = threadIdx.x, t = blockIdx.x;
    const bool mine = q < d4;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = q; i < S * S; i += blockDim.x) m_sm[i] = mix[i];
    if (q < S) { b_sm[q] = b[q]; a_sm[q] = a[q]; }
    const float4 wv = mine ? reinterpret_cast<const float4*>(w)[q] : none;
    pdl_wait();
    pdl_launch_dependents();
    float4* xr = reinterpret_cast<float4*>(x) + (size_t)t * S * d4 + q;
    float4 old[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) old[s] = (mine && s < S) ? xr[(size_t)s * d4] : none;
    const float4 yv = mine ? reinterpret_cast<const float4*>(y)[(size_t)t * d4 + q] : none;
    __syncthreads();
    float4 u = none;
#pragma unroll
    for (int j = 0; j < SMAX; ++j) {
        if (j < S) {
            const float bj = b_sm[j];
            float4 v = make_float4(bj * yv.x, bj * yv.y, bj * yv.z, bj * yv.w);
#pragma unroll
            for (int s = 0; s < SMAX; ++s)
                if (s < S) v = fma4(m_sm[s * S + j], old[s], v);
            if (mine) xr[(size_t)j * d4] = v;
            u = fma4(a_sm[j], v, u);
        }
    }
    finish_quad_row(u, wv, out + (size_t)t * 4 * d4, q, d4, eps, red);
}

// the write alone (the last of a pass: 8 rows of 4 x 2,048 inside a decode step 10.3 -> 1.9 us)
template <int SMAX>
__global__ void __launch_bounds__(STQ_MAX_D / 4)
streams_write_quads_kernel(float* __restrict__ x, const float* __restrict__ mix, const float* __restrict__ b, const float* __restrict__ y, int d4, int S) {
    __shared__ float m_sm[SMAX * SMAX], b_sm[SMAX];
    const int q = threadIdx.x, t = blockIdx.x;
    for (int i = q; i < S * S; i += blockDim.x) m_sm[i] = mix[i];
    if (q < S) b_sm[q] = b[q];
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    if (q >= d4) return;
    float4* xr = reinterpret_cast<float4*>(x) + (size_t)t * S * d4 + q;
    float4 old[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) old[s] = s < S ? xr[(size_t)s * d4] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 yv = reinterpret_cast<const float4*>(y)[(size_t)t * d4 + q];
#pragma unroll
    for (int j = 0; j < SMAX; ++j) {
        if (j < S) {
            const float bj = b_sm[j];
            float4 v = make_float4(bj * yv.x, bj * yv.y, bj * yv.z, bj * yv.w);
#pragma unroll
            for (int s = 0; s < SMAX; ++s)
                if (s < S) v = fma4(m_sm[s * S + j], old[s], v);
            xr[(size_t)j * d4] = v;
        }
    }
}

template <int SMAX, typename OT>
__global__ void __launch_bounds__(STQ_MAX_D / 4)
streams_read_norm_quads_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ a,
                               const float* __restrict__ w, OT* __restrict__ out, int d4, int S, float eps) {
    __shared__ float red[32];
    const int q = threadIdx.x, r = blockIdx.x;
    const bool mine = q < d4;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    float coef[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) coef[s] = s < S ? (a ? a[s] : 1.f) : 0.f;
    const float4 wv = mine ? reinterpret_cast<const float4*>(w)[q] : none;
    pdl_wait();
    pdl_launch_dependents();
    const float4* xr = reinterpret_cast<const float4*>(x) + (size_t)(rows ? rows[r] : r) * S * d4 + q;
    float4 v[SMAX];
#pragma unroll
    for (int s = 0; s < SMAX; ++s) v[s] = (mine && s < S) ? xr[(size_t)s * d4] : none;
    float4 u = none;
#pragma unroll
    for (int s = 0; s < SMAX; ++s)
        if (s < S) u = fma4(coef[s], v[s], u);
    finish_quad_row(u, wv, out + (size_t)r * 4 * d4, q, d4, eps, red);
}

template <typename WT>
__global__ void __launch_bounds__(STQ_MAX_D / 4)
embed_streams_quads_kernel(const WT* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int d4, int V,
                           int S, float scale, int* __restrict__ dev_err) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x, q = threadIdx.x;
    int id = tokens[t];
    if (id < 0 || id >= V) {
        if (q == 0) atomicOr(dev_err, VLRF_DEVERR_TOKEN_RANGE);
        id = min(max(id, 0), V - 1);
    }
    if (q >= d4) return;
    float4 v;
    if constexpr (sizeof(WT) == 4) v = reinterpret_cast<const float4*>(table)[(size_t)id * d4 + q];
    else {
        const uint2 two = reinterpret_cast<const uint2*>(table)[(size_t)id * d4 + q];
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&two.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&two.y);
        v = make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
    }
    v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
    float4* out = reinterpret_cast<float4*>(x) + (size_t)t * S * d4 + q;
    for (int s = 0; s < S; ++s) out[(size_t)s * d4] = v;
}

bool quads_take(int d, uintptr_t all) { return d % 4 == 0 && d <= STQ_MAX_D && all % 16 == 0; }
unsigned quad_threads(int d) { return (unsigned)((d / 4 + 31) / 32 * 32); }

__global__ void softcap_kernel(float* __restrict__ v, long long n, float cap) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = cap * tanhf(v[i] / cap);
}
}  // namespace

extern "C" int vlrf_embed_streams(const void* table, int w_dtype, const int* tokens, float* x, int T, int d, int V, int S,
                                  float scale, int* dev_err, cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && d > 0 && V > 0 && S > 0, "embed_streams: bad sizes");
    VLRF_REQUIRE(dev_err != nullptr, "embed_streams: needs the device error word");
    if (T == 0) return VLRF_OK;
    if (quads_take(d, (uintptr_t)table | (uintptr_t)x) && (w_dtype == VLRF_F32 || w_dtype == VLRF_BF16)) {
        if (w_dtype == VLRF_F32)
            launch_chained(embed_streams_quads_kernel<float>, dim3(T), dim3(quad_threads(d)), (size_t)0, stream, (const float*)table, tokens, x,
                           d / 4, V, S, scale, dev_err);
        else
            launch_chained(embed_streams_quads_kernel<__nv_bfloat16>, dim3(T), dim3(quad_threads(d)), (size_t)0, stream,
                           (const __nv_bfloat16*)table, tokens, x, d / 4, V, S, scale, dev_err);
        return vlrf_check_launch("embed_streams");
    }
    if (w_dtype == VLRF_F32)
        launch_chained(embed_streams_kernel<float>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const float*)table, tokens, x, d, V, S,
                       scale, dev_err);
    else if (w_dtype == VLRF_BF16)
        launch_chained(embed_streams_kernel<__nv_bfloat16>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const __nv_bfloat16*)table,
                       tokens, x, d, V, S, scale, dev_err);
    else
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "embed_streams: unknown dtype %d", w_dtype);
    return vlrf_check_launch("embed_streams");
}

extern "C" int vlrf_streams_read_norm(const float* x, const int* rows, const float* a, const float* w, void* out, int out_dtype,
                                      int n_rows, int d, int S, float eps, cudaStream_t stream) {
    VLRF_REQUIRE(n_rows >= 0 && d > 0 && S > 0 && S <= ST_MAX_STREAMS, "streams_read_norm: bad sizes rows=%d d=%d streams=%d", n_rows, d, S);
    VLRF_REQUIRE((size_t)d * sizeof(float) <= 160 * 1024, "streams_read_norm: a row of %d numbers does not fit shared memory", d);
    if (n_rows == 0) return VLRF_OK;
    if (S <= STQ_MAX_STREAMS && quads_take(d, (uintptr_t)x | (uintptr_t)w | (uintptr_t)out) && (out_dtype == VLRF_F32 || out_dtype == VLRF_BF16)) {
#define GO(M, OT) launch_chained(streams_read_norm_quads_kernel<M, OT>, dim3(n_rows), dim3(quad_threads(d)), (size_t)0, stream, x, rows, a, w, (OT*)out, d / 4, S, eps)
#define GO_S(OT) do { if (S == 1) GO(1, OT); else if (S <= 4) GO(4, OT); else GO(8, OT); } while (0)
        if (out_dtype == VLRF_F32) GO_S(float); else GO_S(__nv_bfloat16);
#undef GO_S
#undef GO
        return vlrf_check_launch("streams_read_norm");
    }
    const size_t smem = (size_t)d * sizeof(float);
    if (out_dtype == VLRF_F32) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(streams_read_norm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_chained(streams_read_norm_kernel<float>, dim3(n_rows), dim3(ST_THREADS), smem, stream, x, rows, a, w, (float*)out, d, S, eps);
    } else if (out_dtype == VLRF_BF16) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(streams_read_norm_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch_chained(streams_read_norm_kernel<__nv_bfloat16>, dim3(n_rows), dim3(ST_THREADS), smem, stream, x, rows, a, w,
                       (__nv_bfloat16*)out, d, S, eps);
    } else {
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "streams_read_norm: unknown output dtype %d", out_dtype);
    }
    return vlrf_check_launch("streams_read_norm");
}

extern "C" int vlrf_streams_write(float* x, const float* mix, const float* b, const float* y, int T, int d, int S,
                                  cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && d > 0 && S > 0 && S <= ST_MAX_STREAMS, "streams_write: bad sizes rows=%d d=%d streams=%d", T, d, S);
    if (T == 0) return VLRF_OK;
    if (S <= STQ_MAX_STREAMS && quads_take(d, (uintptr_t)x | (uintptr_t)y)) {
        const dim3 block(quad_threads(d));
        if (S <= 2) launch_chained(streams_write_quads_kernel<2>, dim3(T), block, (size_t)0, stream, x, mix, b, y, d / 4, S);
        else if (S <= 4) launch_chained(streams_write_quads_kernel<4>, dim3(T), block, (size_t)0, stream, x, mix, b, y, d / 4, S);
        else launch_chained(streams_write_quads_kernel<8>, dim3(T), block, (size_t)0, stream, x, mix, b, y, d / 4, S);
        return vlrf_check_launch("streams_write");
    }
    // (the streams of a column are held in registers: the kernel is instantiated for up to 2, 4, 8 and 16 of them)
    if (S <= 2) launch_chained(streams_write_kernel<2>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, x, mix, b, y, d, S);
    else if (S <= 4) launch_chained(streams_write_kernel<4>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, x, mix, b, y, d, S);
    else if (S <= 8) launch_chained(streams_write_kernel<8>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, x, mix, b, y, d, S);
    else launch_chained(streams_write_kernel<16>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, x, mix, b, y, d, S);
    return vlrf_check_launch("streams_write");
}

extern "C" int vlrf_streams_write_read(float* x, const float* mix, const float* b, const float* y, const float* a, const float* w,
                                       void* out, int out_dtype, int T, int d, int S, float eps, cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && d > 0 && S > 0 && S <= ST_MAX_STREAMS, "streams_write_read: bad sizes rows=%d d=%d streams=%d", T, d, S);
    VLRF_REQUIRE((size_t)d * sizeof(float) <= 160 * 1024, "streams_write_read: a row of %d numbers does not fit shared memory", d);
    VLRF_REQUIRE(out_dtype == VLRF_F32 || out_dtype == VLRF_BF16, "streams_write_read: unknown output dtype %d", out_dtype);
    VLRF_REQUIRE(a != nullptr, "streams_write_read: the read needs its coefficients");
    if (T == 0) return VLRF_OK;
    if (S <= STQ_MAX_STREAMS && quads_take(d, (uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (uintptr_t)out)) {
#define GO(M, OT) launch_chained(streams_write_read_quads_kernel<M, OT>, dim3(T), dim3(quad_threads(d)), (size_t)0, stream, x, mix, b, y, a, w, (OT*)out, d / 4, S, eps)
#define GO_S(OT) do { if (S <= 2) GO(2, OT); else if (S <= 4) GO(4, OT); else GO(8, OT); } while (0)
        if (out_dtype == VLRF_F32) GO_S(float); else GO_S(__nv_bfloat16);
#undef GO_S
#undef GO
        return vlrf_check_launch("streams_write_read");
    }
    const size_t smem = (size_t)d * sizeof(float);
#define GO(M, OT) do { if (smem > 48 * 1024) cudaFuncSetAttribute(streams_write_read_kernel<M, OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        launch_chained(streams_write_read_kernel<M, OT>, dim3(T), dim3(ST_THREADS), smem, stream, x, mix, b, y, a, w, (OT*)out, d, S, eps); } while (0)
#define GO_S(OT) do { if (S <= 2) GO(2, OT); else if (S <= 4) GO(4, OT); else if (S <= 8) GO(8, OT); else GO(16, OT); } while (0)
    if (out_dtype == VLRF_F32) GO_S(float); else GO_S(__nv_bfloat16);
#undef GO_S
#undef GO
    return vlrf_check_launch("streams_write_read");
}

extern "C" int vlrf_embed_sinusoid(const void* table, int w_dtype, const int* tokens, const int* tok_slot, const int* tok_pos,
                                   const double* freq, float* x, int T, int d, int V, float scale, int* dev_err, cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && d > 0 && V > 0, "embed_sinusoid: bad sizes T=%d d=%d V=%d", T, d, V);
    VLRF_REQUIRE(freq != nullptr && dev_err != nullptr, "embed_sinusoid: needs the frequencies and the error word");
    if (T == 0) return VLRF_OK;
    if (w_dtype == VLRF_F32)
        launch_chained(embed_sinusoid_kernel<float>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const float*)table, tokens, tok_slot,
                       tok_pos, freq, x, d, V, scale, dev_err);
    else if (w_dtype == VLRF_BF16)
        launch_chained(embed_sinusoid_kernel<__nv_bfloat16>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const __nv_bfloat16*)table,
                       tokens, tok_slot, tok_pos, freq, x, d, V, scale, dev_err);
    else
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "embed_sinusoid: unknown dtype %d", w_dtype);
    return vlrf_check_launch("embed_sinusoid");
}

extern "C" int vlrf_embed_bigram(const void* table, const void* pairs, int w_dtype, const int* tokens, const int* tok_slot,
                                 const int* tok_pos, const int* seq_start, int n_seqs, int* kept, float* x, int T, int d, int V,
                                 int buckets, int mul_prev, int mul_cur, float scale, void* also, int* dev_err, cudaStream_t stream) {
    VLRF_REQUIRE(T >= 0 && d > 0 && V > 0 && buckets > 0 && n_seqs >= 0, "embed_bigram: bad sizes");
    VLRF_REQUIRE(dev_err != nullptr && kept != nullptr && seq_start != nullptr, "embed_bigram: needs the error word, the kept tokens and the sequences' rows");
    if (T == 0 || n_seqs == 0) return VLRF_OK;
    if (w_dtype == VLRF_F32)
        launch_chained(embed_bigram_kernel<float>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const float*)table, (const float*)pairs,
                       tokens, tok_slot, tok_pos, seq_start, n_seqs, kept, x, T, d, V, buckets, mul_prev, mul_cur, scale, (__nv_bfloat16*)also,
                       dev_err);
    else if (w_dtype == VLRF_BF16)
        launch_chained(embed_bigram_kernel<__nv_bfloat16>, dim3(T), dim3(ST_THREADS), (size_t)0, stream, (const __nv_bfloat16*)table,
                       (const __nv_bfloat16*)pairs, tokens, tok_slot, tok_pos, seq_start, n_seqs, kept, x, T, d, V, buckets, mul_prev,
                       mul_cur, scale, (__nv_bfloat16*)also, dev_err);
    else
        return vlrf_fail(VLRF_ERR_INVALID_ARG, "embed_bigram: unknown dtype %d", w_dtype);
    return vlrf_check_launch("embed_bigram");
}

extern "C" int vlrf_scale_values(float* v, long long n, float factor, cudaStream_t stream) {
    VLRF_REQUIRE(n >= 0, "scale_values: bad size");
    if (n == 0) return VLRF_OK;
    launch_chained(scale_values_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), (size_t)0, stream, v, n, factor);
    return vlrf_check_launch("scale_values");
}

extern "C" int vlrf_softcap(float* v, long long n, float cap, cudaStream_t stream) {
    VLRF_REQUIRE(n >= 0 && cap > 0.f, "softcap: bad sizes or a cap that is not positive");
    if (n == 0) return VLRF_OK;
    launch_chained(softcap_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), (size_t)0, stream, v, n, cap);
    return vlrf_check_launch("softcap");
}
