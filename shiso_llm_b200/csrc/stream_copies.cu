// Row kernels of models that keep several copies of the residual stream and mix tokens with
// their predecessor: the hashed-pair embedding, the read/write of stream copies
// (hyper-connections) fused with the RMS norm, the token-shift blends, and a unary map.
//
// Everything here is float arithmetic on float streams; only the rows handed to a product are
// rounded to the activation type.
#include <type_traits>

#include "common.cuh"

// --------------------------------------------------------------------------- hashed-pair embedding

__device__ __forceinline__ int step_token(const int* ids, const int* feed_index, const int* fed_tokens, int t) {
    int id = ids[t];
    if (feed_index) {
        const int from = feed_index[t];
        if (from >= 0) id = fed_tokens[from];
    }
    return id;
}

// x_t = scale * E[id_t] + B[(id_{t-1} * mul_prev + id_t * mul_cur) mod buckets]; B[buckets] for a
// sequence's first token.  The previous token of a portion's first row is what the request's
// slot holds (token + 1).  The slots are written by the kernel below, after this one.  A step's first
// kernel, launched in full order: common.cuh says why.
template <typename WT>
__global__ void embed_hashed_pair_kernel(const int* ids, const int* feed_index, const int* fed_tokens,
                                         const WT* __restrict__ table, const WT* __restrict__ pair_table,
                                         const int* seq_of_token, const int* q_start,
                                         const int* start_pos, const int* slots,
                                         const int* state, long long state_stride, float* __restrict__ out,
                                         int hidden, int vocab, float scale, int buckets, int mul_prev, int mul_cur) {
    pdl_begin();
    const int t = blockIdx.x;
    const int id = step_token(ids, feed_index, fed_tokens, t);
    const int s = seq_of_token[t];
    int prev = -1;
    if (t > q_start[s]) prev = step_token(ids, feed_index, fed_tokens, t - 1);
    else if (start_pos[s] > 0) prev = state[(long long)slots[s] * state_stride] - 1;
    const bool valid = id >= 0 && id < vocab;
    long long row = buckets;
    if (prev >= 0 && valid) row = ((long long)prev * mul_prev + (long long)id * mul_cur) % buckets;
    const WT* e = table + (size_t)(valid ? id : 0) * hidden;
    const WT* b = pair_table + (size_t)row * hidden;
    float* dst = out + (size_t)t * hidden;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) dst[i] = valid ? to_f32(e[i]) * scale + to_f32(b[i]) : 0.0f;
}

__global__ void store_last_token_kernel(const int* ids, const int* feed_index, const int* fed_tokens,
                                        const int* q_start, const int* slots, int* state,
                                        long long state_stride, int num_seqs) {
    pdl_begin();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= num_seqs) return;
    const int a = q_start[s], e = q_start[s + 1];
    if (e > a) state[(long long)slots[s] * state_stride] = step_token(ids, feed_index, fed_tokens, e - 1) + 1;
}

SHISO_API int shiso_embed_hashed_pair(const int* ids, const int* feed_index, const int* fed_tokens, const void* table,
                                      const void* pair_table, int table_dtype, const int* seq_of_token, const int* q_start,
                                      const int* start_pos, const int* slots, int* state, long long state_stride, float* out,
                                      int tokens, int num_seqs, int hidden, int vocab, float scale, int buckets, int mul_prev,
                                      int mul_cur, cudaStream_t stream) {
    if (tokens <= 0) return SHISO_OK;
    if ((feed_index == nullptr) != (fed_tokens == nullptr) || buckets <= 0) return SHISO_ERR_SHAPE;
    const int threads = hidden >= 1024 ? 256 : 128;
    if (table_dtype == SHISO_F32)
        launch_in_order(embed_hashed_pair_kernel<float>, tokens, threads, 0, stream, ids, feed_index, fed_tokens, (const float*)table,
                      (const float*)pair_table, seq_of_token, q_start, start_pos, slots, (const int*)state, state_stride, out,
                      hidden, vocab, scale, buckets, mul_prev, mul_cur);
    else if (table_dtype == SHISO_BF16)
        launch_in_order(embed_hashed_pair_kernel<__nv_bfloat16>, tokens, threads, 0, stream, ids, feed_index, fed_tokens,
                      (const __nv_bfloat16*)table, (const __nv_bfloat16*)pair_table, seq_of_token, q_start, start_pos, slots,
                      (const int*)state, state_stride, out, hidden, vocab, scale, buckets, mul_prev, mul_cur);
    else
        return SHISO_ERR_DTYPE;
    launch_kernel(store_last_token_kernel, ceil_div_u(num_seqs, 128), 128, 0, stream, ids, feed_index, fed_tokens, q_start, slots,
                  state, state_stride, num_seqs);
    return launch_status();
}

// --------------------------------------------------------------------------- copies of the stream

constexpr int MAX_COPIES = 8;

// One block per token row.  With `y`: the copies become x_r' = sum_s mix[s, r] x_s + write[r] * y
// (stored to `dst` when given).  With `read`: u = sum_r read[r] x_r' is normalised,
// u * rsqrt(mean(u^2) + eps) * norm_w, into `normed`.  With `sum_out`: sum_r x_r'.  `src` has
// `copies` lanes `src_stride` floats apart (0: one stream stands for every copy).
template <typename AT>
__global__ void hyper_mix_kernel(const float* src, long long src_stride, const AT* y,
                                 const float* __restrict__ mix, const float* __restrict__ write, float* dst, long long dst_stride,
                                 const float* __restrict__ read, const float* __restrict__ norm_w, float eps,
                                 AT* __restrict__ normed, float* __restrict__ sum_out, int hidden, int copies) {
    extern __shared__ float row_u[];  // [hidden] when `read`
    __shared__ float scratch[33];
    __shared__ float s_mix[MAX_COPIES * MAX_COPIES], s_write[MAX_COPIES], s_read[MAX_COPIES];
    if (threadIdx.x < copies * copies && y) s_mix[threadIdx.x] = mix[threadIdx.x];
    if (threadIdx.x < copies) {
        if (y) s_write[threadIdx.x] = write[threadIdx.x];
        if (read) s_read[threadIdx.x] = read[threadIdx.x];
    }
    __syncthreads();
    pdl_begin();
    const size_t at = (size_t)blockIdx.x * hidden;
    float squares = 0.0f;
    // W neighbouring elements a thread: 4 (16-byte loads and stores of the float copies) where rows allow it
    auto walk = [&](auto width) {
        constexpr int W = decltype(width)::value;
        for (int i = threadIdx.x * W; i < hidden; i += blockDim.x * W) {
            float x[MAX_COPIES][W], nx[MAX_COPIES][W];
#pragma unroll
            for (int s = 0; s < MAX_COPIES; ++s) {
                if (s < copies) {
                    const float* p = src + (size_t)s * src_stride + at + i;
                    if (W == 4) {
                        const float4 v = *reinterpret_cast<const float4*>(p);
                        x[s][0] = v.x; x[s][W > 1 ? 1 : 0] = v.y; x[s][W > 2 ? 2 : 0] = v.z; x[s][W > 3 ? 3 : 0] = v.w;
                    } else {
                        x[s][0] = p[0];
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < W; ++e) x[s][e] = 0.0f;
                }
            }
            if (y) {
                float yy[W];
#pragma unroll
                for (int e = 0; e < W; ++e) yy[e] = to_f32(y[at + i + e]);
#pragma unroll
                for (int r = 0; r < MAX_COPIES; ++r) {
#pragma unroll
                    for (int e = 0; e < W; ++e) nx[r][e] = 0.0f;
                    if (r < copies) {
#pragma unroll
                        for (int e = 0; e < W; ++e) {
                            float v = 0.0f;
#pragma unroll
                            for (int s = 0; s < MAX_COPIES; ++s)
                                if (s < copies) v += s_mix[s * copies + r] * x[s][e];
                            nx[r][e] = v + s_write[r] * yy[e];
                        }
                        if (dst) {
                            float* p = dst + (size_t)r * dst_stride + at + i;
                            if (W == 4) *reinterpret_cast<float4*>(p) = make_float4(nx[r][0], nx[r][W > 1 ? 1 : 0], nx[r][W > 2 ? 2 : 0], nx[r][W > 3 ? 3 : 0]);
                            else p[0] = nx[r][0];
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < MAX_COPIES; ++r)
#pragma unroll
                    for (int e = 0; e < W; ++e) nx[r][e] = x[r][e];
            }
#pragma unroll
            for (int e = 0; e < W; ++e) {
                if (read) {
                    float u = 0.0f;
#pragma unroll
                    for (int r = 0; r < MAX_COPIES; ++r)
                        if (r < copies) u += s_read[r] * nx[r][e];
                    row_u[i + e] = u;
                    squares += u * u;
                }
                if (sum_out) {
                    float total = 0.0f;
#pragma unroll
                    for (int r = 0; r < MAX_COPIES; ++r)
                        if (r < copies) total += nx[r][e];
                    sum_out[at + i + e] = total;
                }
            }
        }
    };
    if (hidden % 4 == 0) walk(std::integral_constant<int, 4>{});
    else walk(std::integral_constant<int, 1>{});
    if (!read) return;
    const float scale = rsqrtf(block_sum(squares, scratch) / (float)hidden + eps);
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) normed[at + i] = from_f32<AT>(row_u[i] * scale * norm_w[i]);
}

// Four neighbouring activations as floats.
template <typename AT> struct Quad;
template <> struct Quad<float> {
    __device__ static float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
    __device__ static void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};
template <> struct Quad<__nv_bfloat16> {
    __device__ static float4 load(const __nv_bfloat16* p) {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
    }
    __device__ static void store(__nv_bfloat16* p, float4 v) {
        __nv_bfloat162 b[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
        *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(b);
    }
};

// The same for two or four copies and rows of up to 512 Q elements, four a 16-byte access: the number of copies is
// known, so that a row's mixing is COPIES x COPIES multiply-adds an element (the kernel above steps over
// MAX_COPIES squared predicated ones), all of a row's loads are asked for at once, and u waits for
// its norm in registers.  A row's traffic bounds it.
// (bfloat16, microseconds, the kernel above first: 2,000 rows of 2,048 with two copies 30.9 and 9.6, with four
// 40.6 and 17.5; 300 rows of 1,024 with two 5.6 and 2.3; 8 rows of 2,048 5.3 and 2.5)
template <typename AT, int COPIES, int Q>
__global__ void __launch_bounds__(128) hyper_mix_quads_kernel(const float* src, long long src_stride, const AT* y, const float* __restrict__ mix,
                                                              const float* __restrict__ write, float* dst, long long dst_stride,
                                                              const float* __restrict__ read, const float* __restrict__ norm_w, float eps,
                                                              AT* __restrict__ normed, float* __restrict__ sum_out, int hidden) {
    __shared__ float scratch[33];
    float m[COPIES][COPIES], wr[COPIES], rd[COPIES];
#pragma unroll
    for (int s = 0; s < COPIES; ++s) {
#pragma unroll
        for (int r = 0; r < COPIES; ++r) m[s][r] = y ? mix[s * COPIES + r] : 0.0f;
        wr[s] = y ? write[s] : 0.0f;
        rd[s] = read ? read[s] : 0.0f;
    }
    const int quads = hidden / 4;
    float4 w4[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * 128;
        w4[q] = read && i < quads ? *reinterpret_cast<const float4*>(norm_w + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    pdl_begin();
    const size_t at = (size_t)blockIdx.x * hidden;
    float x[Q][COPIES][4], yy[Q][4], u[Q][4];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * 128;
        const bool in = i < quads;
#pragma unroll
        for (int s = 0; s < COPIES; ++s) {
            const float4 v = in ? *reinterpret_cast<const float4*>(src + (size_t)s * src_stride + at + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x[q][s][0] = v.x, x[q][s][1] = v.y, x[q][s][2] = v.z, x[q][s][3] = v.w;
        }
        const float4 v = in && y ? Quad<AT>::load(y + at + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        yy[q][0] = v.x, yy[q][1] = v.y, yy[q][2] = v.z, yy[q][3] = v.w;
    }
    float squares = 0.0f;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * 128;
        float nx[COPIES][4], total[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            u[q][e] = 0.0f, total[e] = 0.0f;
#pragma unroll
            for (int r = 0; r < COPIES; ++r) {
                float v = 0.0f;
                if (y) {
#pragma unroll
                    for (int s = 0; s < COPIES; ++s) v += m[s][r] * x[q][s][e];
                    v = v + wr[r] * yy[q][e];
                } else {
                    v = x[q][r][e];
                }
                nx[r][e] = v;
                u[q][e] += rd[r] * v;
                total[e] += v;
            }
            squares += u[q][e] * u[q][e];
        }
        if (i < quads) {
            if (y && dst)
#pragma unroll
                for (int r = 0; r < COPIES; ++r)
                    *reinterpret_cast<float4*>(dst + (size_t)r * dst_stride + at + 4 * i) = make_float4(nx[r][0], nx[r][1], nx[r][2], nx[r][3]);
            if (sum_out) *reinterpret_cast<float4*>(sum_out + at + 4 * i) = make_float4(total[0], total[1], total[2], total[3]);
        }
    }
    if (!read) return;
    const float scale = rsqrtf(block_sum(squares, scratch) / (float)hidden + eps);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * 128;
        if (i < quads)
            Quad<AT>::store(normed + at + 4 * i, make_float4(u[q][0] * scale * w4[q].x, u[q][1] * scale * w4[q].y, u[q][2] * scale * w4[q].z, u[q][3] * scale * w4[q].w));
    }
}

// Whether it takes the call; launched then.
template <typename AT>
static bool hyper_mix_quads(const float* src, long long src_stride, const AT* y, const float* mix, const float* write, float* dst,
                            long long dst_stride, const float* read, const float* norm_w, float eps, AT* normed, float* sum_out, int tokens,
                            int hidden, int copies, cudaStream_t stream) {
    if ((copies != 2 && copies != 4) || hidden % 4 || hidden > 2048 || src_stride % 4 || dst_stride % 4 ||
        (((uintptr_t)src | (uintptr_t)y | (uintptr_t)dst | (uintptr_t)normed | (uintptr_t)norm_w | (uintptr_t)sum_out) & 15))
        return false;
    const int q = (hidden / 4 + 127) / 128;
    auto go = [&](auto kernel) {
        launch_kernel(kernel, tokens, 128, 0, stream, src, src_stride, y, mix, write, dst, dst_stride, read, norm_w, eps, normed, sum_out, hidden);
    };
    if (copies == 2) {
        if (q <= 1) go(hyper_mix_quads_kernel<AT, 2, 1>);
        else if (q <= 2) go(hyper_mix_quads_kernel<AT, 2, 2>);
        else go(hyper_mix_quads_kernel<AT, 2, 4>);
    } else {
        if (q <= 1) go(hyper_mix_quads_kernel<AT, 4, 1>);
        else if (q <= 2) go(hyper_mix_quads_kernel<AT, 4, 2>);
        else go(hyper_mix_quads_kernel<AT, 4, 4>);
    }
    return true;
}

SHISO_API int shiso_hyper_mix(const float* src, long long src_stride, const void* y, const float* mix, const float* write,
                              float* dst, long long dst_stride, const float* read, const float* norm_w, float eps, void* normed,
                              float* sum_out, int act_dtype, int tokens, int hidden, int copies, cudaStream_t stream) {
    if (tokens <= 0) return SHISO_OK;
    if (copies < 1 || copies > MAX_COPIES || hidden > 12000) return SHISO_ERR_SHAPE;
    if ((y != nullptr) != (mix != nullptr) || (y != nullptr) != (write != nullptr) || (read != nullptr) != (normed != nullptr))
        return SHISO_ERR_UNSUPPORTED;
    if (act_dtype == SHISO_F32 ? hyper_mix_quads<float>(src, src_stride, (const float*)y, mix, write, dst, dst_stride, read, norm_w, eps, (float*)normed,
                                                        sum_out, tokens, hidden, copies, stream)
                               : act_dtype == SHISO_BF16 &&
                                     hyper_mix_quads<__nv_bfloat16>(src, src_stride, (const __nv_bfloat16*)y, mix, write, dst, dst_stride, read, norm_w,
                                                                    eps, (__nv_bfloat16*)normed, sum_out, tokens, hidden, copies, stream))
        return launch_status();
    const int threads = hidden >= 2048 ? 256 : 128;
    const size_t smem = read ? (size_t)hidden * sizeof(float) : 0;
    if (act_dtype == SHISO_F32)
        launch_kernel(hyper_mix_kernel<float>, tokens, threads, smem, stream, src, src_stride, (const float*)y, mix, write, dst,
                      dst_stride, read, norm_w, eps, (float*)normed, sum_out, hidden, copies);
    else if (act_dtype == SHISO_BF16)
        launch_kernel(hyper_mix_kernel<__nv_bfloat16>, tokens, threads, smem, stream, src, src_stride, (const __nv_bfloat16*)y, mix,
                      write, dst, dst_stride, read, norm_w, eps, (__nv_bfloat16*)normed, sum_out, hidden, copies);
    else
        return SHISO_ERR_DTYPE;
    return launch_status();
}

// --------------------------------------------------------------------------- token shift

// out[c, t, :] = h_t + (h_{t-1} - h_t) * mu[c, :] for c < blends, with h_{t-1} the row before in
// the same sequence, the request's stored row for a portion's first token, zeros at position 0.
template <typename AT>
__global__ void token_shift_blend_kernel(const AT* h, const float* __restrict__ mu, const float* state,
                                         long long state_stride, const int* seq_of_token,
                                         const int* q_start, const int* start_pos,
                                         const int* slots, AT* __restrict__ out, int tokens, int hidden, int blends) {
    pdl_begin();
    const int t = blockIdx.x;
    const int s = seq_of_token[t];
    const bool first = t == q_start[s];
    const bool none = first && start_pos[s] == 0;
    const float* kept = state + (long long)slots[s] * state_stride;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        const float cur = to_f32(h[(size_t)t * hidden + i]);
        const float prev = none ? 0.0f : (first ? kept[i] : to_f32(h[(size_t)(t - 1) * hidden + i]));
        const float diff = prev - cur;
        for (int c = 0; c < blends; ++c)
            out[((size_t)c * tokens + t) * hidden + i] = from_f32<AT>(cur + diff * mu[(size_t)c * hidden + i]);
    }
}

// The same for four neighbouring channels a thread and runs of SHIFT_RUN rows, which share their blends' factors:
// 8- and 16-byte accesses, every row read once and its predecessor taken from the row before.  The rows written
// bound it.
// (bfloat16, microseconds, the kernel above first: 2,000 rows of 2,048 in five blends 29.9 and 11.4, 300 of 1,024 7.4 and 5.0)
constexpr int SHIFT_RUN = 4;
template <typename AT>
__global__ void __launch_bounds__(128) token_shift_blend_quads_kernel(const AT* h, const float* __restrict__ mu, const float* state,
                                                                      long long state_stride, const int* seq_of_token,
                                                                      const int* q_start, const int* start_pos,
                                                                      const int* slots, AT* __restrict__ out, int tokens,
                                                                      int hidden, int blends) {
    pdl_begin();
    const int i = (blockIdx.y * 128 + threadIdx.x) * 4;
    if (i >= hidden) return;
    const int t0 = blockIdx.x * SHIFT_RUN;
    float4 cur[SHIFT_RUN], diff[SHIFT_RUN];
    int seq[SHIFT_RUN];
    const float4 before = Quad<AT>::load(h + (size_t)(t0 > 0 ? t0 - 1 : 0) * hidden + i);
#pragma unroll
    for (int r = 0; r < SHIFT_RUN; ++r) {
        const int t = min(t0 + r, tokens - 1);
        cur[r] = Quad<AT>::load(h + (size_t)t * hidden + i);
        seq[r] = seq_of_token[t];
    }
#pragma unroll
    for (int r = 0; r < SHIFT_RUN; ++r) {
        const int t = min(t0 + r, tokens - 1);
        float4 prev = r > 0 ? cur[r - 1] : before;
        if (t == q_start[seq[r]])
            prev = start_pos[seq[r]] == 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f)
                                          : *reinterpret_cast<const float4*>(state + (long long)slots[seq[r]] * state_stride + i);
        diff[r] = make_float4(prev.x - cur[r].x, prev.y - cur[r].y, prev.z - cur[r].z, prev.w - cur[r].w);
    }
    for (int c = 0; c < blends; ++c) {
        const float4 m = *reinterpret_cast<const float4*>(mu + (size_t)c * hidden + i);
#pragma unroll
        for (int r = 0; r < SHIFT_RUN; ++r)
            if (t0 + r < tokens)
                Quad<AT>::store(out + ((size_t)c * tokens + t0 + r) * hidden + i,
                                make_float4(cur[r].x + diff[r].x * m.x, cur[r].y + diff[r].y * m.y, cur[r].z + diff[r].z * m.z, cur[r].w + diff[r].w * m.w));
    }
}

template <typename AT>
__global__ void store_last_row_kernel(const AT* h, float* state, long long state_stride,
                                      const int* q_start, const int* slots, int hidden) {
    pdl_begin();
    const int s = blockIdx.x;
    const int a = q_start[s], e = q_start[s + 1];
    if (e <= a) return;
    float* kept = state + (long long)slots[s] * state_stride;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) kept[i] = to_f32(h[(size_t)(e - 1) * hidden + i]);
}

SHISO_API int shiso_token_shift_blend(const void* h, int act_dtype, const float* mu, float* state, long long state_stride,
                                      const int* seq_of_token, const int* q_start, const int* start_pos, const int* slots,
                                      void* out, int tokens, int num_seqs, int hidden, int blends, cudaStream_t stream) {
    if (tokens <= 0) return SHISO_OK;
    if (act_dtype != SHISO_F32 && act_dtype != SHISO_BF16) return SHISO_ERR_DTYPE;
    auto go = [&](auto zero) {
        typedef decltype(zero) AT;
        const int threads = hidden >= 1024 ? 256 : 128;
        if (hidden % 4 == 0 && state_stride % 4 == 0 && (((uintptr_t)h | (uintptr_t)mu | (uintptr_t)state | (uintptr_t)out) & 15) == 0)
            launch_kernel(token_shift_blend_quads_kernel<AT>, dim3(ceil_div_u(tokens, SHIFT_RUN), ceil_div_u(hidden / 4, 128)), 128, 0, stream, (const AT*)h, mu,
                          (const float*)state, state_stride, seq_of_token, q_start, start_pos, slots, (AT*)out, tokens, hidden, blends);
        else
            launch_kernel(token_shift_blend_kernel<AT>, tokens, threads, 0, stream, (const AT*)h, mu, (const float*)state, state_stride,
                          seq_of_token, q_start, start_pos, slots, (AT*)out, tokens, hidden, blends);
        launch_kernel(store_last_row_kernel<AT>, num_seqs, threads, 0, stream, (const AT*)h, state, state_stride, q_start, slots, hidden);
    };
    if (act_dtype == SHISO_F32) go(0.0f);
    else go(__nv_bfloat16());
    return launch_status();
}

// --------------------------------------------------------------------------- unary maps

enum { SHISO_UNARY_TANH = 0, SHISO_UNARY_SILU = 1, SHISO_UNARY_RELU2 = 2, SHISO_UNARY_COPY = 3 };  // relu2: the square of max(x, 0); copy: the value in the output's type

template <typename IT, typename OT>
__global__ void unary_kernel(const IT* x, OT* __restrict__ out, long long count, int kind) {
    pdl_begin();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
        const float v = to_f32(x[i]);
        float r;
        if (kind == SHISO_UNARY_TANH) r = tanhf(v);
        else if (kind == SHISO_UNARY_SILU) r = v / (1.0f + expf(-v));
        else if (kind == SHISO_UNARY_RELU2) r = v > 0.0f ? v * v : 0.0f;
        else r = v;
        out[i] = from_f32<OT>(r);
    }
}

SHISO_API int shiso_unary(const void* x, int in_dtype, void* out, int out_dtype, long long count, int kind, cudaStream_t stream) {
    if (count <= 0) return SHISO_OK;
    if (kind < SHISO_UNARY_TANH || kind > SHISO_UNARY_COPY) return SHISO_ERR_UNSUPPORTED;
    const unsigned blocks = (unsigned)((count + 255) / 256 < 4096 ? (count + 255) / 256 : 4096);
    if (in_dtype == SHISO_F32 && out_dtype == SHISO_F32)
        launch_kernel(unary_kernel<float, float>, blocks, 256, 0, stream, (const float*)x, (float*)out, count, kind);
    else if (in_dtype == SHISO_F32 && out_dtype == SHISO_BF16)
        launch_kernel(unary_kernel<float, __nv_bfloat16>, blocks, 256, 0, stream, (const float*)x, (__nv_bfloat16*)out, count, kind);
    else if (in_dtype == SHISO_BF16 && out_dtype == SHISO_BF16)
        launch_kernel(unary_kernel<__nv_bfloat16, __nv_bfloat16>, blocks, 256, 0, stream, (const __nv_bfloat16*)x,
                      (__nv_bfloat16*)out, count, kind);
    else if (in_dtype == SHISO_BF16 && out_dtype == SHISO_F32)
        launch_kernel(unary_kernel<__nv_bfloat16, float>, blocks, 256, 0, stream, (const __nv_bfloat16*)x, (float*)out, count, kind);
    else
        return SHISO_ERR_DTYPE;
    return launch_status();
}
