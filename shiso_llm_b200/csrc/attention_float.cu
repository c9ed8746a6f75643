// Paged attention of prompt portions in true 32-bit floats: tiles of query rows that share their keys.
//
// The general kernel (attention.cu) has a warp per (row, head) whose lanes each read a key row of their
// own, 256 bytes apart: every load is 32 sectors, every row reads all its keys again, and 300 rows of 16
// heads of 64 took 286 us for what is 0.2 GFLOP.  Here a CTA takes 32 query rows of one sequence and one head;
// tiles of 32 keys and their values come to shared memory once (16-byte cp.async through the block table, two
// stages), a thread has 2 rows x 4 keys of the scores and then 4 rows x HEAD / 16 columns of the output.
//
// Every result has the general kernel's bits: a score is one chain over the channels, keys are folded in
// groups of 32 counted from the sequence's start, a group's weights are summed as the warp's butterfly sums them (i and
// i + 16, + 8, + 4, + 2, + 1), and an output is one chain over the keys in their order.  So which of the two
// runs, and how a prompt was cut, changes no bit of a row.
//
// What bounds it: the multiply-add chains of the few warps an SM has (a portion of 300 rows is 160 CTAs).
//
// Measured beside the general kernel, microseconds: 300 rows of 16 heads of 64 286 and 32; 24 rows 13 and 6; 2 rows at 500
// 220 and 49; 100 rows beside three single ones, up to 2,000 keys, 889 and 186; 256 rows of 16 heads of 128 at 300 1,008 and 99.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int ROWS = 32, KEYS = 32, THREADS = 128;

struct FloatAttentionArgs {
    const float *q, *k_cache, *v_cache;
    const int *block_table, *q_start, *start_pos;
    float* out;
    int table_width, num_seqs, heads, kv_heads, page_size;
    float scale;
};

__device__ __forceinline__ void cp16(float* dst, const float* src, bool valid) {
    const int bytes = valid ? 16 : 0;  // the rest of the 16 becomes zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

template <int HEAD>
struct FloatTiles {
    static constexpr int STRIDE = HEAD + 4;  // floats of a padded row: eight rows' 16-byte reads meet all banks once
    float q[ROWS][STRIDE];
    float k[2][KEYS][STRIDE], v[2][KEYS][STRIDE];
    float p[KEYS][ROWS + 4];     // a group's weights, key by key
    float correction[ROWS], total[ROWS];
};

template <int HEAD>
__global__ void __launch_bounds__(THREADS) float_prefill_kernel(const FloatAttentionArgs a) {
    extern __shared__ __align__(16) uint8_t raw[];
    FloatTiles<HEAD>& s = *reinterpret_cast<FloatTiles<HEAD>*>(raw);
    constexpr int PIECES = HEAD / 4, COLS = HEAD / 16;  // COLS: output columns of a thread
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    // the last tiles of a portion have the most keys: they take the first CTAs of every head
    int left = gridDim.y - 1 - blockIdx.y, seq = 0, len = 0;
    for (; seq < a.num_seqs; ++seq) {
        len = a.q_start[seq + 1] - a.q_start[seq];
        const int tiles = (len + ROWS - 1) / ROWS;
        if (left < tiles) break;
        left -= tiles;
    }
    if (seq == a.num_seqs) return;
    const int first_token = a.q_start[seq] + left * ROWS, rows = min(ROWS, len - left * ROWS);
    const int first_pos = a.start_pos[seq] + left * ROWS, last_pos = first_pos + rows - 1;
    const int head = blockIdx.x, kv_head = head / (a.heads / a.kv_heads);
    const int* table = a.block_table + (size_t)seq * a.table_width;

    for (int c = tid; c < ROWS * PIECES; c += THREADS) {
        const int r = c / PIECES, piece = c % PIECES;
        const bool valid = r < rows;
        cp16(&s.q[r][piece * 4], a.q + ((size_t)(first_token + (valid ? r : 0)) * a.heads + head) * HEAD + piece * 4, valid);
    }
    auto load = [&](int g, int stage) {
        for (int c = tid; c < KEYS * PIECES; c += THREADS) {
            const int r = c / PIECES, piece = c % PIECES, key = g * KEYS + r;
            const bool valid = key <= last_pos;
            size_t row = 0;
            if (valid) row = (size_t)table[key / a.page_size] * a.page_size + key % a.page_size;
            const size_t at = (row * a.kv_heads + kv_head) * HEAD + piece * 4;
            cp16(&s.k[stage][r][piece * 4], a.k_cache + at, valid);
            cp16(&s.v[stage][r][piece * 4], a.v_cache + at, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, 0);

    const int tx = lane & 7, ty = warp * 4 + (lane >> 3);  // scores: rows 2 ty, 2 ty + 1, keys tx + 8 j
    const int ox = tid & 15, oy = tid >> 4;                // output: rows 4 oy .. + 3, columns 4 ox .. + 3 (+ 64)
    float run_max[2] = {-INFINITY, -INFINITY}, run_sum[2] = {0.0f, 0.0f};
    float acc[4][COLS];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[i][c] = 0.0f;
    const int groups = last_pos / KEYS + 1;
    for (int g = 0; g < groups; ++g) {
        const int stage = g & 1;
        if (g + 1 < groups) load(g + 1, stage ^ 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float dot[2][4] = {};
#pragma unroll 4
        for (int d = 0; d < HEAD; d += 4) {
            float4 q4[2], k4[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) q4[i] = *reinterpret_cast<const float4*>(&s.q[2 * ty + i][d]);
#pragma unroll
            for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(&s.k[stage][tx + 8 * j][d]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    dot[i][j] = fmaf(q4[i].x, k4[j].x, dot[i][j]);
                    dot[i][j] = fmaf(q4[i].y, k4[j].y, dot[i][j]);
                    dot[i][j] = fmaf(q4[i].z, k4[j].z, dot[i][j]);
                    dot[i][j] = fmaf(q4[i].w, k4[j].w, dot[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int pos = first_pos + 2 * ty + i;
            float m = -INFINITY, w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                dot[i][j] = g * KEYS + tx + 8 * j <= pos ? __fmul_rn(dot[i][j], a.scale) : -INFINITY;
                m = fmaxf(m, dot[i][j]);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            // (a group behind a row's last key leaves the row as it is: its weights are zero and its correction one)
            const float new_max = fmaxf(run_max[i], m);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                w[j] = g * KEYS + tx + 8 * j <= pos ? expf(dot[i][j] - new_max) : 0.0f;
                s.p[tx + 8 * j][2 * ty + i] = w[j];
            }
            float sum = (w[0] + w[2]) + (w[1] + w[3]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float correction = expf(run_max[i] - new_max);  // exp(-inf) = 0 on the first group
            run_sum[i] = run_sum[i] * correction + sum;
            run_max[i] = new_max;
            if (tx == 0) s.correction[2 * ty + i] = correction;
        }
        __syncthreads();
        {
            const float4 c4 = *reinterpret_cast<const float4*>(&s.correction[4 * oy]);
            const float c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < COLS; ++e) acc[i][e] *= c[i];
        }
        // (where some row does not see a key, that row does not add it at all: the value may be anything)
        auto values = [&](int count, auto masked) {
#pragma unroll 4
            for (int key = 0; key < count; ++key) {
                const float4 p4 = *reinterpret_cast<const float4*>(&s.p[key][4 * oy]);
                const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                for (int h = 0; h < COLS / 4; ++h) {
                    const float4 v4 = *reinterpret_cast<const float4*>(&s.v[stage][key][64 * h + 4 * ox]);
                    const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (!decltype(masked)::value || g * KEYS + key <= first_pos + 4 * oy + i) acc[i][4 * h + e] = fmaf(p[i], v[e], acc[i][4 * h + e]);
                }
            }
        };
        if (g * KEYS + KEYS - 1 <= first_pos) values(KEYS, std::false_type());
        else values(min(KEYS, last_pos - g * KEYS + 1), std::true_type());
        __syncthreads();  // the stage and the weights are written anew by the next group
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (tx == 0) s.total[2 * ty + i] = run_sum[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * oy + i;
        if (r >= rows) continue;
        const float inv = s.total[r] > 0.0f ? 1.0f / s.total[r] : 0.0f;
#pragma unroll
        for (int h = 0; h < COLS / 4; ++h)
            *reinterpret_cast<float4*>(a.out + ((size_t)(first_token + r) * a.heads + head) * HEAD + 64 * h + 4 * ox) =
                make_float4(acc[i][4 * h] * inv, acc[i][4 * h + 1] * inv, acc[i][4 * h + 2] * inv, acc[i][4 * h + 3] * inv);
    }
}

template <int HEAD>
int launch_float_prefill(const FloatAttentionArgs& a, int tiles, cudaStream_t stream) {
    const size_t smem = sizeof(FloatTiles<HEAD>);
    auto kernel = float_prefill_kernel<HEAD>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    launch_kernel(kernel, dim3(a.heads, tiles), THREADS, smem, stream, a);
    return launch_status();
}

}  // namespace

// Whether the kernel takes these: head sizes of 64 and 128, everything on 16-byte boundaries.
SHISO_API int shiso_float_prefill_supported(const void* q, const void* k_cache, const void* v_cache, const void* out, int head_dim) {
    return (head_dim == 64 || head_dim == 128) && (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) == 0;
}

// q and out [T, heads * head_dim], caches [pages, page_size, kv_heads, head_dim], all float; no window; `tiles`: an
// upper bound of the 32-row tiles over all sequences.
SHISO_API int shiso_float_prefill(const void* q, const void* k_cache, const void* v_cache, const int* block_table, int table_width,
                                  const int* q_start, const int* start_pos, void* out, int num_seqs, int tiles, int heads, int kv_heads,
                                  int head_dim, int page_size, float scale, cudaStream_t stream) {
    if (num_seqs <= 0 || tiles <= 0) return SHISO_OK;
    if (kv_heads <= 0 || heads % kv_heads || page_size <= 0 || tiles > 65535) return SHISO_ERR_SHAPE;
    if (!shiso_float_prefill_supported(q, k_cache, v_cache, out, head_dim)) return SHISO_ERR_UNSUPPORTED;
    FloatAttentionArgs a = {(const float*)q, (const float*)k_cache, (const float*)v_cache, block_table, q_start, start_pos, (float*)out,
                            table_width, num_seqs, heads, kv_heads, page_size, scale};
    return head_dim == 64 ? launch_float_prefill<64>(a, tiles, stream) : launch_float_prefill<128>(a, tiles, stream);
}
