// Y[T, N] = X[T, K] * W[N, K]^T (+ bias) in 32-bit floats on the tensor cores (tcgen05), from products of bfloat16
// pieces.
//
// A float is the sum of three bfloat16 values h + m + l, each what the ones before leave rounded to nearest (the sum is exact: the
// rest behind two such roundings has seven bits; the method is Henry, Tang and Heinecke's, "Leveraging the bfloat16 artificial
// intelligence datatype for higher-precision computations", 2019), and a product of two floats is the sum of nine products of pieces, each exact
// in float.  The six largest are taken - hh, hm, mh, mm, hl, lh.  m is below 2^-8 and l below 2^-17 of its
// float, of either sign, so the others are below 2^-24 of the product together, like the rounding of a multiply-add, and do not
// add up over many products.  (bfloat16 ends at 2^-133, so an operand below 2^-110 keeps that as an absolute error.)  The tensor core
// forms a chunk of 64 columns in 24 instructions, the small products first and hh in the last four; what its own additions lose (they
// cut off, towards zero) is below 2^-21 of the products' magnitudes, and a chunk's sum is then added to a float register by an ordinary
// addition, so that this never grows with K.
//
// Error against 64 bits, 2-norm over that of the result, the multiply-adds of gemm_simple.cu first: operands of either sign 2.1e-7 and 1.0e-7 (300 x
// 1,024 x 1,024), 3.2e-7 and 1.2e-7 (x 1,024 x 4,608), 4.1e-7 and 1.0e-7 (x 9,216 x 1,024), 5.7e-7 and 1.1e-7 (8 x 65,536 x 1,024). Where all products have
// one sign what is cut off does not average out, 8.4e-8 of a result on average whatever the sizes: 2.5e-7 and 1.0e-7 (9,216 x
// 1,024), but 0.8e-7 and 1.0e-7 (1,024 x 1,024), 0.9e-7 and 1.1e-7 (1,024 x 4,608). A result that one product dominates is right to 2^-22, by a multiply-add to 2^-24.
//
// A CTA has 128 rows of W (the MMA's M operand) x NT rows of X and walks one group of K, or all of them:
//   warps 0-7    read the floats of W two chunks ahead (two 16-byte loads for eight columns of a row), split
//                them and store the three pieces where the 128-byte swizzle puts them.  Up to 32 rows of X go the
//                same way; more are split once for all CTAs, by a kernel of its own, and come by TMA.  (With every CTA
//                splitting its rows of X too and one chunk ahead, 2,048 x 9,216 x 1,024 took 570 us, now 449; with the pieces
//                of W in tensor memory, a row of W a thread, 463.)
//   warps 8-15   a thread has one row of W (a lane of tensor memory) and half of the rows of X: adds the
//                chunk's sums to its registers while the tensor core forms the next chunk's (two accumulators)
// and warp 8 also issues the products, a chunk's before it adds the chunk's before (a seventeenth warp would leave 96
// registers a thread instead of 128; issued by a splitting warp, which then splits late, 2,048 x 9,216 x 1,024 took 487 us).
// Where a result is not finite it is formed again as one chain of multiply-adds over its group, so infinities and NaN come out as
// from such a chain.  (An infinity leaves a rest that is NaN, and so does a float that rounds up to one as a bfloat16, above 3.39e38: every
// result that such an operand has a part in is formed again.)
//
// The order of a sum: chunks of 64 columns of a group in their order, groups in their order.  Groups are a
// function of N and K alone, so a row's result depends neither on how many rows share the launch nor on
// where it lies (gemm_simple.cu has the same property, with other bits).
//
// What bounds it: waits. Of the 17 cycles between two instructions of a warp nine go to loads and three to barriers, the schedulers issue in a
// sixth of all cycles and the tensor core works in a quarter of the active ones (300 x 9,216 x 1,024; profiles/float_products.md);
// that shape's 216 CTAs are one and a half for every SM.
//
// Measured, microseconds, gemm_simple.cu's first (rows x N x K): 1 x 9,216 x 1,024 34 and 15, 8 x 65,536 x 1,024 133 and 105, 1 x 1,024 x 4,608
// 17 and 13, 24 x 9,216 x 1,024 68 and 16, 64 x 1,024 x 4,608 38 and 17, 300 x 9,216 x 1,024 171 and 110, 300 x 1,024 x 4,608 81 and 51, 300 x 1,024
// x 1,024 26 and 23, 2,048 x 9,216 x 1,024 861 and 457.  (With pieces that were cut off instead of rounded 300 x 9,216 x 1,024 took 109, 2,048 rows 449.)
//
// Every wait is bounded by a clock limit and reports through the status word.
#include <type_traits>

#include "tcgen05.cuh"

namespace {

using namespace tc;

constexpr int TILE_N = 128;                     // rows of W
constexpr int SPLITTERS = 8, ADDERS = 8;        // warps
constexpr int THREADS = (SPLITTERS + ADDERS) * 32;
constexpr int ROW = 128;                        // bytes of a piece's row: 64 bfloat16
constexpr int W_PIECE = TILE_N * ROW;
constexpr int DIRECT_ROWS = 32;                 // rows of X that every CTA splits for itself

struct FloatArgs {
    const float *x, *w, *bias;
    int x_rows;      // PIECES: rows of a piece of X in the workspace [3][x_rows][K]
    float* y;        // ALL: the result
    float* partial;  // else: [groups, T, N]
    int* status;
    int T, N, K, group;
};

// Eight neighbouring floats as three words of eight bfloat16 each.
__device__ __forceinline__ void split8(const float4& a, const float4& b, uint4 (&out)[3]) {
    float rest[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint32_t* o = reinterpret_cast<uint32_t*>(&out[p]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 pair = __floats2bfloat162_rn(rest[2 * i], rest[2 * i + 1]);
            o[i] = *reinterpret_cast<const uint32_t*>(&pair);
            rest[2 * i] -= __uint_as_float(o[i] << 16);
            rest[2 * i + 1] -= __uint_as_float(o[i] & 0xffff0000u);
        }
    }
}

// The chain that stands in for a result that is not finite.
__device__ __forceinline__ float plain_sum(const float* x, const float* w, int k_begin, int k_end) {
    float sum = 0.0f;
#pragma unroll 1
    for (int k = k_begin; k < k_end; ++k) sum = fmaf(x[k], w[k], sum);
    return sum;
}

// X as its three pieces, one behind the other (a multiple of eight floats).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* x, __nv_bfloat16* pieces, long long count) {
    pdl_begin();
    const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) * 8;
    if (at >= count) return;
    uint4 out[3];
    split8(*(const float4*)(x + at), *(const float4*)(x + at + 4), out);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(pieces + p * count + at) = out[p];
}

template <int NT, bool ALL>
__global__ void __launch_bounds__(THREADS, 1) gemm_float_tc_kernel(const __grid_constant__ CUtensorMap map_x, const FloatArgs a) {
    constexpr int X_PIECE = NT * ROW, STAGE_BYTES = 3 * (W_PIECE + X_PIECE), STAGES = NT > 64 ? 2 : 3;
    constexpr bool PIECES = NT > DIRECT_ROWS;                                    // X comes in pieces already
    constexpr int COLS = NT / 2;                                          // rows of X an adding thread has
    constexpr int TMEM_COLS = 2 * NT < 32 ? 32 : 2 * NT;
    constexpr int W_UNITS = TILE_N * 8 / (SPLITTERS * 32);                // eight-column units of a chunk a splitting thread has
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;  // [2]
    uint64_t* acc_empty = acc_full + 2;   // [2]
    uint64_t* products_done = acc_empty + 2;  // nothing of this CTA is left in the tensor core
    uint32_t* tmem_slot = (uint32_t*)(products_done + 1);
    int* failed = (int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * TILE_N, t0 = blockIdx.y * NT;
    const int k_begin = ALL ? 0 : blockIdx.z * a.group, k_end = ALL ? a.K : min(a.K, k_begin + a.group);
    const int chunks = (k_end - k_begin + 63) / 64;
    const int per_group = a.group / 64;  // chunks (a group is a multiple of 64 columns)

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], PIECES ? SPLITTERS + 1 : SPLITTERS);  // (and the bytes of X)
            mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], ADDERS);
        }
        mbar_init(products_done, 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // splitting warps: unit u of a chunk is columns 8 (u % 8) .. + 7 of row u / 8
    typedef std::integral_constant<int, 0> Even;
    typedef std::integral_constant<int, 1> Odd;
    const int row0 = threadIdx.x >> 3, piece = threadIdx.x & 7;
    const bool has_x = !PIECES && row0 < NT;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 wr[2][W_UNITS][2], xr[2][2];  // [chunk parity]
    auto load_w = [&](int c, auto parity) {
        const int k = k_begin + c * 64 + piece * 8;
#pragma unroll
        for (int i = 0; i < W_UNITS; ++i) {
            const int n = n0 + row0 + 32 * i;
            const float* p = a.w + (size_t)n * a.K + k;
            wr[parity][i][0] = n < a.N && k < k_end ? __ldg((const float4*)p) : zero;
            wr[parity][i][1] = n < a.N && k + 4 < k_end ? __ldg((const float4*)p + 1) : zero;
        }
    };
    auto load_x = [&](int c, auto parity) {
        const int k = k_begin + c * 64 + piece * 8, t = t0 + row0;
        const float* p = a.x + (size_t)t * a.K + k;
        xr[parity][0] = has_x && t < a.T && k < k_end ? *(const float4*)p : zero;
        xr[parity][1] = has_x && t < a.T && k + 4 < k_end ? *((const float4*)p + 1) : zero;
    };
    if (warp < SPLITTERS) {
        load_w(0, Even());  // (weights are no predecessor's output)
        if (chunks > 1) load_w(1, Odd());
    }
    pdl_wait();
    if (warp < SPLITTERS && !PIECES) {
        load_x(0, Even());
        if (chunks > 1) load_x(1, Odd());
    }
    // (behind the wait: no CTA holds tensor memory, or waits for it, while another grid's CTAs still work with theirs)
    if (warp == SPLITTERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp < SPLITTERS) {
        auto work = [&](int c, auto parity) {
            const int s = c % STAGES;
            if (c >= STAGES && !mbar_wait(&empty[s], ((c / STAGES) - 1) & 1)) *failed = 1;
            uint8_t* ws = smem + s * STAGE_BYTES;
            uint8_t* xs = ws + 3 * W_PIECE;
            if (PIECES && threadIdx.x == 0) {
                mbar_expect_tx(&full[s], 3 * X_PIECE);
                for (int p = 0; p < 3; ++p) tma_load_2d(xs + p * X_PIECE, &map_x, k_begin + c * 64, p * a.x_rows + t0, &full[s]);
            }
#pragma unroll
            for (int i = 0; i < W_UNITS; ++i) {
                const int r = row0 + 32 * i;
                uint4 pieces[3];
                split8(wr[parity][i][0], wr[parity][i][1], pieces);
#pragma unroll
                for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(ws + p * W_PIECE + r * ROW + ((piece ^ (r & 7)) << 4)) = pieces[p];
            }
            if (c + 2 < chunks) load_w(c + 2, parity);
            if (has_x) {
                uint4 pieces[3];
                split8(xr[parity][0], xr[parity][1], pieces);
#pragma unroll
                for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(xs + p * X_PIECE + row0 * ROW + ((piece ^ (row0 & 7)) << 4)) = pieces[p];
                if (c + 2 < chunks) load_x(c + 2, parity);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // written by threads, read by the MMA
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        };
        int worked = 0;
        for (int c = 0; c < chunks; c += 2) {
            if (__any_sync(0xffffffffu, *(volatile int*)failed)) break;  // (a wait ran out: no further one is begun)
            work(c, Even());
            if (c + 1 < chunks) work(c + 1, Odd());
            worked = min(chunks, c + 2);
        }
        if (PIECES && threadIdx.x == 0)  // the shared memory is not given back before the last copies into it have landed
            for (int c = max(0, worked - STAGES); c < worked; ++c)
                if (!mbar_wait(&full[c % STAGES], (c / STAGES) & 1)) {
                    *failed = 1;
                    break;
                }
    } else {
        // ---- adders: row n of W, rows t .. t + COLS - 1 of X
        const uint32_t idesc = umma_idesc(TILE_N, NT);
        auto issue = [&](int c) {  // chunk c's products
            const int s = c % STAGES, acc = c & 1;
            if (c >= 2 && !mbar_wait(&acc_empty[acc], ((c >> 1) - 1) & 1)) *failed = 1;
            if (!mbar_wait(&full[s], (c / STAGES) & 1)) *failed = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t w_addr = smem_u32(smem + s * STAGE_BYTES);
            const uint64_t dw = umma_desc(w_addr), dx = umma_desc(w_addr + 3 * W_PIECE);  // (an address counts in units of 16 bytes)
            constexpr int PW[6] = {2, 0, 1, 1, 0, 0}, PX[6] = {0, 2, 1, 0, 1, 0};  // lh, hl, mm, mh, hm, hh
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int k = 0; k < 64 / UMMA_K; ++k)
                    umma_bf16(tmem_base + acc * NT, dw + ((PW[p] * W_PIECE + k * UMMA_K * 2) >> 4), dx + ((PX[p] * X_PIECE + k * UMMA_K * 2) >> 4),
                              idesc, (p > 0 || k > 0) ? 1u : 0u);
            umma_commit(&empty[s]);
            umma_commit(&acc_full[acc]);
        };
        const int q = warp & 3, half = (warp - SPLITTERS) >> 2;
        const int n = n0 + q * 32 + lane, t = t0 + half * COLS;
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + half * COLS;
        const bool live = n < a.N;
        float sum[COLS];
        bool fresh = true;  // the next chunk is a group's first
        for (int c = 0; c < chunks; ++c) {
            if (__any_sync(0xffffffffu, *(volatile int*)failed)) break;
            if (warp == SPLITTERS) {
                if (lane == 0) {
                    if (c == 0) issue(0);
                    if (c + 1 < chunks) issue(c + 1);
                }
                __syncwarp();
            }
            const int acc = c & 1;
            if (!mbar_wait(&acc_full[acc], (c >> 1) & 1)) {
                *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            constexpr int STEP = COLS < 16 ? 8 : 16;
#pragma unroll
            for (int j = 0; j < COLS; j += STEP) {
                float v[STEP];
                if constexpr (STEP == 8) tmem_ld8(taddr + acc * NT + j, v);
                else tmem_ld16(taddr + acc * NT + j, v);
#pragma unroll
                for (int e = 0; e < STEP; ++e) sum[j + e] = fresh ? v[e] : sum[j + e] + v[e];
            }
            fresh = false;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
            const bool last = c + 1 == chunks, group_ends = last || (ALL && (c + 1) % per_group == 0);
            if (!group_ends) continue;
            // a group's sums: on their own, or joined to those of the groups before in the result
            const int g = ALL ? c / per_group : blockIdx.z;
            const int from = g * a.group, to = min(a.K, from + a.group);
            float* out = ALL ? a.y : a.partial + (size_t)g * a.T * a.N;
            const float b = ALL && last && a.bias && live ? a.bias[n] : 0.0f;
            unsigned long long odd = 0;  // results that are not finite
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                if (!live || t + j >= a.T) continue;
                float* at = out + (size_t)(t + j) * a.N + n;
                if (fabsf(sum[j]) < INFINITY) *at = ALL && g > 0 ? *at + sum[j] + b : sum[j] + b;
                else odd |= 1ull << j;
            }
#pragma unroll 1
            for (int j = 0; odd; ++j, odd >>= 1) {
                if (!(odd & 1)) continue;
                float* at = out + (size_t)(t + j) * a.N + n;
                const float v = plain_sum(a.x + (size_t)(t + j) * a.K, a.w + (size_t)n * a.K, from, to);
                *at = ALL && g > 0 ? *at + v + b : v + b;
            }
            fresh = true;
        }
        if (threadIdx.x == SPLITTERS * 32) {
            umma_commit(products_done);
            if (!mbar_wait(products_done, 0)) *failed = 1;
        }
    }
    pdl_trigger();
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*failed != 0 && threadIdx.x == 0 && a.status) atomicExch(a.status, 1);
    if (warp == SPLITTERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// y = the groups' sums in their order (+ bias).
__global__ void __launch_bounds__(256) float_join_kernel(const float* partial, const float* __restrict__ bias, float* y, long long count, int N, int groups) {
    pdl_begin();
    const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    if (at >= count) return;
    if (count % 4 == 0) {
        float4 v = *(const float4*)(partial + at);
#pragma unroll 8
        for (int g = 1; g < groups; ++g) {
            const float4 q = *(const float4*)(partial + (size_t)g * count + at);
            v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
        }
        if (bias) v.x += bias[at % N], v.y += bias[(at + 1) % N], v.z += bias[(at + 2) % N], v.w += bias[(at + 3) % N];
        *(float4*)(y + at) = v;
    } else {
        for (int e = 0; e < 4 && at + e < count; ++e) {
            float v = partial[at + e];
            for (int g = 1; g < groups; ++g) v += partial[(size_t)g * count + at + e];
            y[at + e] = bias ? v + bias[(at + e) % N] : v;
        }
    }
}

template <int NT>
int launch_float_tc(const FloatArgs& a, int groups, __nv_bfloat16* pieces, cudaStream_t stream) {
    constexpr int STAGES = NT > 64 ? 2 : 3;
    constexpr int SMEM = STAGES * 3 * (W_PIECE + NT * ROW) + 1024 + 256;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_float_tc_kernel<NT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_float_tc_kernel<NT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    CUtensorMap map = {};
    if (NT > DIRECT_ROWS) {
        if (!tc::tensor_map(pieces, 3 * a.x_rows, a.K, NT, &map)) return SHISO_ERR_UNSUPPORTED;
        const long long count = (long long)a.T * a.K;
        launch_kernel(split_rows_kernel, ceil_div_u(count, 2048), 256, 0, stream, a.x, pieces, count);
        const int status = launch_status();
        if (status != SHISO_OK) return status;
    }
    const dim3 grid(ceil_div_u(a.N, TILE_N), ceil_div_u(a.T, NT), groups > 1 ? groups : 1);
    if (groups <= 1) {
        launch_kernel(gemm_float_tc_kernel<NT, true>, grid, THREADS, SMEM, stream, map, a);
        return launch_status();
    }
    launch_kernel(gemm_float_tc_kernel<NT, false>, grid, THREADS, SMEM, stream, map, a);
    const int status = launch_status();
    if (status != SHISO_OK) return status;
    const long long count = (long long)a.T * a.N;
    launch_kernel(float_join_kernel, ceil_div_u(count, 1024), 256, 0, stream, (const float*)a.partial, a.bias, a.y, count, a.N, groups);
    return launch_status();
}

}  // namespace

// Whether the kernel takes the product: rows of whole 16-byte words, in pieces too, on 16-byte boundaries, matrices of at
// least half a tile and four chunks (below that a chain has few roundings; others stay with gemm_simple.cu; the line is a function of N and K, as the bits are).
SHISO_API int shiso_gemm_float_tc_supported(const void* x, const void* w, const void* y, int T, int N, int K) {
    return T > 0 && T <= 65535 * 16 && N >= 64 && K >= 256 && K % 8 == 0 && (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) == 0 &&
           tc::encode_fn() != nullptr;
}

// How many rows of X go without a workspace for their pieces.
SHISO_API int shiso_gemm_float_tc_direct_rows() { return DIRECT_ROWS; }

// `group`: columns of a group of K (rounded up to a multiple of 64 here); `partial`: room for ceil(K / group) x T x N
// floats, groups then have CTAs of their own, or null: one CTA walks all of them.  Neither changes a bit.
// `pieces`: room for 3 x T x K bfloat16 where T exceeds the direct rows.
SHISO_API int shiso_gemm_float_tc(const void* x, const void* w, const float* bias, void* y, void* partial, void* pieces, int T, int N, int K,
                                  int group, cudaStream_t stream) {
    if (T <= 0 || N <= 0) return SHISO_OK;
    if (group <= 0 || (T > DIRECT_ROWS && !pieces)) return SHISO_ERR_SHAPE;
    if (!shiso_gemm_float_tc_supported(x, w, y, T, N, K)) return SHISO_ERR_UNSUPPORTED;
    if (((uintptr_t)partial | (uintptr_t)pieces) & 15) return SHISO_ERR_ALIGN;
    group = (group + 63) / 64 * 64;
    const int groups = partial ? (K + group - 1) / group : 1;
    FloatArgs a = {(const float*)x, (const float*)w, bias, T, (float*)y, (float*)partial, shiso_tc_status_word(), T, N, K, group};
    __nv_bfloat16* room = (__nv_bfloat16*)pieces;
    if (T <= 16) return launch_float_tc<16>(a, groups, room, stream);
    if (T <= DIRECT_ROWS) return launch_float_tc<32>(a, groups, room, stream);
    if (T <= 64) return launch_float_tc<64>(a, groups, room, stream);
    return launch_float_tc<128>(a, groups, room, stream);
}
