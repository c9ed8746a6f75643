// Y[T, N] = X[T, K] * W[N, K]^T (+ bias) with float accumulation on the CUDA cores.
//
// gemm_float_kernel is the matrix product of the true 32-bit path where K is a multiple of four and
// the operands lie on 16-byte boundaries.  gemm_simple_kernel is the float product otherwise, and the product
// for any combination of element types the tensor-core kernels do not take (a matrix kept in 32-bit
// beside 16-bit activations); T, N, K >= 1.
//
// Sums are fused multiply-adds over k in ascending order: gemm_simple_kernel's over k = 0 .. K-1,
// gemm_float_kernel's within groups of K whose sums are then added up in their order.  The groups are a
// function of N and K, so with either kernel a row's result depends neither on how many rows share the
// launch nor on where the row lies in it - the property the reference calls row-exact
// (crates/shiso-engine/src/projection.rs:972-978).
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename WT, typename XT, typename OT>
__global__ void __launch_bounds__(256)
gemm_simple_kernel(const XT* x, const WT* __restrict__ w, const float* __restrict__ bias,
                   OT* __restrict__ y, int T, int N, int K) {
    pdl_wait();
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int ty = tid / (BN / TN), tx = tid % (BN / TN);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = tid; e < BM * BK; e += 256) {
            const int r = e / BK, c = e % BK;
            const int gr = row0 + r, gk = k0 + c;
            xs[c][r] = (gr < T && gk < K) ? to_f32(x[(size_t)gr * K + gk]) : 0.0f;
        }
#pragma unroll
        for (int e = tid; e < BN * BK; e += 256) {
            const int r = e / BK, c = e % BK;
            const int gn = col0 + r, gk = k0 + c;
            ws[c][r] = (gn < N && gk < K) ? to_f32(w[(size_t)gn * K + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gr = row0 + ty * TM + i;
        if (gr >= T) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = col0 + tx * TN + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[gn];
            y[(size_t)gr * N + gn] = from_f32<OT>(v);
        }
    }
}

template <typename WT, typename XT, typename OT>
int launch(const void* x, const void* w, const float* bias, void* y, int T, int N, int K, cudaStream_t stream) {
    dim3 grid(ceil_div_u(N, BN), ceil_div_u(T, BM));
    launch_kernel(gemm_simple_kernel<WT, XT, OT>, grid, 256, 0, stream, (const XT*)x, (const WT*)w, bias, (OT*)y, T, N, K);
    return launch_status();
}

// ---- all float, rows of four values on 16-byte boundaries: the products of the true 32-bit path ----
// The kernel above reads four bytes a lane, waits for every tile's loads, and gives a matrix of 1,024
// rows 80 CTAs at 300 tokens (10 TFLOP/s).  Here a thread has 8 x 8 (4 x 8, 1 x 8) outputs as pairs for
// the packed multiply-adds (fma.rn.f32x2: both halves are the products and sums of fmaf), the next 16
// columns are on their way while these are worked on, and K is cut into groups so that few tiles still
// fill the chip.  What bounds it: the multiply-add pipe, 32 packed instructions beside 4 16-byte reads of
// shared memory for a column of a thread's 8 x 8 outputs.
//
// The order of a sum: k ascending within a group of K, the groups' sums added in their order.  The
// groups are a function of N and K alone, so a row's result still depends neither on how many rows share
// the launch nor on where it lies, whichever tile height runs and whether one CTA walks all groups (many
// tiles) or each group has CTAs of its own, whose sums a second kernel adds up (few tiles).
constexpr int PN = 128, PK = 16, P_THREADS = 128;

// TM: rows of x a thread has; a CTA has 8 TM.  ALL: the CTA walks every group of K (grid.z = 1), else
// group blockIdx.z, whose sums go to partial[blockIdx.z][T][N].
template <int TM, bool ALL>
__global__ void __launch_bounds__(P_THREADS, TM == 8 ? 2 : 4)
gemm_float_kernel(const float* x, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ y,
                  float* __restrict__ partial, int T, int N, int K, int group) {
    constexpr int PM = 8 * TM, XROW = PM + 4, WROW = PN + 4;
    __shared__ __align__(16) float xs[2][PK][XROW], ws[2][PK][WROW];
    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * PM, col0 = blockIdx.x * PN;
    const int tx = tid % 16, ty = tid / 16;
    // what a thread copies: four columns (from 4 (tid % 4)) of rows tid / 4, + 32, ...
    const int copy_k = (tid % 4) * 4, copy_row = tid / 4;
    constexpr int XC = PM >= 32 ? PM / 32 : 1, WC = PN / 32;
    const bool copies_x = copy_row < PM;
    const int k_begin = ALL ? 0 : blockIdx.z * group, k_end = ALL ? K : min(K, k_begin + group);
    float4 xr[XC], wr[WC];
    auto load_w = [&](int k0) {
        const int k = k0 + copy_k;
#pragma unroll
        for (int c = 0; c < WC; ++c) {
            const int n = col0 + copy_row + 32 * c;
            wr[c] = (n < N && k < k_end) ? __ldg((const float4*)(w + (size_t)n * K + k)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto load_x = [&](int k0) {
        const int k = k0 + copy_k;
#pragma unroll
        for (int c = 0; c < XC; ++c) {
            const int t = row0 + copy_row + 32 * c;
            xr[c] = (copies_x && t < T && k < k_end) ? *(const float4*)(x + (size_t)t * K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto put = [&](int s) {
#pragma unroll
        for (int c = 0; c < WC; ++c) {
            float* to = &ws[s][copy_k][copy_row + 32 * c];
            to[0] = wr[c].x; to[WROW] = wr[c].y; to[2 * WROW] = wr[c].z; to[3 * WROW] = wr[c].w;
        }
        if (copies_x) {
#pragma unroll
            for (int c = 0; c < XC; ++c) {
                float* to = &xs[s][copy_k][copy_row + 32 * c];
                to[0] = xr[c].x; to[XROW] = xr[c].y; to[2 * XROW] = xr[c].z; to[3 * XROW] = xr[c].w;
            }
        }
    };
    // a thread's rows: 4 ty .. + 3 of every 32 of the tile (TM = 1: row ty); its columns: 4 tx .. + 3 of either half
    f32x2 acc[TM][4], total[ALL ? TM : 1][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0ull;
            if (ALL) total[i][j] = 0ull;
        }
    load_w(k_begin);  // (weights are no predecessor's output)
    pdl_wait();
    load_x(k_begin);
    put(0);
    __syncthreads();
    int s = 0, left = group;  // columns left of this group (a multiple of PK)
    for (int k0 = k_begin; k0 < k_end; k0 += PK) {
        const bool more = k0 + PK < k_end;
        if (more) {
            load_w(k0 + PK);
            load_x(k0 + PK);
        }
#pragma unroll
        for (int k = 0; k < PK; ++k) {
            float a[TM];
            if constexpr (TM == 1) {
                a[0] = xs[s][k][ty];
            } else {
#pragma unroll
                for (int h = 0; h < TM / 4; ++h) {
                    const float4 a4 = *(const float4*)&xs[s][k][32 * h + 4 * ty];
                    a[4 * h] = a4.x; a[4 * h + 1] = a4.y; a[4 * h + 2] = a4.z; a[4 * h + 3] = a4.w;
                }
            }
            const ulonglong2 b0 = *(const ulonglong2*)&ws[s][k][4 * tx], b1 = *(const ulonglong2*)&ws[s][k][PN / 2 + 4 * tx];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const f32x2 ai = pair_of(a[i], a[i]);
                acc[i][0] = fma2(ai, b0.x, acc[i][0]);
                acc[i][1] = fma2(ai, b0.y, acc[i][1]);
                acc[i][2] = fma2(ai, b1.x, acc[i][2]);
                acc[i][3] = fma2(ai, b1.y, acc[i][3]);
            }
        }
        if (more) put(s ^ 1);
        s ^= 1;
        if (ALL) {
            left -= PK;
            if (left == 0 || !more) {
                left = group;
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        total[i][j] = add2(total[i][j], acc[i][j]);
                        acc[i][j] = 0ull;
                    }
            }
        }
        __syncthreads();
    }
    pdl_trigger();
    float* to = ALL ? y : partial + (size_t)blockIdx.z * T * N;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int t = row0 + (TM == 1 ? ty : (i / 4) * 32 + 4 * ty + i % 4);
        if (t >= T) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = col0 + h * (PN / 2) + 4 * tx;
            float v[4];
            halves(ALL ? total[ALL ? i : 0][2 * h] : acc[i][2 * h], v[0], v[1]);
            halves(ALL ? total[ALL ? i : 0][2 * h + 1] : acc[i][2 * h + 1], v[2], v[3]);
            if (ALL && bias) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < N) v[e] += bias[n + e];
            }
            if (n + 3 < N && N % 4 == 0) {
                *(float4*)(to + (size_t)t * N + n) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < N) to[(size_t)t * N + n + e] = v[e];
            }
        }
    }
}

// y = the groups' sums in their order (+ bias).
__global__ void __launch_bounds__(256) gemm_float_join_kernel(const float* partial, const float* __restrict__ bias,
                                                              float* __restrict__ y, long long count, int N, int groups) {
    pdl_begin();
    const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    if (at >= count) return;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (count % 4 == 0) {
#pragma unroll 8
        for (int g = 0; g < groups; ++g) {
            const float4 q = *(const float4*)(partial + (size_t)g * count + at);
            v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
        }
    } else {
        for (int g = 0; g < groups; ++g)
            for (int e = 0; e < 4 && at + e < count; ++e) v[e] += partial[(size_t)g * count + at + e];
    }
    for (int e = 0; e < 4 && at + e < count; ++e) y[at + e] = bias ? v[e] + bias[(at + e) % N] : v[e];
}

// The columns of K in a group: as many groups as give a single tile of tokens about GROUP_CTAS CTAs, of at
// least GROUP_MIN columns each.  (Both fix the order of every sum: they are no device's SM count, and N and K
// are all that may be asked for.)
constexpr int GROUP_CTAS = 128, GROUP_MIN = 128;
int group_size(int N, int K) {
    const int tiles = (N + PN - 1) / PN;
    int groups = (GROUP_CTAS + tiles - 1) / tiles;
    if (groups > K / GROUP_MIN) groups = K / GROUP_MIN;
    if (groups < 1) groups = 1;
    return ((K + groups - 1) / groups + PK - 1) / PK * PK;
}

bool float_takes(const void* x, const void* w, const void* y, int T, int K) {
    return K % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0 && (uintptr_t)y % 16 == 0 && (T + 31) / 32 <= 65535;
}

// Rows of a thread: 8, unless tiles of 32 rows pad T less; one row each for a handful.
int rows_of_thread(int T) { return T <= 8 ? 1 : ((T + 31) / 32 * 32 < (T + 63) / 64 * 64 ? 4 : 8); }

// One CTA walks all groups of a tile when the tiles alone give every SM two CTAs (as many as are resident with eight
// rows a thread), or when the groups' sums would take more than ROOM floats (256 MiB: what an engine sets aside
// for them).  Neither changes a bit.  (Groups of their own against one CTA, microseconds: 600 rows x 1,024 x 4,608 164 and
// 329, 2,048 rows 418 and 516 with 128 MiB, 4,600 rows x 512 x 4,608 504 and 536 with 288 MiB; where the tiles suffice,
// 2,300 rows x 1,024 x 1,024, 118 and 115.)
constexpr long long ROOM = 1ll << 26;
bool walks_all(int T, int N, int K, int sm_count) {
    const int tm = rows_of_thread(T), group = group_size(N, K);
    const long long tiles = (long long)((T + 8 * tm - 1) / (8 * tm)) * ((N + PN - 1) / PN), groups = (K + group - 1) / group;
    return groups < 2 || tiles >= 2 * sm_count || groups * T * N > ROOM;
}

template <int TM>
int launch_float(const float* x, const float* w, const float* bias, float* y, float* partial, int T, int N, int K, bool all, cudaStream_t stream) {
    const int group = group_size(N, K), groups = (K + group - 1) / group;
    const dim3 grid(ceil_div_u(N, PN), ceil_div_u(T, 8 * TM), all ? 1 : groups);
    if (all) {
        launch_kernel(gemm_float_kernel<TM, true>, grid, P_THREADS, 0, stream, x, w, bias, y, partial, T, N, K, group);
        return launch_status();
    }
    launch_kernel(gemm_float_kernel<TM, false>, grid, P_THREADS, 0, stream, x, w, bias, y, partial, T, N, K, group);
    const int status = launch_status();
    if (status != SHISO_OK) return status;
    const long long count = (long long)T * N;
    launch_kernel(gemm_float_join_kernel, ceil_div_u(count, 1024), 256, 0, stream, (const float*)partial, bias, y, count, N, groups);
    return launch_status();
}

}  // namespace

// Groups of K whose sums shiso_gemm_float wants room for, [groups, T, N] floats on a 16-byte boundary; 0:
// none; -1: it does not take the product.
SHISO_API int shiso_gemm_float_groups(const void* x, const void* w, const void* y, int T, int N, int K, int sm_count) {
    if (T <= 0 || N <= 0 || K <= 0 || !float_takes(x, w, y, T, K)) return -1;
    if (walks_all(T, N, K, sm_count)) return 0;
    const int group = group_size(N, K);
    return (K + group - 1) / group;
}

// The columns of such a group: a function of N and K.
SHISO_API int shiso_gemm_float_group_columns(int N, int K) { return N > 0 && K > 0 ? group_size(N, K) : 0; }

SHISO_API int shiso_gemm_float(const void* x, const void* w, const float* bias, void* y, void* partial, int T, int N, int K,
                               int sm_count, cudaStream_t stream) {
    if (T <= 0 || N <= 0) return SHISO_OK;
    if (K <= 0) return SHISO_ERR_SHAPE;
    if (!float_takes(x, w, y, T, K)) return SHISO_ERR_ALIGN;
    const bool all = walks_all(T, N, K, sm_count);
    if (!all && (!partial || (uintptr_t)partial % 16)) return SHISO_ERR_ALIGN;
    const float *xf = (const float*)x, *wf = (const float*)w;
    switch (rows_of_thread(T)) {
        case 1: return launch_float<1>(xf, wf, bias, (float*)y, (float*)partial, T, N, K, all, stream);
        case 4: return launch_float<4>(xf, wf, bias, (float*)y, (float*)partial, T, N, K, all, stream);
        default: return launch_float<8>(xf, wf, bias, (float*)y, (float*)partial, T, N, K, all, stream);
    }
}

SHISO_API int shiso_gemm_simple(const void* x, int x_dtype, const void* w, int w_dtype, const float* bias,
                                void* y, int y_dtype, int T, int N, int K, cudaStream_t stream) {
    if (T <= 0 || N <= 0) return SHISO_OK;
    if (K <= 0) return SHISO_ERR_SHAPE;
    using bf = __nv_bfloat16;
    const int code = x_dtype * 4 + w_dtype * 2 + y_dtype;
    switch (code) {
        case 0: return launch<float, float, float>(x, w, bias, y, T, N, K, stream);
        case 1: return launch<float, float, bf>(x, w, bias, y, T, N, K, stream);
        case 2: return launch<bf, float, float>(x, w, bias, y, T, N, K, stream);
        case 3: return launch<bf, float, bf>(x, w, bias, y, T, N, K, stream);
        case 4: return launch<float, bf, float>(x, w, bias, y, T, N, K, stream);
        case 5: return launch<float, bf, bf>(x, w, bias, y, T, N, K, stream);
        case 6: return launch<bf, bf, float>(x, w, bias, y, T, N, K, stream);
        case 7: return launch<bf, bf, bf>(x, w, bias, y, T, N, K, stream);
        default: return SHISO_ERR_DTYPE;
    }
}
