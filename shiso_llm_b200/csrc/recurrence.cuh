// What the kernels of decaying matrix states share (recurrence.cu, which says what they compute, and
// decay_walk.cu): their arguments, the operations whose roundings have to be the same, and the row kernel that
// takes unnormalised outputs to unit RMS.
#pragma once
#include "common.cuh"

namespace {

constexpr int REC_MAX_DIM = 256;

struct RecurrenceArgs {
    const void* q; const void* k; const void* v; const void* gate;
    long long q_ld, k_ld, v_ld, gate_ld, out_ld;
    void* out;
    float* state; long long state_stride;  // [slots][heads][dim][vdim], slots `state_stride` floats apart
    const int* q_start; const int* slots; const int* positions;
    const float* decay_logits; long long logits_ld; const float* decay_bias; const float* bonus;  // channel decay
    const float* head_loss; const float* inv_freq; int rotary_dim; float key_scale;               // head decay
    const float* out_weight;
    float eps, out_scale;
    int heads, dim, vdim;
    // With `raw` (float [T, heads * vdim]) a head's value columns are shared out over col_parts CTAs
    // (blockIdx.z), which leave the unnormalised outputs there; unit RMS, weight and gate follow in
    // a row kernel.  For long portions: more SMs walk the same tokens, each with fewer columns.
    float* raw; int col_parts;
};

// What a value of the state and a rotated channel become, with every rounding written out: the kernels of
// recurrence.cu and decay_walk.cu give the same bits.  minus_w is -(1 - w).
template <bool CHANNEL>
__device__ __forceinline__ float state_moves(float S, float minus_w, float k, float v) {
    const float kept = fmaf(minus_w, S, S);
    return CHANNEL ? __fadd_rn(kept, __fmul_rn(k, v)) : fmaf(k, v, kept);
}
__device__ __forceinline__ float turned(float x, float other, float cs, float sn, bool first_half) {
    return fmaf(x, cs, __fmul_rn(other, first_half ? -sn : sn));
}

// Unit RMS over a head's value channels, times weight, silu(gate) and a constant: what follows the
// recurrence when its outputs were left unnormalised.  A warp per (row, head).
template <typename AT>
__global__ void unit_rms_gate_kernel(const float* raw, const AT* gate, long long gate_ld,
                                     const float* out_weight, AT* __restrict__ out, long long out_ld, int tokens,
                                     int heads, int vdim, float eps, float out_scale) {
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= (long long)tokens * heads) return;
    const int t = (int)(item / heads), head = (int)(item % heads);
    const float* o = raw + ((size_t)t * heads + head) * vdim;
    float vals[REC_MAX_DIM / 32];
    float squares = 0.0f;
#pragma unroll
    for (int e = 0; e < REC_MAX_DIM / 32; ++e) {
        const int c = e * 32 + lane;
        vals[e] = c < vdim ? o[c] : 0.0f;
        squares = fmaf(vals[e], vals[e], squares);
    }
    const float unit = rsqrtf(warp_sum(squares) / (float)vdim + eps);
#pragma unroll
    for (int e = 0; e < REC_MAX_DIM / 32; ++e) {
        const int c = e * 32 + lane;
        if (c < vdim) {
            float y = vals[e] * unit;
            if (out_weight) y *= out_weight[head * vdim + c];
            if (gate) {
                const float g = to_f32(gate[(size_t)t * gate_ld + (size_t)head * vdim + c]);
                y *= g / (1.0f + expf(-g));
            }
            out[(size_t)t * out_ld + (size_t)head * vdim + c] = from_f32<AT>(y * out_scale);
        }
    }
}

// two neighbouring activations
__device__ __forceinline__ float2 load_two(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_two(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }
__device__ __forceinline__ void store_two(float* p, float x, float y) { *reinterpret_cast<float2*>(p) = make_float2(x, y); }
__device__ __forceinline__ void store_two(__nv_bfloat16* p, float x, float y) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(x, y);
}

// The same bits with two channels of every 32 a lane, 16 lanes to a row of a head: lane l adds the squares up
// for the lanes 2 l and 2 l + 1 of the kernel above.
template <typename AT, int VDIM>
__global__ void unit_rms_gate_pairs_kernel(const float* raw, const AT* gate, long long gate_ld,
                                           const float* out_weight, AT* __restrict__ out, long long out_ld, int tokens,
                                           int heads, float eps, float out_scale) {
    pdl_begin();
    constexpr int PAIRS = VDIM / 32;
    const int sub = threadIdx.x % 16;
    const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 16;
    const bool on = item < (long long)tokens * heads;
    const int t = on ? (int)(item / heads) : 0, head = on ? (int)(item % heads) : 0;
    const size_t at = (size_t)head * VDIM + 2 * sub;
    float2 o[PAIRS], g[PAIRS];
#pragma unroll
    for (int e = 0; e < PAIRS; ++e) {
        o[e] = *reinterpret_cast<const float2*>(raw + (size_t)t * heads * VDIM + at + 32 * e);
        if (gate) g[e] = load_two(gate + (size_t)t * gate_ld + at + 32 * e);
    }
    float2 squares = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int e = 0; e < PAIRS; ++e) squares = make_float2(fmaf(o[e].x, o[e].x, squares.x), fmaf(o[e].y, o[e].y, squares.y));
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) {
        squares.x += __shfl_xor_sync(0xffffffffu, squares.x, off);
        squares.y += __shfl_xor_sync(0xffffffffu, squares.y, off);
    }
    const float unit = rsqrtf((squares.x + squares.y) / (float)VDIM + eps);
    if (!on) return;
#pragma unroll
    for (int e = 0; e < PAIRS; ++e) {
        float2 y = make_float2(o[e].x * unit, o[e].y * unit);
        if (out_weight) {
            y.x *= out_weight[at + 32 * e];
            y.y *= out_weight[at + 32 * e + 1];
        }
        if (gate) {
            y.x *= g[e].x / (1.0f + expf(-g[e].x));
            y.y *= g[e].y / (1.0f + expf(-g[e].y));
        }
        store_two(out + (size_t)t * out_ld + at + 32 * e, y.x * out_scale, y.y * out_scale);
    }
}

template <typename AT>
int launch_unit_rms_gate(const RecurrenceArgs& a, int tokens, cudaStream_t stream) {
    const float* raw = a.raw;
    const AT* gate = (const AT*)a.gate;
    AT* out = (AT*)a.out;
    const long long items = (long long)tokens * a.heads;
    const uintptr_t two = 2 * sizeof(AT);
    const bool wide = (uintptr_t)gate % two == 0 && (uintptr_t)out % two == 0 && a.gate_ld % 2 == 0 && a.out_ld % 2 == 0 && (uintptr_t)raw % 8 == 0;
    if (wide && a.vdim == 64)
        launch_kernel(unit_rms_gate_pairs_kernel<AT, 64>, ceil_div_u(items, 16), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out,
                      a.out_ld, tokens, a.heads, a.eps, a.out_scale);
    else if (wide && a.vdim == 128)
        launch_kernel(unit_rms_gate_pairs_kernel<AT, 128>, ceil_div_u(items, 16), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out,
                      a.out_ld, tokens, a.heads, a.eps, a.out_scale);
    else
        launch_kernel(unit_rms_gate_kernel<AT>, ceil_div_u(items, 8), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out, a.out_ld,
                      tokens, a.heads, a.vdim, a.eps, a.out_scale);
    return launch_status();
}

// The arguments both entry points are called with; false where they contradict one another.
inline bool fill_recurrence(RecurrenceArgs& a, const void* q, const void* k, const void* v, const void* gate, long long q_ld,
                            long long k_ld, long long v_ld, long long gate_ld, void* out, long long out_ld, float* state,
                            long long state_stride, const int* q_start, const int* slots, const int* positions,
                            const float* decay_logits, long long logits_ld, const float* decay_bias, const float* bonus,
                            const float* head_loss, const float* inv_freq, int rotary_dim, float key_scale, const float* out_weight,
                            float eps, float out_scale, float* raw, int col_parts, int heads, int dim, int vdim) {
    const bool channel = decay_logits != nullptr;
    if (channel == (head_loss != nullptr)) return false;
    if (channel && (!decay_bias || !bonus)) return false;
    if (rotary_dim && (channel || !inv_freq || rotary_dim % 2 || rotary_dim > dim)) return false;
    a.q = q; a.k = k; a.v = v; a.gate = gate;
    a.q_ld = q_ld; a.k_ld = k_ld; a.v_ld = v_ld; a.gate_ld = gate_ld; a.out_ld = out_ld;
    a.out = out; a.state = state; a.state_stride = state_stride;
    a.q_start = q_start; a.slots = slots; a.positions = positions;
    a.decay_logits = decay_logits; a.logits_ld = logits_ld; a.decay_bias = decay_bias; a.bonus = bonus;
    a.head_loss = head_loss; a.inv_freq = inv_freq; a.rotary_dim = rotary_dim; a.key_scale = key_scale;
    a.out_weight = out_weight; a.eps = eps; a.out_scale = out_scale;
    a.heads = heads; a.dim = dim; a.vdim = vdim;
    a.raw = raw; a.col_parts = raw ? col_parts : 1;
    return true;
}

}  // namespace
