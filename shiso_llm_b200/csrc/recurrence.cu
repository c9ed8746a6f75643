// Linear recurrences with a matrix state per head, walked token by token in float.
//
// One CTA per (head, sequence) holds the head's state S[key, value] in registers and walks the
// sequence's rows of this step in order, so a position's output does not depend on how the
// sequence was cut into steps or on what else is in the batch.  Two forms:
//
// A decay w multiplies the state as S - (1 - w) S with 1 - w formed directly (expm1f; the host
// hands over 1 - decay_h): a decay close to 1 rounded to float32 as such would be off by 2^-24 of
// itself per step, which a thousand steps multiply, while 1 - w keeps its own 24 bits.
//
//   channel decay (time mixing of the RWKV family)
//       w_t = exp(-exp(logit_t + bias))                       per key channel
//       o_t = (S_{t-1} + diag(bonus) k_t v_t^T)^T q_t
//       S_t = diag(w_t) S_{t-1} + k_t v_t^T
//   head decay (retention)
//       q_t, k_t rotated by the position (half-split pairs), k_t times key_scale
//       S_t = decay_h S_{t-1} + k_t v_t^T                 (head_loss = 1 - decay_h is what is handed over)
//       o_t = S_t^T q_t
//
// then, for both, o_t brought to unit RMS over the head's value channels, times an optional
// weight, times silu(gate), times a constant, rounded to the activation type.
//
// Thread layout: a value column j of the state belongs to SPLIT neighbouring lanes, each
// holding dim / SPLIT neighbouring rows in registers; the SPLIT partial sums of o_j meet in
// a few shuffles.  q, k and the decays of eight tokens at a time are staged in shared memory; a
// thread walks the eight tokens over its rows of the state without meeting the others, so a
// batch costs two barriers (the staged batch; the sums of squares of its eight outputs), and what
// the next batch brings is asked for from global memory while this one is walked.  The sums a
// token takes part in and their order are the same whatever the batch: cuts change no bit.
#include "common.cuh"

constexpr int REC_MAX_DIM = 256;
constexpr int REC_MAX_STATE = 32768;  // floats of one head's state: what a CTA keeps in registers

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
    // The walk of long portions: a state and a decay per segment (see there).
    int seqs;
    float* segment_state; float* segment_decay;
};

// Threads a CTA may have so that RPT rows of the state (and what else a thread needs) stay in registers.
constexpr int rec_max_threads(int rpt) { return rpt <= 32 ? 512 : (rpt <= 128 ? 256 : 128); }

constexpr int REC_BATCH = 8;   // tokens staged and walked between two barriers
constexpr int REC_STAGED = 4;  // channels of q and k a thread stages per batch, at most

template <typename AT, int RPT, int SPLIT, bool CHANNEL>
__global__ void __launch_bounds__(rec_max_threads(RPT)) decay_recurrence_kernel(const RecurrenceArgs a) {
    __shared__ __align__(16) float sq[REC_BATCH][REC_MAX_DIM], sk[REC_BATCH][REC_MAX_DIM], sw[CHANNEL ? REC_BATCH : 1][REC_MAX_DIM];
    __shared__ __align__(16) float su[REC_MAX_DIM];
    __shared__ float red[REC_BATCH][32];
    const int head = blockIdx.x, seq = blockIdx.y;
    const int tid = threadIdx.x, threads = blockDim.x;
    const int part = tid % SPLIT;
    const int dim = a.dim, vdim = a.vdim;
    const int cols = vdim / a.col_parts;  // value columns of this CTA
    const int j = blockIdx.z * cols + tid / SPLIT;  // this thread's column
    const int rpt = dim / SPLIT;  // rows of the state per thread (dim is a multiple of SPLIT)
    const bool owns = tid / SPLIT < cols;
    const int lane = tid & 31, warp = tid >> 5, nwarps = (threads + 31) >> 5;
    // tokens per batch: what the threads can stage with REC_STAGED channels each (at least two:
    // the CTA has half as many threads as there are key channels)
    const int batch = min(REC_BATCH, REC_STAGED * threads / dim);

    if (CHANNEL)
        for (int c = tid; c < dim; c += threads) su[c] = a.bonus[head * dim + c];
    const float head_loss = CHANNEL ? 0.0f : a.head_loss[head];  // 1 - decay
    const int half = a.rotary_dim / 2;
    // what a thread stages of every batch: element e = tid + l * threads is channel e % dim of token e / dim
    int st_token[REC_STAGED], st_chan[REC_STAGED];
    float st_const[REC_STAGED];  // the channel's decay bias, or its rotation frequency
#pragma unroll
    for (int l = 0; l < REC_STAGED; ++l) {
        const int e = tid + l * threads;
        st_token[l] = e / dim;
        st_chan[l] = e % dim;
        st_const[l] = 0.0f;
        if (st_token[l] < batch) {
            const int c = st_chan[l];
            if (CHANNEL) st_const[l] = a.decay_bias[head * dim + c];
            else if (c < a.rotary_dim) st_const[l] = a.inv_freq[c < half ? c : c - half];
        }
    }
    const float out_weight = (a.out_weight && owns) ? a.out_weight[head * vdim + j] : 1.0f;
    pdl_wait();
    const int first = a.q_start[seq], last = a.q_start[seq + 1];
    if (last <= first) return;
    __syncthreads();  // the bonus is staged
    // a thread's rows of the state are neighbours: row = part * rpt + ii
    const int row0 = part * rpt;
    const bool wide = rpt % 4 == 0;  // its slices of the staged vectors are read 16 bytes at a time
    float* state = a.state + (long long)a.slots[seq] * a.state_stride + (size_t)head * dim * vdim;
    float S[RPT];
#pragma unroll
    for (int ii = 0; ii < RPT; ++ii) {
        S[ii] = (owns && ii < rpt) ? state[(size_t)(row0 + ii) * vdim + j] : 0.0f;
    }

    const AT* q = (const AT*)a.q + (size_t)head * dim;
    const AT* k = (const AT*)a.k + (size_t)head * dim;
    const AT* v = (const AT*)a.v + (size_t)head * vdim;
    const AT* gate = a.gate ? (const AT*)a.gate + (size_t)head * vdim : nullptr;
    AT* out = (AT*)a.out + (size_t)head * vdim;

    // What a batch of tokens brings is asked for one batch ahead: the loads are in flight while the
    // state walks the batch before.
    struct Raw { float q[REC_STAGED], k[REC_STAGED], q_other[REC_STAGED], k_other[REC_STAGED], v[REC_BATCH]; };
    // (Every load below has a valid address whatever n is - a token index beyond the batch is the
    // batch's last, an idle thread's column is the CTA's first - and nothing is converted before all
    // are asked for: a branch or a conversion between two loads would make each wait for the one before.)
    const int jc = owns ? j : blockIdx.z * cols;
    auto fetch = [&](int t0, int n, Raw& r) {
        AT raw_q[REC_STAGED], raw_k[REC_STAGED], raw_qo[REC_STAGED], raw_ko[REC_STAGED], raw_v[REC_BATCH];
        float raw_logit[REC_STAGED];
#pragma unroll
        for (int l = 0; l < REC_STAGED; ++l) {
            const int t = t0 + min(st_token[l], n - 1), c = st_chan[l];
            raw_q[l] = q[(size_t)t * a.q_ld + c];
            raw_k[l] = k[(size_t)t * a.k_ld + c];
            if (CHANNEL) {
                raw_logit[l] = a.decay_logits[(size_t)t * a.logits_ld + head * dim + c];
            } else {
                const int other = c < a.rotary_dim ? (c < half ? c + half : c - half) : c;
                raw_qo[l] = q[(size_t)t * a.q_ld + other];
                raw_ko[l] = k[(size_t)t * a.k_ld + other];
            }
        }
#pragma unroll
        for (int i = 0; i < REC_BATCH; ++i) raw_v[i] = v[(size_t)(t0 + min(i, n - 1)) * a.v_ld + jc];
#pragma unroll
        for (int l = 0; l < REC_STAGED; ++l) {
            r.q[l] = to_f32(raw_q[l]);
            r.k[l] = to_f32(raw_k[l]);
            r.q_other[l] = CHANNEL ? raw_logit[l] : to_f32(raw_qo[l]);
            r.k_other[l] = CHANNEL ? 0.0f : to_f32(raw_ko[l]);
        }
#pragma unroll
        for (int i = 0; i < REC_BATCH; ++i) r.v[i] = to_f32(raw_v[i]);
    };
    auto stage = [&](int t0, int n, const Raw& r) {
#pragma unroll
        for (int l = 0; l < REC_STAGED; ++l) {
            if (st_token[l] >= n) continue;
            const int i = st_token[l], c = st_chan[l];
            float qc = r.q[l], kc = r.k[l];
            if (!CHANNEL) {
                if (c < a.rotary_dim) {
                    float sn, cs;
                    sincosf((float)a.positions[t0 + i] * st_const[l], &sn, &cs);
                    qc = c < half ? qc * cs - r.q_other[l] * sn : qc * cs + r.q_other[l] * sn;
                    kc = c < half ? kc * cs - r.k_other[l] * sn : kc * cs + r.k_other[l] * sn;
                }
                kc *= a.key_scale;
            } else {
                sw[i][c] = -expm1f(-expf(r.q_other[l] + st_const[l]));  // 1 - w, exact to the last bit also where w is close to 1
            }
            sq[i][c] = qc;
            sk[i][c] = kc;
        }
    };
    // one row of the state takes one token
    auto take = [&](int ii, float qv, float kval, float wv, float uv, float vj, float& o) {
        const float kv = kval * vj;
        if (CHANNEL) {
            o += qv * (S[ii] + uv * kv);
            S[ii] = fmaf(-wv, S[ii], S[ii]) + kv;
        } else {
            S[ii] = fmaf(-head_loss, S[ii], S[ii]) + kv;
            o += qv * S[ii];
        }
    };
    Raw cur, next;
    fetch(first, min(batch, last - first), cur);
    stage(first, min(batch, last - first), cur);
    for (int t0 = first; t0 < last; t0 += batch) {
        const int n = min(batch, last - t0);
        const int n_next = min(batch, last - t0 - n);
        if (n_next > 0) fetch(t0 + n, n_next, next);
        float gates[REC_BATCH];  // asked for now, needed after the batch is walked
        if (gate && !a.raw) {
            AT raw_gate[REC_BATCH];
#pragma unroll
            for (int i = 0; i < REC_BATCH; ++i) raw_gate[i] = gate[(size_t)(t0 + min(i, n - 1)) * a.gate_ld + jc];
#pragma unroll
            for (int i = 0; i < REC_BATCH; ++i) gates[i] = to_f32(raw_gate[i]);
        } else {
#pragma unroll
            for (int i = 0; i < REC_BATCH; ++i) gates[i] = 0.0f;
        }
        __syncthreads();  // the batch is staged
        float o[REC_BATCH];
#pragma unroll
        for (int i = 0; i < REC_BATCH; ++i) {
            o[i] = 0.0f;
            if (i < n) {
                const float vj = cur.v[i];
                // (the sum over a thread's rows runs in row order, as four interleaved chains)
                float o4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (wide) {
#pragma unroll
                    for (int g4 = 0; g4 < RPT / 4; ++g4) {
                        if (4 * g4 < rpt) {
                            const float4 q4 = *reinterpret_cast<const float4*>(&sq[i][row0 + 4 * g4]);
                            const float4 k4 = *reinterpret_cast<const float4*>(&sk[i][row0 + 4 * g4]);
                            float4 w4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u4 = w4;
                            if (CHANNEL) {
                                w4 = *reinterpret_cast<const float4*>(&sw[i][row0 + 4 * g4]);
                                u4 = *reinterpret_cast<const float4*>(&su[row0 + 4 * g4]);
                            }
                            take(4 * g4 + 0, q4.x, k4.x, w4.x, u4.x, vj, o4[0]);
                            take(4 * g4 + 1, q4.y, k4.y, w4.y, u4.y, vj, o4[1]);
                            take(4 * g4 + 2, q4.z, k4.z, w4.z, u4.z, vj, o4[2]);
                            take(4 * g4 + 3, q4.w, k4.w, w4.w, u4.w, vj, o4[3]);
                        }
                    }
                } else {
#pragma unroll
                    for (int ii = 0; ii < RPT; ++ii)
                        if (ii < rpt) take(ii, sq[i][row0 + ii], sk[i][row0 + ii], CHANNEL ? sw[i][row0 + ii] : 0.0f, CHANNEL ? su[row0 + ii] : 0.0f, vj, o4[ii & 3]);
                }
                o[i] = (o4[0] + o4[1]) + (o4[2] + o4[3]);
            }
        }
#pragma unroll
        for (int i = 0; i < REC_BATCH; ++i) {
#pragma unroll
            for (int off = 1; off < SPLIT; off <<= 1) o[i] += __shfl_xor_sync(0xffffffffu, o[i], off);
            if (a.raw) {
                if (owns && i % SPLIT == part && i < n) a.raw[(size_t)(t0 + i) * a.heads * vdim + (size_t)head * vdim + j] = o[i];
            } else {
                const float partial = warp_sum((owns && part == 0) ? o[i] * o[i] : 0.0f);
                if (lane == 0) red[i][warp] = partial;
            }
        }
        __syncthreads();  // every thread has read the staged batch; the sums of squares are written
        if (owns && !a.raw) {
            // (every lane of a column holds the column's sums: the lanes share the batch's tokens)
#pragma unroll
            for (int i = 0; i < REC_BATCH; ++i) {
                if (i % SPLIT == part && i < n) {
                    float squares = 0.0f;
                    for (int w = 0; w < nwarps; ++w) squares += red[i][w];
                    float y = o[i] * rsqrtf(squares / (float)vdim + a.eps) * out_weight;
                    if (gate) y *= gates[i] / (1.0f + expf(-gates[i]));
                    out[(size_t)(t0 + i) * a.out_ld + j] = from_f32<AT>(y * a.out_scale);
                }
            }
        }
        if (n_next > 0) {
            stage(t0 + n, n_next, next);
            cur = next;
        }
        // (the next batch's first barrier orders these writes before its reads, and this batch's
        // reads of the sums before their next writes)
    }
    pdl_trigger();
#pragma unroll
    for (int ii = 0; ii < RPT; ++ii)
        if (owns && ii < rpt) state[(size_t)(row0 + ii) * vdim + j] = S[ii];
}

template <typename AT, int SPLIT, bool CHANNEL>
static int launch_recurrence(const RecurrenceArgs& a, int num_seqs, cudaStream_t stream) {
    const int rpt = a.dim / SPLIT;
    // a thread per lane of a column, and at least half as many threads as key channels (they stage q and k)
    const int columns = (a.vdim / a.col_parts * SPLIT + 31) / 32 * 32, stagers = ((a.dim + 1) / 2 + 31) / 32 * 32;
    const unsigned threads = (unsigned)(columns > stagers ? columns : stagers);
    const dim3 grid(a.heads, num_seqs, a.col_parts);
#define SHISO_REC(R)                                                                                          \
    if constexpr (R * SPLIT <= REC_MAX_DIM) {                                                                 \
        if (rpt <= R) {                                                                                       \
            if (threads > (unsigned)rec_max_threads(R)) return SHISO_ERR_SHAPE;                               \
            launch_kernel(decay_recurrence_kernel<AT, R, SPLIT, CHANNEL>, grid, threads, 0, stream, a);       \
            return launch_status();                                                                           \
        }                                                                                                     \
    }
    SHISO_REC(8) SHISO_REC(16) SHISO_REC(32) SHISO_REC(64) SHISO_REC(128) SHISO_REC(256)
#undef SHISO_REC
    return SHISO_ERR_SHAPE;
}

static int rows_bucket(int rpt) {
    for (int r = 8; r <= REC_MAX_DIM; r *= 2)
        if (rpt <= r) return r;
    return REC_MAX_DIM;
}

// Into how many lanes a column of the state is split: as many (8, 4, 2, 1) as divide the key size
// and leave the CTA within the threads its rows per thread allow; 0 when nothing fits.
static int choose_split(int dim, int vdim) {
    for (int split = 8; split >= 1; split /= 2) {
        if (dim % split || dim / split < 1) continue;
        const int columns = (vdim * split + 31) / 32 * 32, stagers = ((dim + 1) / 2 + 31) / 32 * 32;
        if ((columns > stagers ? columns : stagers) <= rec_max_threads(rows_bucket(dim / split))) return split;
    }
    return 0;
}

SHISO_API int shiso_decay_recurrence_supported(int dim, int vdim) {
    return dim > 0 && vdim > 0 && dim <= REC_MAX_DIM && vdim <= REC_MAX_DIM && dim * vdim <= REC_MAX_STATE && choose_split(dim, vdim) > 0;
}

template <typename AT, bool CHANNEL>
static int pick_split(const RecurrenceArgs& a, int num_seqs, cudaStream_t stream) {
    switch (choose_split(a.dim, a.vdim / a.col_parts)) {
        case 8: return launch_recurrence<AT, 8, CHANNEL>(a, num_seqs, stream);
        case 4: return launch_recurrence<AT, 4, CHANNEL>(a, num_seqs, stream);
        case 2: return launch_recurrence<AT, 2, CHANNEL>(a, num_seqs, stream);
        case 1: return launch_recurrence<AT, 1, CHANNEL>(a, num_seqs, stream);
    }
    return SHISO_ERR_SHAPE;
}

// ---- long portions, key size 64 ------------------------------------------------------------
// The kernel above has a thread or two per SM lane however long the portion is, and the threads that walk
// the state also convert, exponentiate or rotate what a batch brings: a token costs some 1,500 cycles of
// latency (1.58 ms for 2,000 tokens of 32 heads of 64 x 64).  Here
//   - a portion is cut into segments of 128 tokens that are walked at the same time.  A first pass walks
//     every segment but the last from a zero state and leaves the state it ends with and the decay over
//     the whole segment; walk_join_kernel carries the sequence's state through them,
//     S <- decay_segment * S + local; a second pass walks every segment from its true state.  The first
//     pass has under half of the second's arithmetic, and both fill the chip;
//   - eight warps of a CTA (64 value columns of a head) do nothing but walk, and four stage the next 16
//     tokens into the other of two buffers: one barrier a batch;
//   - a lane has 4 rows of 4 columns of the state as pairs of rows for the packed multiply-adds
//     (fma.rn.f32x2): 32 of them a token with a channel decay beside four 16-byte reads of shared memory
//     (8 rows of one column: 6 reads for half the state, and the reads bound the walk);
//   - the sixteen partial sums of a column meet for 4 tokens x 4 columns at once: every exchange halves
//     what a lane keeps, 15 shuffles instead of 64.
// All sums and states are float; the decay over a segment is the product of the same float factors the
// state takes, rounded no more often than the state itself.
// (One pass without segments, 128 CTAs of four walking warps: 432 us, 6.7 cycles between two instructions
// of a scheduler's only walking warp.)
constexpr int WALK_DIM = 64, WALK_COLS = 64, WALK_BATCH = 16, WALK_SEGMENT = 128;
constexpr int WALKERS = 256, STAGERS = 128, WALK_THREADS = WALKERS + STAGERS;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair_of(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float pair_sum(f32x2 v) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    return x + y;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// four neighbouring activations in one load, kept as they are until they are staged
template <typename AT> struct Four;
template <> struct Four<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void get(float (&f)[4]) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
};
template <> struct Four<__nv_bfloat16> {
    uint2 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void get(float (&f)[4]) const {
        f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
        f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
    }
};

// The segment behind a slot.  Segment `seg` of sequence s has slot q_start[s] / 128 + s + seg: slots of
// different segments never meet, and there are tokens / 128 + sequences of them.
struct Segment { int seq, seg, first, last; bool only, final; };
__device__ __forceinline__ bool find_segment(const int* q_start, int seqs, int slot, Segment& out) {
    int lo = 0, hi = seqs - 1;  // the last sequence whose first slot is not behind `slot`
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (q_start[mid] / WALK_SEGMENT + mid <= slot) lo = mid;
        else hi = mid - 1;
    }
    const int start = q_start[lo], end = q_start[lo + 1];
    out.seq = lo;
    out.seg = slot - (start / WALK_SEGMENT + lo);
    out.first = start + out.seg * WALK_SEGMENT;
    if (out.seg < 0 || out.first >= end) return false;
    out.last = min(end, out.first + WALK_SEGMENT);
    out.only = end - start <= WALK_SEGMENT;
    out.final = out.last == end;
    return true;
}

// FULL: the second pass (outputs to a.raw); else the first (states and decays of whole segments).
template <typename AT, bool CHANNEL, bool FULL>
__global__ void __launch_bounds__(WALK_THREADS, 2) decay_walk_kernel(const RecurrenceArgs a) {
    struct Buffer {
        float q[FULL ? WALK_BATCH : 1][WALK_DIM], k[WALK_BATCH][WALK_DIM], loss[CHANNEL ? WALK_BATCH : 1][WALK_DIM];  // loss: -(1 - w)
        float v[WALK_BATCH][WALK_COLS];
    };
    __shared__ __align__(16) Buffer buffers[2];
    __shared__ float decays[CHANNEL && !FULL ? 8 : 1][WALK_DIM];
    const int head = blockIdx.x, slot = blockIdx.y, col0 = blockIdx.z * WALK_COLS;
    const int tid = threadIdx.x;
    const int vdim = a.vdim;
    pdl_wait();
    Segment at;
    if (!find_segment(a.q_start, a.seqs, slot, at) || (!FULL && at.final)) return;
    const int batches = (at.last - at.first + WALK_BATCH - 1) / WALK_BATCH;

    if (tid >= WALKERS) {
        // ---- staging: chunk e of a batch is channels 4 (e % 16) .. + 3 of token e / 16
        constexpr int CHUNKS = WALK_BATCH * WALK_DIM / 4 / STAGERS, EVERY = STAGERS / 16;
        const int s = tid - WALKERS;
        const int c = (s % 16) * 4, token0 = s / 16;
        const int half = a.rotary_dim / 2;
        const bool turns = !CHANNEL && c < a.rotary_dim;
        const int other = turns ? (c < half ? c + half : c - half) : c;
        float constant[4];  // the channels' decay bias, or their rotation frequency
#pragma unroll
        for (int x = 0; x < 4; ++x)
            constant[x] = CHANNEL ? a.decay_bias[head * WALK_DIM + c + x] : (turns ? a.inv_freq[(c < half ? c : c - half) + x] : 0.0f);
        const AT* q = (const AT*)a.q + (size_t)head * WALK_DIM;
        const AT* k = (const AT*)a.k + (size_t)head * WALK_DIM;
        const AT* v = (const AT*)a.v + (size_t)head * vdim + col0;
        Four<AT> rq[CHUNKS], rk[CHUNKS], rq_other[CHUNKS], rk_other[CHUNKS], rv[CHUNKS];
        float4 logit[CHUNKS];
        int position[CHUNKS];
        float over[4] = {1.0f, 1.0f, 1.0f, 1.0f};  // the decay over this thread's tokens of the segment
        // (a token index beyond the segment's last is the last: every load has a valid address)
        auto fetch = [&](int b) {
#pragma unroll
            for (int l = 0; l < CHUNKS; ++l) {
                const int t = min(at.first + b * WALK_BATCH + token0 + l * EVERY, at.last - 1);
                if (FULL) rq[l].load(q + (size_t)t * a.q_ld + c);
                rk[l].load(k + (size_t)t * a.k_ld + c);
                rv[l].load(v + (size_t)t * a.v_ld + c);
                if (CHANNEL) {
                    logit[l] = *reinterpret_cast<const float4*>(a.decay_logits + (size_t)t * a.logits_ld + head * WALK_DIM + c);
                } else {
                    if (FULL) rq_other[l].load(q + (size_t)t * a.q_ld + other);
                    rk_other[l].load(k + (size_t)t * a.k_ld + other);
                    position[l] = a.rotary_dim ? a.positions[t] : 0;
                }
            }
        };
        auto stage = [&](Buffer& to) {
#pragma unroll
            for (int l = 0; l < CHUNKS; ++l) {
                const int i = token0 + l * EVERY;
                float fq[4], fk[4], fv[4];
                if (FULL) rq[l].get(fq);
                rk[l].get(fk);
                rv[l].get(fv);
                if (CHANNEL) {
                    const float z[4] = {logit[l].x, logit[l].y, logit[l].z, logit[l].w};
                    float loss[4];
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        loss[x] = expm1f(-expf(z[x] + constant[x]));
                        if (!FULL) over[x] = fmaf(loss[x], over[x], over[x]);
                    }
                    *reinterpret_cast<float4*>(&to.loss[i][c]) = make_float4(loss[0], loss[1], loss[2], loss[3]);
                } else {
                    if (turns) {
                        float oq[4], ok[4];
                        if (FULL) rq_other[l].get(oq);
                        rk_other[l].get(ok);
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            float sn, cs;
                            sincosf((float)position[l] * constant[x], &sn, &cs);
                            if (c < half) sn = -sn;
                            if (FULL) fq[x] = fq[x] * cs + oq[x] * sn;
                            fk[x] = fk[x] * cs + ok[x] * sn;
                        }
                    }
#pragma unroll
                    for (int x = 0; x < 4; ++x) fk[x] *= a.key_scale;
                }
                if (FULL) *reinterpret_cast<float4*>(&to.q[i][c]) = make_float4(fq[0], fq[1], fq[2], fq[3]);
                *reinterpret_cast<float4*>(&to.k[i][c]) = make_float4(fk[0], fk[1], fk[2], fk[3]);
                *reinterpret_cast<float4*>(&to.v[i][c]) = make_float4(fv[0], fv[1], fv[2], fv[3]);
            }
        };
        fetch(0);
        stage(buffers[0]);
        if (batches > 1) fetch(1);
        for (int b = 0; b < batches; ++b) {
            __syncthreads();  // batch b is staged, batch b - 1 is walked
            if (b + 1 < batches) stage(buffers[(b + 1) & 1]);
            if (b + 2 < batches) fetch(b + 2);
        }
        pdl_trigger();
        if (CHANNEL && !FULL) {
#pragma unroll
            for (int x = 0; x < 4; ++x) decays[token0][c + x] = over[x];
            asm volatile("bar.sync 1, %0;" ::"n"(STAGERS) : "memory");
            if (s < WALK_DIM && blockIdx.z == 0) {
                float product = 1.0f;
#pragma unroll
                for (int g = 0; g < EVERY; ++g) product *= decays[g][s];
                a.segment_decay[((size_t)slot * a.heads + head) * WALK_DIM + s] = product;
            }
        }
        return;
    }

    // ---- the walk: 16 lanes share 4 columns, 4 rows of the state each
    const int part = tid & 15, cg = (tid >> 4) * 4;  // cg: first of the lane's columns within the CTA's
    const size_t own = ((size_t)part * 4) * vdim + col0 + cg;
    float* segment_state = a.segment_state + ((size_t)slot * a.heads + head) * WALK_DIM * vdim + own;
    float* cache_state = a.state + (long long)a.slots[at.seq] * a.state_stride + (size_t)head * WALK_DIM * vdim + own;
    f32x2 S[4][2], bonus[2];  // [column][pair of rows]
    {
        const float* from = at.only ? cache_state : segment_state;
        float4 r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = FULL ? *reinterpret_cast<const float4*>(from + (size_t)i * vdim) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            S[0][p] = pair_of(r[2 * p].x, r[2 * p + 1].x);
            S[1][p] = pair_of(r[2 * p].y, r[2 * p + 1].y);
            S[2][p] = pair_of(r[2 * p].z, r[2 * p + 1].z);
            S[3][p] = pair_of(r[2 * p].w, r[2 * p + 1].w);
            const float* u = a.bonus + head * WALK_DIM + part * 4 + 2 * p;
            bonus[p] = CHANNEL && FULL ? pair_of(u[0], u[1]) : 0ull;
        }
    }
    const float head_loss = CHANNEL ? 0.0f : -a.head_loss[head];
    const f32x2 loss_all = pair_of(head_loss, head_loss);
    float* raw = FULL ? a.raw + (size_t)head * vdim + col0 + cg : nullptr;
    const size_t raw_ld = (size_t)a.heads * vdim;
    // one token: the state moves on; o[c]: this lane's share of the output
    auto token = [&](const Buffer& from, int i, float (&o)[4]) {
        const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&from.k[i][part * 4]);
        const float4 v4 = *reinterpret_cast<const float4*>(&from.v[i][cg]);
        ulonglong2 w2 = make_ulonglong2(loss_all, loss_all), q2 = make_ulonglong2(0ull, 0ull);
        if (CHANNEL) w2 = *reinterpret_cast<const ulonglong2*>(&from.loss[i][part * 4]);
        if (FULL) q2 = *reinterpret_cast<const ulonglong2*>(&from.q[i][part * 4]);
        const f32x2 vv[4] = {pair_of(v4.x, v4.x), pair_of(v4.y, v4.y), pair_of(v4.z, v4.z), pair_of(v4.w, v4.w)};
        f32x2 now = 0ull;  // q u k: what the token itself adds, before its value
        if (CHANNEL && FULL) now = fma2(mul2(q2.y, bonus[1]), k2.y, mul2(mul2(q2.x, bonus[0]), k2.x));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            f32x2 sum = 0ull;
            if (CHANNEL && FULL) sum = fma2(q2.y, S[c][1], fma2(q2.x, S[c][0], mul2(now, vv[c])));
            S[c][0] = fma2(k2.x, vv[c], fma2(w2.x, S[c][0], S[c][0]));
            S[c][1] = fma2(k2.y, vv[c], fma2(w2.y, S[c][1], S[c][1]));
            if (!CHANNEL && FULL) sum = fma2(q2.y, S[c][1], mul2(q2.x, S[c][0]));
            if (FULL) o[c] = pair_sum(sum);
        }
    };
    for (int b = 0; b < batches; ++b) {
        __syncthreads();  // batch b is staged
        const Buffer& from = buffers[b & 1];
        const int t0 = at.first + b * WALK_BATCH, n = min(WALK_BATCH, at.last - t0);
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += 4) {
            float o[16];  // [token][column]
            auto four = [&](int count) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float mine[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    if (i < count) token(from, i0 + i, mine);
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[4 * i + c] = mine[c];
                }
            };
            if (i0 + 4 <= n) four(4);  // (no branch between two tokens)
            else four(n - i0);
            if (FULL) {
#pragma unroll
                for (int bit = 1, kept = 8; bit < 16; bit *= 2, kept /= 2) {
                    const bool upper = part & bit;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (i < kept) {
                            const float keeps = upper ? o[2 * i + 1] : o[2 * i], gives = upper ? o[2 * i] : o[2 * i + 1];
                            o[i] = keeps + __shfl_xor_sync(0xffffffffu, gives, bit);
                        }
                    }
                }
                // o[0] is now the sum for token part / 4 and column part % 4
                if (i0 + part / 4 < n) raw[(size_t)(t0 + i0 + part / 4) * raw_ld + part % 4] = o[0];
            }
        }
    }
    pdl_trigger();
    if (FULL && !at.final) return;
    float* to = FULL ? cache_state : segment_state;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float x[4], y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) asm("mov.b64 {%0, %1}, %2;" : "=f"(x[c]), "=f"(y[c]) : "l"(S[c][p]));
        *reinterpret_cast<float4*>(to + (size_t)(2 * p) * vdim) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(to + (size_t)(2 * p + 1) * vdim) = make_float4(y[0], y[1], y[2], y[3]);
    }
}

// Carries each sequence's state through its segments: a segment's place first holds the state its first
// pass ended with, then the state it begins with.  Four values of a head's state a thread.
template <bool CHANNEL>
__global__ void __launch_bounds__(256) walk_join_kernel(const RecurrenceArgs a) {
    pdl_begin();
    const int head = blockIdx.x, seq = blockIdx.y;
    const int start = a.q_start[seq], count = a.q_start[seq + 1] - start;
    const int segments = (count + WALK_SEGMENT - 1) / WALK_SEGMENT;
    if (segments < 2) return;
    const int at = (blockIdx.z * 256 + threadIdx.x) * 4;  // within the head's state
    if (at >= WALK_DIM * a.vdim) return;
    const int row = at / a.vdim;
    const int slot0 = start / WALK_SEGMENT + seq;
    float decay = 1.0f;
    if (!CHANNEL) {
        const float loss = -a.head_loss[head];
        for (int i = 0; i < WALK_SEGMENT; ++i) decay = fmaf(loss, decay, decay);
    }
    float4 S = *reinterpret_cast<const float4*>(a.state + (long long)a.slots[seq] * a.state_stride + (size_t)head * WALK_DIM * a.vdim + at);
    const size_t step = (size_t)a.heads * WALK_DIM * a.vdim;
    float* place = a.segment_state + (size_t)slot0 * step + (size_t)head * WALK_DIM * a.vdim + at;
    const float* over = a.segment_decay + ((size_t)slot0 * a.heads + head) * WALK_DIM + row;
    const size_t over_step = (size_t)a.heads * WALK_DIM;
    for (int g0 = 0; g0 < segments; g0 += 4) {
        // four segments asked for before the first is needed (the last segment has no first pass)
        float4 local[4];
        float w[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const bool walked = g0 + g + 1 < segments;
            local[g] = walked ? *reinterpret_cast<const float4*>(place + g * step) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w[g] = CHANNEL ? (walked ? over[g * over_step] : 0.0f) : decay;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            if (g0 + g < segments) *reinterpret_cast<float4*>(place + g * step) = S;
            S.x = fmaf(w[g], S.x, local[g].x);
            S.y = fmaf(w[g], S.y, local[g].y);
            S.z = fmaf(w[g], S.z, local[g].z);
            S.w = fmaf(w[g], S.w, local[g].w);
        }
        place += 4 * step;
        over += 4 * over_step;
    }
}

// What the walk reads four values at a time has to lie on their boundary.
static bool walk_takes(const RecurrenceArgs& a, int act_dtype) {
    const uintptr_t four = act_dtype == SHISO_F32 ? 16 : 8;
    auto aligned = [](const void* p, uintptr_t to) { return (uintptr_t)p % to == 0; };
    if (!a.raw || !a.segment_state || a.dim != WALK_DIM || a.vdim % WALK_COLS || a.col_parts != a.vdim / WALK_COLS) return false;
    if (!aligned(a.q, four) || !aligned(a.k, four) || !aligned(a.v, four) || a.q_ld % 4 || a.k_ld % 4 || a.v_ld % 4) return false;
    if (!aligned(a.state, 16) || a.state_stride % 4 || !aligned(a.segment_state, 16)) return false;
    if (a.decay_logits) return aligned(a.decay_logits, 16) && a.logits_ld % 4 == 0;
    return a.rotary_dim % 8 == 0;  // four channels turn together
}

template <typename AT, bool CHANNEL>
static int launch_walk(const RecurrenceArgs& a, int tokens, int longest, cudaStream_t stream) {
    const int slots = tokens / WALK_SEGMENT + a.seqs;
    if (slots > 65535 || a.seqs > 65535) return SHISO_ERR_SHAPE;
    const dim3 grid(a.heads, slots, a.col_parts);
    if (longest > WALK_SEGMENT) {
        launch_kernel(decay_walk_kernel<AT, CHANNEL, false>, grid, WALK_THREADS, 0, stream, a);
        launch_kernel(walk_join_kernel<CHANNEL>, dim3(a.heads, a.seqs, ceil_div_u(WALK_DIM * a.vdim, 1024)), 256, 0, stream, a);
    }
    launch_kernel(decay_walk_kernel<AT, CHANNEL, true>, grid, WALK_THREADS, 0, stream, a);
    return launch_status();
}

// Unit RMS over a head's value channels, times weight, silu(gate) and a constant: what follows the
// recurrence when its outputs were left unnormalised.  A warp per (row, head).
template <typename AT>
__global__ void unit_rms_gate_kernel(const float* __restrict__ raw, const AT* __restrict__ gate, long long gate_ld,
                                     const float* __restrict__ out_weight, AT* __restrict__ out, long long out_ld, int tokens,
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
        squares += vals[e] * vals[e];
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

// The same with a quarter of the lanes to a row of a head and 16-byte accesses: LANES = vdim / 4.
// (2,048 rows of 32 heads of 64: 24 us with a lane's values 128 bytes apart.)
template <typename AT, int LANES>
__global__ void unit_rms_gate_vec_kernel(const float* __restrict__ raw, const AT* __restrict__ gate, long long gate_ld,
                                         const float* __restrict__ out_weight, AT* __restrict__ out, long long out_ld, int tokens,
                                         int heads, float eps, float out_scale) {
    pdl_begin();
    constexpr int VDIM = 4 * LANES;
    const int sub = threadIdx.x % LANES;
    const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const bool on = item < (long long)tokens * heads;
    const int t = on ? (int)(item / heads) : 0, head = on ? (int)(item % heads) : 0;
    const size_t at = (size_t)head * VDIM + sub * 4;
    const float4 o4 = *reinterpret_cast<const float4*>(raw + (size_t)t * heads * VDIM + at);
    Four<AT> g4;
    if (gate) g4.load(gate + (size_t)t * gate_ld + at);
    float o[4] = {o4.x, o4.y, o4.z, o4.w};
    float squares = (o[0] * o[0] + o[1] * o[1]) + (o[2] * o[2] + o[3] * o[3]);
#pragma unroll
    for (int off = 1; off < LANES; off *= 2) squares += __shfl_xor_sync(0xffffffffu, squares, off);
    const float unit = rsqrtf(squares / (float)VDIM + eps);
    float g[4];
    if (gate) g4.get(g);
    if (!on) return;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        o[x] *= unit;
        if (out_weight) o[x] *= out_weight[at + x];
        if (gate) o[x] *= g[x] / (1.0f + expf(-g[x]));
        o[x] *= out_scale;
    }
    AT* to = out + (size_t)t * out_ld + at;
    if constexpr (sizeof(AT) == 4) {
        *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
        *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    }
}

template <typename AT>
static int launch_unit_rms_gate(const RecurrenceArgs& a, int tokens, cudaStream_t stream) {
    const float* raw = a.raw;
    const AT* gate = (const AT*)a.gate;
    AT* out = (AT*)a.out;
    const long long items = (long long)tokens * a.heads;
    const uintptr_t four = 4 * sizeof(AT);
    const bool wide = (uintptr_t)gate % four == 0 && (uintptr_t)out % four == 0 && a.gate_ld % 4 == 0 && a.out_ld % 4 == 0;
    if (wide && a.vdim == 64)
        launch_kernel(unit_rms_gate_vec_kernel<AT, 16>, ceil_div_u(items, 16), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out,
                      a.out_ld, tokens, a.heads, a.eps, a.out_scale);
    else if (wide && a.vdim == 128)
        launch_kernel(unit_rms_gate_vec_kernel<AT, 32>, ceil_div_u(items, 8), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out,
                      a.out_ld, tokens, a.heads, a.eps, a.out_scale);
    else
        launch_kernel(unit_rms_gate_kernel<AT>, ceil_div_u(items, 8), 256, 0, stream, raw, gate, a.gate_ld, a.out_weight, out, a.out_ld,
                      tokens, a.heads, a.vdim, a.eps, a.out_scale);
    return launch_status();
}

SHISO_API int shiso_decay_recurrence(const void* q, const void* k, const void* v, const void* gate, long long q_ld, long long k_ld,
                                     long long v_ld, long long gate_ld, void* out, long long out_ld, int act_dtype, float* state,
                                     long long state_stride, const int* q_start, const int* slots, const int* positions,
                                     const float* decay_logits, long long logits_ld, const float* decay_bias, const float* bonus,
                                     const float* head_loss, const float* inv_freq, int rotary_dim, float key_scale,
                                     const float* out_weight, float eps, float out_scale, float* raw, int col_parts, float* room,
                                     int longest, int tokens,
                                     int num_seqs, int heads, int dim, int vdim, cudaStream_t stream) {
    if (num_seqs <= 0 || heads <= 0) return SHISO_OK;
    if (dim <= 0 || vdim <= 0 || dim > REC_MAX_DIM || vdim > REC_MAX_DIM || dim * vdim > REC_MAX_STATE) return SHISO_ERR_SHAPE;
    const bool channel = decay_logits != nullptr;
    if (channel == (head_loss != nullptr)) return SHISO_ERR_UNSUPPORTED;
    if (channel && (!decay_bias || !bonus)) return SHISO_ERR_UNSUPPORTED;
    if (rotary_dim && (channel || !inv_freq || rotary_dim % 2 || rotary_dim > dim)) return SHISO_ERR_UNSUPPORTED;
    RecurrenceArgs a;
    a.q = q; a.k = k; a.v = v; a.gate = gate;
    a.q_ld = q_ld; a.k_ld = k_ld; a.v_ld = v_ld; a.gate_ld = gate_ld; a.out_ld = out_ld;
    a.out = out; a.state = state; a.state_stride = state_stride;
    a.q_start = q_start; a.slots = slots; a.positions = positions;
    a.decay_logits = decay_logits; a.logits_ld = logits_ld; a.decay_bias = decay_bias; a.bonus = bonus;
    a.head_loss = head_loss; a.inv_freq = inv_freq; a.rotary_dim = rotary_dim; a.key_scale = key_scale;
    a.out_weight = out_weight; a.eps = eps; a.out_scale = out_scale;
    a.heads = heads; a.dim = dim; a.vdim = vdim;
    a.raw = raw; a.col_parts = raw ? col_parts : 1;
    if (a.col_parts < 1 || vdim % a.col_parts || !shiso_decay_recurrence_supported(dim, vdim / a.col_parts)) return SHISO_ERR_SHAPE;
    a.seqs = num_seqs;
    a.segment_state = room;
    a.segment_decay = room ? room + (size_t)(tokens / WALK_SEGMENT + num_seqs) * heads * dim * vdim : nullptr;
    int status;
    if (walk_takes(a, act_dtype) && act_dtype == SHISO_F32)
        status = channel ? launch_walk<float, true>(a, tokens, longest, stream) : launch_walk<float, false>(a, tokens, longest, stream);
    else if (walk_takes(a, act_dtype) && act_dtype == SHISO_BF16)
        status = channel ? launch_walk<__nv_bfloat16, true>(a, tokens, longest, stream) : launch_walk<__nv_bfloat16, false>(a, tokens, longest, stream);
    else if (act_dtype == SHISO_F32) status = channel ? pick_split<float, true>(a, num_seqs, stream) : pick_split<float, false>(a, num_seqs, stream);
    else if (act_dtype == SHISO_BF16)
        status = channel ? pick_split<__nv_bfloat16, true>(a, num_seqs, stream) : pick_split<__nv_bfloat16, false>(a, num_seqs, stream);
    else return SHISO_ERR_DTYPE;
    if (status != SHISO_OK || !raw) return status;
    return act_dtype == SHISO_F32 ? launch_unit_rms_gate<float>(a, tokens, stream) : launch_unit_rms_gate<__nv_bfloat16>(a, tokens, stream);
}
