// Decaying matrix states with 64 key channels (recurrence.cu says what they are), long portions.
//
// The kernel of recurrence.cu has a thread or two per SM lane however long the portion is, and the threads that
// walk the state also convert, exponentiate or rotate what a batch brings: a token costs some 1,800 cycles of
// latency.  Here
//   - the state alone walks first: decay_walk_states_kernel takes a portion of more than 128 tokens in
//     order, without q and without outputs - two or three multiply-adds a value and token, nothing that lanes
//     have to exchange - and leaves the state at every 128th token;
//   - decay_walk_kernel then walks all segments of 128 tokens at the same time, each from its true state,
//     and forms the outputs;
//   - of a CTA's warps some do nothing but walk, and the others stage the next tokens into the other of
//     two buffers: one barrier a batch;
//   - a lane's rows of the state are pairs for the packed multiply-adds;
//   - the partial sums of a column meet for 4 tokens x 4 columns at once: every exchange halves what a
//     lane keeps, 15 shuffles instead of 64.
// Every operation on a value of the state and every sum of an output is the general kernel's with a column
// over 8 lanes, in its order: which of the two runs, and where a portion is cut, changes no bit of the
// state and none of the outputs before their unit RMS.
//
// Measured with the row kernel, bfloat16, microseconds, the general kernel's first: 2,000 tokens of 32 heads of
// 64 x 64, channel decay, 1,938 and 158; of 16 heads of 64 x 128, head decay, 1,239 and 134; eight portions of 250
// tokens 655 and 127, 319 and 102; one of 64 tokens 66 and 16, 44 and 14.  What bounds the first walk: a batch's staging
// (the loads' latency, exponentials or rotations), which every CTA of a head repeats; the second: multiply-adds and reads
// of shared memory.  (Segments walked from a zero state and joined by their decays, S <- w S + local, took 125 and
// 109 us for the 2,000 tokens, but every cut of a prompt had other bits then.)
#include "recurrence.cuh"

namespace {

constexpr int WALK_DIM = 64, WALK_SEGMENT = 128;
// The second walk's CTA, and the first's: 16 value columns, so that few heads still fill the chip, and twice the
// tokens and staging warps, because there the staging is what a batch waits for.
struct OutputWalk { static constexpr int COLS = 64, BATCH = 16, WALKERS = 256, STAGERS = 128; static constexpr bool OUT = true; };
struct StateWalk { static constexpr int COLS = 16, BATCH = 32, WALKERS = 128, STAGERS = 256; static constexpr bool OUT = false; };

// state_moves for two rows.  The product of two bfloat16 values is exact in float, so that one fused operation
// rounds as a product and a sum do.  (Where it is not, the two stand as scalar intrinsics, which nothing
// may join.)
template <typename AT, bool CHANNEL>
__device__ __forceinline__ f32x2 state_moves2(f32x2 S, f32x2 minus_w, f32x2 k, f32x2 v) {
    const f32x2 kept = fma2(minus_w, S, S);
    if constexpr (!CHANNEL || sizeof(AT) == 2) return fma2(k, v, kept);
    float kx, ky, vx, vy, x, y;
    halves(k, kx, ky);
    halves(v, vx, vy);
    halves(kept, x, y);
    return pair_of(__fadd_rn(x, __fmul_rn(kx, vx)), __fadd_rn(y, __fmul_rn(ky, vy)));
}

struct WalkArgs : RecurrenceArgs {
    int seqs;
    float* segment_state;  // the states that segments begin with; null: every sequence is walked in one piece
};

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

// Where the states of a sequence's segments lie: segment `seg` of a sequence of more than 128 tokens has
// place 2 (q_start / 128) + seg.  n tokens > 128 have at most 2 (n / 128) segments, so the places of
// different sequences never meet and there are 2 (tokens / 128) of them.
__device__ __forceinline__ int state_place(int start, int seg) { return 2 * (start / WALK_SEGMENT) + seg; }

// The segment behind a grid row of the second walk.  Segment `seg` of sequence s has row
// q_start[s] / 128 + s + seg: rows of different segments never meet, and there are
// tokens / 128 + sequences of them.  Without a first walk a sequence's only segment is all of it.
struct Segment { int seq, seg, start, first, last; bool only, final; };
__device__ __forceinline__ bool find_segment(const int* q_start, int seqs, int row, bool whole, Segment& out) {
    int lo = 0, hi = seqs - 1;  // the last sequence whose first row is not behind `row`
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (q_start[mid] / WALK_SEGMENT + mid <= row) lo = mid;
        else hi = mid - 1;
    }
    const int start = q_start[lo], end = q_start[lo + 1];
    out.seq = lo;
    out.seg = row - (start / WALK_SEGMENT + lo);
    out.start = start;
    out.first = start + out.seg * WALK_SEGMENT;
    if (out.seg < 0 || out.first >= end || (whole && out.seg > 0)) return false;
    out.last = whole ? end : min(end, out.first + WALK_SEGMENT);
    out.only = whole || end - start <= WALK_SEGMENT;
    out.final = out.last == end;
    return true;
}

// Staged tokens.  The second walk: with q, and the channels of q, k and the losses in the order in which a
// lane wants them - of every eight, 0 1 4 5 and then 2 3 6 7.  The first: without q, in their own order, and every
// value twice, as the packed operations take it.
template <typename W, bool CHANNEL> struct WalkBuffer {
    float q[W::OUT ? W::BATCH : 1][WALK_DIM], k[W::BATCH][WALK_DIM], loss[CHANNEL ? W::BATCH : 1][WALK_DIM];  // loss: -(1 - w)
    float v[W::BATCH][W::OUT ? W::COLS : 2 * W::COLS];
};

// What a staging thread does: chunk e of a batch is channels 4 (e % 16) .. + 3 of token e / 16.
// Meets the walkers at one barrier a batch.
template <typename AT, typename W, bool CHANNEL>
__device__ __forceinline__ void walk_stage(const WalkArgs& a, WalkBuffer<W, CHANNEL> (&buffers)[2], int s, int head, int col0,
                                           int first, int last, int batches) {
    constexpr bool OUT = W::OUT;
    constexpr int CHUNKS = W::BATCH * WALK_DIM / 4 / W::STAGERS, EVERY = W::STAGERS / 16;
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
    const AT* v = (const AT*)a.v + (size_t)head * a.vdim + col0;
    // (values: as many chunks as the columns have, the first walk's for half of the threads)
    constexpr int VCHUNKS = OUT ? CHUNKS : 1;
    const bool has_v = OUT || s < W::BATCH * W::COLS / 4;
    const int vc = OUT ? c : (s % (W::COLS / 4)) * 4, vtoken = OUT ? token0 : s / (W::COLS / 4);
    struct Raw {
        Four<AT> q[OUT ? CHUNKS : 1], k[CHUNKS], q_other[OUT ? CHUNKS : 1], k_other[CHUNKS], v[VCHUNKS];
        float4 logit[CHUNKS];
        int position[CHUNKS];
    };
    // (a token index beyond the segment's last is the last: every load has a valid address)
    auto fetch = [&](int b, Raw& r) {
#pragma unroll
        for (int l = 0; l < CHUNKS; ++l) {
            const int t = min(first + b * W::BATCH + token0 + l * EVERY, last - 1);
            if (OUT) r.q[l].load(q + (size_t)t * a.q_ld + c);
            r.k[l].load(k + (size_t)t * a.k_ld + c);
            if (CHANNEL) {
                r.logit[l] = *reinterpret_cast<const float4*>(a.decay_logits + (size_t)t * a.logits_ld + head * WALK_DIM + c);
            } else {
                if (OUT) r.q_other[l].load(q + (size_t)t * a.q_ld + other);
                r.k_other[l].load(k + (size_t)t * a.k_ld + other);
                r.position[l] = a.rotary_dim ? a.positions[t] : 0;
            }
        }
#pragma unroll
        for (int l = 0; l < VCHUNKS; ++l) {
            const int t = min(first + b * W::BATCH + vtoken + l * EVERY, last - 1);
            if (has_v) r.v[l].load(v + (size_t)t * a.v_ld + vc);
        }
    };
    auto put = [&](float (&to)[WALK_DIM], const float (&f)[4]) {
        if (OUT) {
            float* at = to + (c & ~7) + (c & 4) / 2;
            *reinterpret_cast<float2*>(at) = make_float2(f[0], f[1]);
            *reinterpret_cast<float2*>(at + 4) = make_float2(f[2], f[3]);
        } else {
            *reinterpret_cast<float4*>(to + c) = make_float4(f[0], f[1], f[2], f[3]);
        }
    };
    auto stage = [&](WalkBuffer<W, CHANNEL>& to, const Raw& r) {
#pragma unroll
        for (int l = 0; l < CHUNKS; ++l) {
            const int i = token0 + l * EVERY;
            float fq[4], fk[4];
            if (OUT) r.q[l].get(fq);
            r.k[l].get(fk);
            if (CHANNEL) {
                const float z[4] = {r.logit[l].x, r.logit[l].y, r.logit[l].z, r.logit[l].w};
                float loss[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) loss[x] = expm1f(-expf(z[x] + constant[x]));
                put(to.loss[i], loss);
            } else {
                if (turns) {
                    float oq[4], ok[4];
                    if (OUT) r.q_other[l].get(oq);
                    r.k_other[l].get(ok);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        float sn, cs;
                        sincosf((float)r.position[l] * constant[x], &sn, &cs);
                        if (OUT) fq[x] = turned(fq[x], oq[x], cs, sn, c < half);
                        fk[x] = turned(fk[x], ok[x], cs, sn, c < half);
                    }
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) fk[x] *= a.key_scale;
            }
            if (OUT) put(to.q[i], fq);
            put(to.k[i], fk);
        }
#pragma unroll
        for (int l = 0; l < VCHUNKS; ++l) {
            float fv[4];
            if (!has_v) continue;
            r.v[l].get(fv);
            float* at = &to.v[vtoken + l * EVERY][OUT ? vc : 2 * vc];
            if (OUT) {
                *reinterpret_cast<float4*>(at) = make_float4(fv[0], fv[1], fv[2], fv[3]);
            } else {
                *reinterpret_cast<float4*>(at) = make_float4(fv[0], fv[0], fv[1], fv[1]);
                *reinterpret_cast<float4*>(at + 4) = make_float4(fv[2], fv[2], fv[3], fv[3]);
            }
        }
    };
    Raw cur, next;
    fetch(0, cur);
    stage(buffers[0], cur);
    if (batches > 1) fetch(1, cur);
    for (int b = 0; b < batches; ++b) {
        __syncthreads();  // batch b is staged, batch b - 1 is walked
        // (the first walk has the registers for two batches on their way: the loads of one behind the staging of the other)
        if (!OUT && b + 2 < batches) fetch(b + 2, next);
        if (b + 1 < batches) stage(buffers[(b + 1) & 1], cur);
        if (OUT && b + 2 < batches) fetch(b + 2, cur);
        if (!OUT) cur = next;
    }
    pdl_trigger();
}

// The first walk: the states of a sequence of more than 128 tokens at every 128th token, the first included.
// 16 lanes share 2 columns of 64 rows, 4 neighbouring rows of the state each.
template <typename AT, bool CHANNEL>
__global__ void __launch_bounds__(StateWalk::WALKERS + StateWalk::STAGERS) decay_walk_states_kernel(const WalkArgs a) {
    __shared__ __align__(16) WalkBuffer<StateWalk, CHANNEL> buffers[2];
    const int head = blockIdx.x, seq = blockIdx.y, col0 = blockIdx.z * StateWalk::COLS;
    const int tid = threadIdx.x, vdim = a.vdim;
    pdl_wait();
    const int first = a.q_start[seq], tokens = a.q_start[seq + 1] - first;
    if (tokens <= WALK_SEGMENT) return;
    const int whole = (tokens - 1) / WALK_SEGMENT;  // all segments but the last, which the second walk takes
    const int batches = whole * (WALK_SEGMENT / StateWalk::BATCH);
    if (tid >= StateWalk::WALKERS) {
        walk_stage<AT, StateWalk, CHANNEL>(a, buffers, tid - StateWalk::WALKERS, head, col0, first, first + whole * WALK_SEGMENT, batches);
        return;
    }
    const int part = tid & 15, cg = (tid >> 4) * 2;
    const size_t own = ((size_t)head * WALK_DIM + part * 4) * vdim + col0 + cg;
    const size_t step = (size_t)a.heads * WALK_DIM * vdim;
    const float* from = a.state + (long long)a.slots[seq] * a.state_stride + own;
    float* to = a.segment_state + state_place(first, 0) * step + own;
    f32x2 S[2][2];  // [column][pair of rows]
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float2 x = *reinterpret_cast<const float2*>(from + (size_t)(2 * p) * vdim);
        const float2 y = *reinterpret_cast<const float2*>(from + (size_t)(2 * p + 1) * vdim);
        S[0][p] = pair_of(x.x, y.x);
        S[1][p] = pair_of(x.y, y.y);
    }
    const float head_loss = CHANNEL ? 0.0f : -a.head_loss[head];
    const f32x2 loss_all = pair_of(head_loss, head_loss);
    auto leave = [&]() {
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            float2 x, y;
            halves(S[0][p], x.x, y.x);
            halves(S[1][p], x.y, y.y);
            *reinterpret_cast<float2*>(to + (size_t)(2 * p) * vdim) = x;
            *reinterpret_cast<float2*>(to + (size_t)(2 * p + 1) * vdim) = y;
        }
        to += step;
    };
    leave();
    for (int b = 0; b < batches; ++b) {
        __syncthreads();  // batch b is staged
        const WalkBuffer<StateWalk, CHANNEL>& at = buffers[b & 1];
#pragma unroll 16
        for (int i = 0; i < StateWalk::BATCH; ++i) {
            const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&at.k[i][part * 4]);
            const ulonglong2 v2 = *reinterpret_cast<const ulonglong2*>(&at.v[i][2 * cg]);
            ulonglong2 w2 = make_ulonglong2(loss_all, loss_all);
            if (CHANNEL) w2 = *reinterpret_cast<const ulonglong2*>(&at.loss[i][part * 4]);
            S[0][0] = state_moves2<AT, CHANNEL>(S[0][0], w2.x, k2.x, v2.x);
            S[0][1] = state_moves2<AT, CHANNEL>(S[0][1], w2.y, k2.y, v2.x);
            S[1][0] = state_moves2<AT, CHANNEL>(S[1][0], w2.x, k2.x, v2.y);
            S[1][1] = state_moves2<AT, CHANNEL>(S[1][1], w2.y, k2.y, v2.y);
        }
        if ((b + 1) % (WALK_SEGMENT / StateWalk::BATCH) == 0) leave();
    }
    pdl_trigger();
}

// The second walk: every segment from the state it begins with; the outputs to a.raw, the state of a
// sequence's last segment to its slot.  16 lanes share 4 columns: lanes 2 e and 2 e + 1 have rows 8 e + 0 1 4 5
// and 8 e + 2 3 6 7, so that a lane's sum over its two pairs of rows is two of the general kernel's four
// chains, and the exchange with its neighbour what follows there.
template <typename AT, bool CHANNEL>
__global__ void __launch_bounds__(OutputWalk::WALKERS + OutputWalk::STAGERS, 2) decay_walk_kernel(const WalkArgs a) {
    __shared__ __align__(16) WalkBuffer<OutputWalk, CHANNEL> buffers[2];
    const int head = blockIdx.x, col0 = blockIdx.z * OutputWalk::COLS;
    const int tid = threadIdx.x, vdim = a.vdim;
    pdl_wait();
    Segment at;
    if (!find_segment(a.q_start, a.seqs, blockIdx.y, a.segment_state == nullptr, at)) return;
    const int batches = (at.last - at.first + OutputWalk::BATCH - 1) / OutputWalk::BATCH;
    if (tid >= OutputWalk::WALKERS) {
        walk_stage<AT, OutputWalk, CHANNEL>(a, buffers, tid - OutputWalk::WALKERS, head, col0, at.first, at.last, batches);
        return;
    }
    const int part = tid & 15, cg = (tid >> 4) * 4;  // cg: first of the lane's columns within the CTA's
    const int row0 = (part >> 1) * 8 + (part & 1) * 2;  // its rows: row0 + 0, 1, 4, 5
    const size_t own = ((size_t)head * WALK_DIM + row0) * vdim + col0 + cg;
    float* cache_state = a.state + (long long)a.slots[at.seq] * a.state_stride + own;
    f32x2 S[4][2], bonus[2];  // [column][pair of rows]
    {
        const float* from = at.only ? cache_state : a.segment_state + state_place(at.start, at.seg) * ((size_t)a.heads * WALK_DIM * vdim) + own;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float4 x = *reinterpret_cast<const float4*>(from + (size_t)(4 * p) * vdim);
            const float4 y = *reinterpret_cast<const float4*>(from + (size_t)(4 * p + 1) * vdim);
            S[0][p] = pair_of(x.x, y.x);
            S[1][p] = pair_of(x.y, y.y);
            S[2][p] = pair_of(x.z, y.z);
            S[3][p] = pair_of(x.w, y.w);
            const float* u = a.bonus + head * WALK_DIM + row0 + 4 * p;
            bonus[p] = CHANNEL ? pair_of(u[0], u[1]) : 0ull;
        }
    }
    const float head_loss = CHANNEL ? 0.0f : -a.head_loss[head];
    const f32x2 loss_all = pair_of(head_loss, head_loss);
    float* raw = a.raw + (size_t)head * vdim + col0 + cg;
    const size_t raw_ld = (size_t)a.heads * vdim;
    // one token: the state moves on; o[c]: this lane's share of the output
    auto token = [&](const WalkBuffer<OutputWalk, CHANNEL>& from, int i, float (&o)[4]) {
        const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&from.k[i][part * 4]);
        const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(&from.q[i][part * 4]);
        const float4 v4 = *reinterpret_cast<const float4*>(&from.v[i][cg]);
        ulonglong2 w2 = make_ulonglong2(loss_all, loss_all);
        if (CHANNEL) w2 = *reinterpret_cast<const ulonglong2*>(&from.loss[i][part * 4]);
        const f32x2 vv[4] = {pair_of(v4.x, v4.x), pair_of(v4.y, v4.y), pair_of(v4.z, v4.z), pair_of(v4.w, v4.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            f32x2 sum = 0ull;
            if (CHANNEL) {
                // (these products are factors: there is nothing to join them with)
                sum = fma2(q2.x, fma2(bonus[0], mul2(k2.x, vv[c]), S[c][0]), sum);
                sum = fma2(q2.y, fma2(bonus[1], mul2(k2.y, vv[c]), S[c][1]), sum);
            }
            S[c][0] = state_moves2<AT, CHANNEL>(S[c][0], w2.x, k2.x, vv[c]);
            S[c][1] = state_moves2<AT, CHANNEL>(S[c][1], w2.y, k2.y, vv[c]);
            if (!CHANNEL) sum = fma2(q2.y, S[c][1], fma2(q2.x, S[c][0], sum));
            float x, y;
            halves(sum, x, y);
            o[c] = x + y;
        }
    };
    for (int b = 0; b < batches; ++b) {
        __syncthreads();  // batch b is staged
        const WalkBuffer<OutputWalk, CHANNEL>& from = buffers[b & 1];
        const int t0 = at.first + b * OutputWalk::BATCH, n = min(OutputWalk::BATCH, at.last - t0);
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
    pdl_trigger();
    if (!at.final) return;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float4 x, y;
        halves(S[0][p], x.x, y.x);
        halves(S[1][p], x.y, y.y);
        halves(S[2][p], x.z, y.z);
        halves(S[3][p], x.w, y.w);
        *reinterpret_cast<float4*>(cache_state + (size_t)(4 * p) * vdim) = x;
        *reinterpret_cast<float4*>(cache_state + (size_t)(4 * p + 1) * vdim) = y;
    }
}

template <typename AT, bool CHANNEL>
int launch_walk(const WalkArgs& a, int tokens, cudaStream_t stream) {
    if (a.segment_state) {
        // (not in its predecessor's tail: about as many CTAs as SMs, each as long as the portion, would share
        // the SMs that happened to be free first)
        const dim3 walks(a.heads, a.seqs, a.vdim / StateWalk::COLS);
        decay_walk_states_kernel<AT, CHANNEL><<<walks, StateWalk::WALKERS + StateWalk::STAGERS, 0, stream>>>(a);
    }
    const dim3 segments(a.heads, tokens / WALK_SEGMENT + a.seqs, a.vdim / OutputWalk::COLS);
    launch_kernel(decay_walk_kernel<AT, CHANNEL>, segments, OutputWalk::WALKERS + OutputWalk::STAGERS, 0, stream, a);
    const int status = launch_status();
    return status == SHISO_OK ? launch_unit_rms_gate<AT>(a, tokens, stream) : status;
}

}  // namespace

// Whether the walk takes a step: what it reads four values at a time has to lie on their boundary, and a
// grid's second dimension ends at 65,535.
SHISO_API int shiso_decay_walk_takes(int act_dtype, const void* q, const void* k, const void* v, long long q_ld, long long k_ld,
                                     long long v_ld, const float* state, long long state_stride, const float* decay_logits,
                                     long long logits_ld, int rotary_dim, int tokens, int num_seqs, int dim, int vdim) {
    if (act_dtype != SHISO_F32 && act_dtype != SHISO_BF16) return 0;
    const uintptr_t four = act_dtype == SHISO_F32 ? 16 : 8;
    auto aligned = [](const void* p, uintptr_t to) { return (uintptr_t)p % to == 0; };
    if (dim != WALK_DIM || vdim <= 0 || vdim > REC_MAX_DIM || vdim % OutputWalk::COLS) return 0;
    if (tokens <= 0 || num_seqs <= 0 || (long long)tokens / WALK_SEGMENT + num_seqs > 65535) return 0;
    if (!aligned(q, four) || !aligned(k, four) || !aligned(v, four) || q_ld % 4 || k_ld % 4 || v_ld % 4) return 0;
    if (!aligned(state, 16) || state_stride % 4) return 0;
    if (decay_logits) return aligned(decay_logits, 16) && logits_ld % 4 == 0;
    return rotary_dim % 8 == 0;  // four channels turn together
}

// raw: [tokens, heads * vdim] floats; room: 2 (tokens / 128) states of all heads for the segments, or null
// where no sequence is worth more than one (a longer one is then walked in one piece).
SHISO_API int shiso_decay_walk(const void* q, const void* k, const void* v, const void* gate, long long q_ld, long long k_ld,
                               long long v_ld, long long gate_ld, void* out, long long out_ld, int act_dtype, float* state,
                               long long state_stride, const int* q_start, const int* slots, const int* positions,
                               const float* decay_logits, long long logits_ld, const float* decay_bias, const float* bonus,
                               const float* head_loss, const float* inv_freq, int rotary_dim, float key_scale,
                               const float* out_weight, float eps, float out_scale, float* raw, float* room, int tokens,
                               int num_seqs, int heads, int dim, int vdim, cudaStream_t stream) {
    if (num_seqs <= 0 || heads <= 0) return SHISO_OK;
    if (!shiso_decay_walk_takes(act_dtype, q, k, v, q_ld, k_ld, v_ld, state, state_stride, decay_logits, logits_ld, rotary_dim, tokens,
                                num_seqs, dim, vdim) || !raw || (uintptr_t)raw % 16 || (uintptr_t)room % 16)
        return SHISO_ERR_ALIGN;
    WalkArgs a;
    if (!fill_recurrence(a, q, k, v, gate, q_ld, k_ld, v_ld, gate_ld, out, out_ld, state, state_stride, q_start, slots, positions,
                         decay_logits, logits_ld, decay_bias, bonus, head_loss, inv_freq, rotary_dim, key_scale, out_weight, eps,
                         out_scale, raw, 1, heads, dim, vdim))
        return SHISO_ERR_UNSUPPORTED;
    a.seqs = num_seqs;
    a.segment_state = room;
    const bool channel = decay_logits != nullptr;
    if (act_dtype == SHISO_F32) return channel ? launch_walk<float, true>(a, tokens, stream) : launch_walk<float, false>(a, tokens, stream);
    return channel ? launch_walk<__nv_bfloat16, true>(a, tokens, stream) : launch_walk<__nv_bfloat16, false>(a, tokens, stream);
}
