// Linear attention with a decayed matrix state: per head a matrix S [key_dim, value_dim], zero at
// a sequence's start, and for every token
//
//     S <- diag(a_t) S + k_t v_t^T          o_t = S^T q_t * q_scale
//
// The decay a_t is one of
//   0  a constant per head (decay[head]); the same for every key channel and token;
//   1  a vector per token and head over the key channels, a = logistic(z)^(1 / tau) with
//      z = gate[row, head * key_dim + d] + gate_bias[head * key_dim + d] (float32), computed as
//      exp(-softplus(-z) / tau).
// q, k and v come from one projected row [q | k | v | ...] of the activation type; with
// silu_inputs they pass silu first.  Everything after the load is float32: the state, the decay
// with its softplus and exponential, the sums.
//
// Other mixers use the same recurrence with other decays and read-outs: linear_attention.cuh.
//
// Two kernels.  linear_attention_prepare does what is the same for every column, once per entry:
// silu of q, k and v where asked, the decay with its softplus and exponential, all to float32 rows
// [row][head][k | q | (decay) | v], the key parts padded with zeros and the values to a multiple of
// 16.  linear_attention_kernel is the recurrence, for every mixer that has one of the kinds of
// linear_attention.cuh.  A column of S (one entry of v and of o) evolves on its own.  16 lanes hold
// COLS neighbouring columns, lane l the key channels 4l .. 4l + 3, 64 + 4l .. of each (runs of four, for
// 16-byte accesses), so that a key, query or decay once loaded serves COLS columns.  One block per
// (sequence, head, 16 columns) walks the sequence's tokens of the step in order.  The tokens come
// through a ring of buffers in shared memory, filled by asynchronous 16-byte copies: a warp copies whole
// tokens, a lane the same pieces of each.  A token's sums over the lanes are not reduced one by one
// (each would be a chain of shuffles that the next token waits behind): every lane leaves its share in
// shared memory, and once a stage of tokens is through, each lane adds up the 16 shares of some
// (token, column) pairs and writes their results.  A row's result depends on its sequence's own
// tokens only, in an order fixed by the sizes.
//
// Prompts with gated decays, bfloat16 rows and keys of 128 go in chunks of 32 tokens instead: linear_attention_chunk_kernel works out what
// a chunk needs beside the state, the walk of chunk_walk.cuh takes the chunks on the tensor cores.
#include <math.h>

#include <algorithm>

#include "chunk_walk.cuh"
#include "linear_attention.cuh"

namespace {

constexpr int kLanes = kRecurrenceLanes;
constexpr int kColumns = kRecurrenceColumns;  // columns of S per block
constexpr int kGroup = 8;                     // tokens between whose loads no store stands
// tokens per buffer, and buffers: fewer tokens for long keys, so that the ring fits
constexpr int stage_tokens(int per) { return per <= 8 ? 16 : 8; }
constexpr int kBuffers = 3;
// floats between the shares of neighbouring columns: the two column groups of a warp store without bank conflicts
constexpr int share_stride(int cols) { return cols == 2 ? 24 : 20; }

__device__ __forceinline__ void copy16_async(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// logistic(z)^(1 / tau) = exp(-softplus(-z) / tau), without overflow; in double on the 32-bit path
template <typename T> __device__ __forceinline__ float logistic_power(float z, float inv_tau) {
    const float log_logistic = fminf(z, 0.f) - log1pf(expf(-fabsf(z)));      // (one way for either sign: no lane waits for another)
    return expf(log_logistic * inv_tau);
}
template <> __device__ __forceinline__ float logistic_power<float>(float z, float inv_tau) {
    const double x = (double)z;
    const double log_logistic = x >= 0.0 ? -log1p(exp(-x)) : x - log1p(exp(x));
    return (float)exp(log_logistic * (double)inv_tau);
}

// prepared [rows][heads][parts * kp + vp] float32: k, q (and the decay) over kp entries each, then
// v over vp entries; entries beyond key_dim and value_dim are zero.
template <typename T>
__global__ void linear_attention_prepare_kernel(float* __restrict__ prepared, const T* __restrict__ proj, int proj_width,
                                                int q_offset, int k_offset, int v_offset, const float* __restrict__ gate,
                                                int gate_width, const float* __restrict__ gate_bias, float inv_tau,
                                                long long n, int n_heads, int key_dim, int value_dim, int kp, int vp,
                                                int parts, int silu_inputs) {
    pdl_launch_dependents();
    pdl_wait();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int per_head = parts * kp + vp;
    const long long unit = e / per_head;
    const int c = (int)(e - unit * per_head);
    const long long row = unit / n_heads;
    const int head = (int)(unit - row * n_heads);
    const T* src = proj + row * proj_width;
    float v = 0.f;
    if (c >= parts * kp) {
        const int d = c - parts * kp;
        if (d < value_dim) {
            v = to_f32<T>(src[v_offset + head * value_dim + d]);
            if (silu_inputs) v = silu_of<T>(v);
        }
    } else {
        const int part = c / kp, d = c - part * kp;
        if (d < key_dim) {
            if (part == 2) {
                v = logistic_power<T>(gate[row * gate_width + head * key_dim + d] + (gate_bias ? gate_bias[head * key_dim + d] : 0.f),
                                      inv_tau);
            } else {
                v = to_f32<T>(src[(part == 0 ? k_offset : q_offset) + head * key_dim + d]);
                if (silu_inputs) v = silu_of<T>(v);
            }
        }
    }
    prepared[e] = v;
}

// The same for bfloat16 rows in whole groups of four entries: a thread per group, 8 bytes in and 16 out (1,531 rows
// of 32 heads of 128 with gated decays on B200: 49 us, 137 above, with 2-byte accesses and two divisions an entry).
__global__ void __launch_bounds__(256) linear_attention_prepare_vec_kernel(
    float* __restrict__ prepared, const __nv_bfloat16* __restrict__ proj, int proj_width, int q_offset, int k_offset, int v_offset,
    const float* __restrict__ gate, int gate_width, const float* __restrict__ gate_bias, float inv_tau, int n_heads, int key_dim,
    int value_dim, int kp, int vp, int parts, int silu_inputs) {
    pdl_launch_dependents();
    pdl_wait();
    using T = __nv_bfloat16;
    const int per_head = parts * kp + vp, item = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (item >= n_heads * per_head) return;
    const int head = item / per_head, c = item - head * per_head;
    const long long row = blockIdx.x;
    const int part = c >= parts * kp ? 3 : c / kp;              // k, q, decay, v
    const int d = part == 3 ? c - parts * kp : c - part * kp;
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (part == 2) {
        if (d < key_dim) {
            const int at = head * key_dim + d;
            out = *reinterpret_cast<const float4*>(gate + row * gate_width + at);
            if (gate_bias) {
                const float4 b = *reinterpret_cast<const float4*>(gate_bias + at);
                out.x += b.x; out.y += b.y; out.z += b.z; out.w += b.w;
            }
            out.x = logistic_power<T>(out.x, inv_tau); out.y = logistic_power<T>(out.y, inv_tau);
            out.z = logistic_power<T>(out.z, inv_tau); out.w = logistic_power<T>(out.w, inv_tau);
        }
    } else if (d < (part == 3 ? value_dim : key_dim)) {
        const T* src = proj + row * proj_width + (part == 3 ? v_offset + head * value_dim : (part == 0 ? k_offset : q_offset) + head * key_dim) + d;
        const uint2 raw = *reinterpret_cast<const uint2*>(src);
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        out = make_float4(lo.x, lo.y, hi.x, hi.y);
        if (silu_inputs) out = make_float4(silu_of<T>(out.x), silu_of<T>(out.y), silu_of<T>(out.z), silu_of<T>(out.w));
    }
    *reinterpret_cast<float4*>(prepared + row * n_heads * per_head + item) = out;
}

// ---------------------------------------------------------------- chunk by chunk, bfloat16

// What a chunk of 32 tokens needs beside the state (chunk_walk.cuh), for one head with a decay per key channel.  Eight threads hold two
// tokens' keys and multiply them by the decay of every token that follows, as the state is token by token, so that no logarithm is taken and
// no product can overflow: what they hold at token i times its query is G_ij, what is left at the chunk's end is what the token adds to
// the state.  Out: G, the queries times the decays up to their token and those keys as planes, the chunk's decay of the state.
// Bound by its 60 KB of planes a chunk and by issue: the decays' logarithms and exponentials, and the 528 pairs of tokens by 128
// channels, which are taken two channels an instruction.  (A key a thread loaded its queries and decays from shared memory twice as often.)  The
// sums over the channels of eight tokens are taken together, by halving (seven exchanges for eight sums).  Six blocks on a multiprocessor: 1,531
// tokens of 32 heads on B200 56 us (five, in three waves: 63; a key a thread: 66).  The whole call for 1,024 tokens 97 us, token by token 181.  The error against 64 bits is the
// same: read-out 7.4e-7 over 300 tokens, 1.63e-6 over 2,000 (token by token 7.4e-7, 1.66e-6), state 1.09e-6 and 1.75e-6 (1.08e-6, 1.78e-6).
constexpr int kChunkThreads = 128, kChunkParts = 8;

__global__ void __launch_bounds__(kChunkThreads, 6) linear_attention_chunk_kernel(
    __nv_bfloat16* __restrict__ scores, __nv_bfloat16* __restrict__ queries, __nv_bfloat16* __restrict__ keys, float* __restrict__ decays,
    const __nv_bfloat16* __restrict__ proj, int proj_width, int q_offset, int k_offset, const float* __restrict__ gate, int gate_width,
    const float* __restrict__ gate_bias, float inv_tau, const int* __restrict__ cu_seqlens, int n_rows, int n_heads) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int C = chunk::kTokens, D = chunk::kKeys;
    __shared__ __align__(16) float a_s[C][D], q_s[C][D], g_s[C][C + 1];
    const int tid = threadIdx.x, j0 = tid / kChunkParts * 2, part = tid % kChunkParts, warp = tid >> 5;
    const int head = blockIdx.y, seq = blockIdx.z;
    const int begin = cu_seqlens[seq], row0 = begin + blockIdx.x * C, n_here = min(C, cu_seqlens[seq + 1] - row0);
    if (n_here <= 0) return;

    // decays, queries and keys of tokens j0 and j0 + 1: channels 4 part + 32 r .. + 3 are this thread's, as two pairs (rows beyond
    // the sequence's: no decay, zeros)
    unsigned long long key[2][8];
    float4 bias[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
        bias[r] = gate_bias ? *reinterpret_cast<const float4*>(gate_bias + head * D + 4 * part + 32 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const int j = j0 + o;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int d = 4 * part + 32 * r;
            float4 a = make_float4(1.f, 1.f, 1.f, 1.f), q = make_float4(0.f, 0.f, 0.f, 0.f);
            uint2 kv = make_uint2(0u, 0u);
            if (j < n_here) {
                const size_t row = row0 + j;
                const __nv_bfloat16* src = proj + row * proj_width + (size_t)head * D + d;
                const uint2 qv = *reinterpret_cast<const uint2*>(src + q_offset);
                kv = *reinterpret_cast<const uint2*>(src + k_offset);
                a = *reinterpret_cast<const float4*>(gate + row * gate_width + head * D + d);
                a.x = logistic_power<__nv_bfloat16>(a.x + bias[r].x, inv_tau); a.y = logistic_power<__nv_bfloat16>(a.y + bias[r].y, inv_tau);
                a.z = logistic_power<__nv_bfloat16>(a.z + bias[r].z, inv_tau); a.w = logistic_power<__nv_bfloat16>(a.w + bias[r].w, inv_tau);
                q = make_float4(chunk::low_half(qv.x), chunk::high_half(qv.x), chunk::low_half(qv.y), chunk::high_half(qv.y));
            }
            key[o][2 * r] = pack2(chunk::low_half(kv.x), chunk::high_half(kv.x));
            key[o][2 * r + 1] = pack2(chunk::low_half(kv.y), chunk::high_half(kv.y));
            *reinterpret_cast<float4*>(&a_s[j][d]) = a;
            *reinterpret_cast<float4*>(&q_s[j][d]) = q;
        }
    }
    __syncthreads();

    // G, eight tokens i at a time, from the eight on whose keys this warp holds
    const int first = 8 * warp;
    auto eight = [&](int i0, bool own) {
        float sum[2][8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u;
            unsigned long long dot[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&q_s[i][4 * part + 32 * r]);
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&a_s[i][4 * part + 32 * r]);
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    if (!own || i > j0 + o) {      // (only the decays of tokens behind the key's)
                        key[o][2 * r] = mul2(key[o][2 * r], a.x);
                        key[o][2 * r + 1] = mul2(key[o][2 * r + 1], a.y);
                    }
                    dot[o] = fma2(q.x, key[o][2 * r], dot[o]);
                    dot[o] = fma2(q.y, key[o][2 * r + 1], dot[o]);
                }
            }
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                float x, y;
                unpack2(dot[o], x, y);
                sum[o][u] = x + y;
            }
        }
        // the eight threads' shares: thread p ends up with token i0 + p
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) {
            const bool upper = part & w;
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int u = 0; u < w; ++u) {
                    const float give = upper ? sum[o][u] : sum[o][u + w];
                    const float got = __shfl_xor_sync(0xffffffffu, give, w);
                    sum[o][u] = (upper ? sum[o][u + w] : sum[o][u]) + got;
                }
        }
        g_s[i0 + part][j0] = sum[0][0];
        g_s[i0 + part][j0 + 1] = sum[1][0];
    };
    eight(first, true);
#pragma unroll 1
    for (int i0 = first + 8; i0 < C; i0 += 8) eight(i0, false);

    const long long plane = (long long)n_rows * chunk::kKeyRow, score_plane = (long long)n_rows * chunk::kScoreRow;
    auto store = [&](__nv_bfloat16* planes, int j, int r, float4 v) {
        const chunk::Split lo = chunk::split(v.x, v.y), hi = chunk::split(v.z, v.w);
        __nv_bfloat16* dst = planes + head * 3 * plane + (size_t)(row0 + j) * chunk::kKeyRow + 4 * part + 32 * r;
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(dst + p * plane) = make_uint2(lo.part[p], hi.part[p]);
    };
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float4 k;
            unpack2(key[o][2 * r], k.x, k.y);
            unpack2(key[o][2 * r + 1], k.z, k.w);
            if (j0 + o < n_here) store(keys, j0 + o, r, k);
        }
    __syncthreads();
    // the decays up to each token, a channel a thread, over the decays themselves
    float upto = 1.f;
#pragma unroll 8
    for (int i = 0; i < C; ++i) {
        upto *= a_s[i][tid];
        a_s[i][tid] = upto;
    }
    decays[((chunk::chunk_place(begin, seq) + blockIdx.x) * n_heads + head) * D + tid] = upto;
    __nv_bfloat16* dst = scores + head * 3 * score_plane + (long long)row0 * chunk::kScoreRow;
#pragma unroll
    for (int e = tid; e < C * C / 2; e += kChunkThreads) {
        const int i = e / (C / 2), c = e % (C / 2) * 2;
        if (i < n_here)
            chunk::store_split(dst + i * chunk::kScoreRow + c, score_plane, c <= i ? g_s[i][c] : 0.f, c + 1 <= i ? g_s[i][c + 1] : 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int j = j0 + o, d = 4 * part + 32 * r;
            const float4 q = *reinterpret_cast<const float4*>(&q_s[j][d]), a = *reinterpret_cast<const float4*>(&a_s[j][d]);
            if (j < n_here) store(queries, j, r, make_float4(q.x * a.x, q.y * a.y, q.z * a.z, q.w * a.w));
        }
}

// PER: key channels per lane (a multiple of 4); KP = 16 * PER: the padded key size.  COLS: columns per lane.
template <int PER, int COLS, int KIND>
__global__ void __launch_bounds__(kLanes * kColumns / COLS) linear_attention_kernel(
    float* __restrict__ o, float* __restrict__ state, const float* __restrict__ keys, long long key_stride, int heads_per_unit,
    const float* __restrict__ values, long long value_stride, const float* __restrict__ per_head,
    const int* __restrict__ cu_seqlens, const int* __restrict__ slots, int n_heads, int key_dim, int value_dim, int vp,
    float q_scale) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int KP = kLanes * PER, kStage = stage_tokens(PER), kThreads = kLanes * kColumns / COLS;
    constexpr int PARTS = KIND == kChannelDecay || KIND == kBonusRead ? 3 : 2;     // k, q (and the decay) per token
    constexpr int TAIL = KIND >= kBonusRead ? kRecurrenceTail : 0;
    constexpr int V_AT = PARTS * KP, TAIL_AT = V_AT + kColumns;
    constexpr int ROW = V_AT + kColumns + TAIL;         // floats of one staged token
    constexpr int PIECES = ROW / 4, WARPS = kThreads / 32, PER_LANE = (PIECES + 31) / 32;
    constexpr int SHARE = share_stride(COLS), WARP_COLS = 2 * COLS;
    extern __shared__ __align__(16) float stage_mem[];  // [kBuffers][kStage][ROW], then the shares [kStage][kColumns][SHARE]
    float* shares = stage_mem + (size_t)kBuffers * kStage * ROW;
    const int seq = blockIdx.z, head = blockIdx.y;
    const int col0 = blockIdx.x * kColumns;
    const int lane = threadIdx.x % kLanes, group = threadIdx.x / kLanes;
    const int own_col = col0 + group * COLS;           // this lane's first column
    const int row0 = cu_seqlens[seq], row1 = cu_seqlens[seq + 1];
    if (row0 >= row1) return;
    const int slot = slots[seq];
    float* S = state + ((size_t)slot * n_heads + head) * (size_t)value_dim * key_dim;
    const int unit = head / heads_per_unit, n_units = n_heads / heads_per_unit;
    const size_t key_step = (size_t)n_units * key_stride, value_step = (size_t)n_heads * value_stride;
    const int n_tokens = row1 - row0;
    const int warp = threadIdx.x >> 5, warp_lane = threadIdx.x & 31;

    // a lane's pieces of a token: where each lies in its row, and how far apart rows are
    const float* piece_src[PER_LANE];
    size_t piece_step[PER_LANE];
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int c = (warp_lane + 32 * j) * 4;
        if (c < V_AT) {
            piece_src[j] = keys + ((size_t)row0 * n_units + unit) * key_stride + c;
            piece_step[j] = key_step;
        } else {
            piece_src[j] = values + ((size_t)row0 * n_heads + head) * value_stride +
                           (TAIL != 0 && c >= TAIL_AT ? vp + (c - TAIL_AT) : col0 + (c - V_AT));
            piece_step[j] = value_step;
        }
    }
    auto issue = [&](int stage) {
        const int first = stage * kStage, n = min(kStage, n_tokens - first);
        float* dst = stage_mem + (size_t)(stage % kBuffers) * kStage * ROW + warp_lane * 4;
        for (int t = warp; t < n; t += WARPS) {
#pragma unroll
            for (int j = 0; j < PER_LANE; ++j)
                if (32 * (j + 1) <= PIECES || warp_lane + 32 * j < PIECES)
                    copy16_async(dst + t * ROW + 128 * j, piece_src[j] + (size_t)(first + t) * piece_step[j]);
        }
    };
    const int n_stages = (n_tokens + kStage - 1) / kStage;
#pragma unroll
    for (int i = 0; i < kBuffers - 1; ++i) {
        if (i < n_stages) issue(i);
        copy_commit();
    }

    const bool whole = key_dim % 4 == 0 && ((uintptr_t)state & 15) == 0;
    float s[COLS][PER];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        const float* src = S + (size_t)min(own_col + c, value_dim - 1) * key_dim;     // idle columns mirror the last one and store nothing
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
            const int d = (i / 4) * (4 * kLanes) + lane * 4;
            if (whole) {                      // a run of four is inside the key or outside as a whole
                const float4 x = d < key_dim ? *reinterpret_cast<const float4*>(src + d) : make_float4(0.f, 0.f, 0.f, 0.f);
                s[c][i] = x.x; s[c][i + 1] = x.y; s[c][i + 2] = x.z; s[c][i + 3] = x.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) s[c][i + j] = d + j < key_dim ? src[d + j] : 0.f;
            }
        }
    }
    const float own = per_head != nullptr ? per_head[head] : 0.f;      // the constant decay, or the skip's factor

    // one token: the sums of its read-out over this lane's channels, and the state behind it
    auto advance = [&](const float* tok, float (&sums)[COLS]) {
        float v[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            v[c] = tok[V_AT + group * COLS + c];
            sums[c] = 0.f;
        }
        float decay = own;
        if (KIND == kSteppedDecay) {
            const float2 tail = *reinterpret_cast<const float2*>(tok + TAIL_AT);
            decay = tail.x;
#pragma unroll
            for (int c = 0; c < COLS; ++c) v[c] *= tail.y;
        }
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
            const int d = (i / 4) * (4 * kLanes) + lane * 4;
            const float4 k = *reinterpret_cast<const float4*>(tok + d);
            const float4 q = *reinterpret_cast<const float4*>(tok + KP + d);
            float4 a = make_float4(decay, decay, decay, decay);
            if (PARTS == 3) a = *reinterpret_cast<const float4*>(tok + 2 * KP + d);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                float* x = s[c] + i;
                if (KIND == kBonusRead) sums[c] += x[0] * q.x + x[1] * q.y + x[2] * q.z + x[3] * q.w;
                x[0] = fmaf(a.x, x[0], k.x * v[c]);      // (one multiply-add links a token's state to the next)
                x[1] = fmaf(a.y, x[1], k.y * v[c]);
                x[2] = fmaf(a.z, x[2], k.z * v[c]);
                x[3] = fmaf(a.w, x[3], k.w * v[c]);
                if (KIND != kBonusRead) sums[c] += x[0] * q.x + x[1] * q.y + x[2] * q.z + x[3] * q.w;
            }
        }
    };
    float* own_share = shares + (size_t)group * COLS * SHARE + lane;

    for (int stage = 0; stage < n_stages; ++stage) {
        copy_wait<kBuffers - 2>();
        __syncthreads();                     // this stage has landed; the buffer of the one before it is free again
        if (stage + kBuffers - 1 < n_stages) issue(stage + kBuffers - 1);
        copy_commit();
        const float* src = stage_mem + (size_t)(stage % kBuffers) * kStage * ROW;
        const int first = stage * kStage, n = min(kStage, n_tokens - first);
        int t0 = 0;
#pragma unroll 1
        for (; t0 + kGroup <= n; t0 += kGroup) {
            float part[kGroup][COLS];
#pragma unroll
            for (int t = 0; t < kGroup; ++t) advance(src + (t0 + t) * ROW, part[t]);
#pragma unroll
            for (int t = 0; t < kGroup; ++t)
#pragma unroll
                for (int c = 0; c < COLS; ++c) own_share[(size_t)((t0 + t) * kColumns + c) * SHARE] = part[t][c];
        }
#pragma unroll 1
        for (; t0 < n; ++t0) {
            float part[COLS];
            advance(src + t0 * ROW, part);
#pragma unroll
            for (int c = 0; c < COLS; ++c) own_share[(size_t)(t0 * kColumns + c) * SHARE] = part[c];
        }
        __syncwarp();
        // the stage's read-outs: this warp's columns, a (token, column) pair per lane and turn
        for (int i = warp_lane; i < n * WARP_COLS; i += 32) {
            const int t = i / WARP_COLS, c = warp * WARP_COLS + i % WARP_COLS;
            const float* share = shares + (size_t)(t * kColumns + c) * SHARE;
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < kLanes; l += 4) {
                const float4 x = *reinterpret_cast<const float4*>(share + l);
                sum += (x.x + x.y) + (x.z + x.w);
            }
            if (col0 + c < value_dim) {
                const float* tok = src + t * ROW;
                float y = sum * q_scale;
                if (KIND == kBonusRead) y += tok[TAIL_AT] * tok[V_AT + c];
                if (KIND == kSteppedDecay) y += own * tok[V_AT + c];
                o[((size_t)(row0 + first + t) * n_heads + head) * value_dim + col0 + c] = y;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        if (own_col + c >= value_dim) break;
        float* dst = S + (size_t)(own_col + c) * key_dim;
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
            const int d = (i / 4) * (4 * kLanes) + lane * 4;
            if (whole) {
                if (d < key_dim) *reinterpret_cast<float4*>(dst + d) = make_float4(s[c][i], s[c][i + 1], s[c][i + 2], s[c][i + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (d + j < key_dim) dst[d + j] = s[c][i + j];
            }
        }
    }
}

template <int PER, int COLS, int KIND>
void launch_one(const RecurrenceArgs& a, cudaStream_t stream) {
    constexpr int KP = kLanes * PER, kStage = stage_tokens(PER);
    constexpr int ROW = (KIND == kChannelDecay || KIND == kBonusRead ? 3 : 2) * KP + kColumns + (KIND >= kBonusRead ? kRecurrenceTail : 0);
    const size_t smem = (size_t)kStage * (kBuffers * ROW + kColumns * share_stride(COLS)) * sizeof(float);
    const dim3 grid((a.value_dim + kColumns - 1) / kColumns, a.n_heads, a.n_seqs);
    auto kernel = linear_attention_kernel<PER, COLS, KIND>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    thn_launch_ordered(kernel, grid, kLanes * kColumns / COLS, smem, stream, a.o, a.state, a.keys, a.key_stride, a.n_heads / a.key_units,
                       a.values, a.value_stride, a.per_head, a.cu_seqlens, a.slots, a.n_heads, a.key_dim, a.value_dim,
                       padded_values(a.value_dim), a.q_scale);
}

int g_columns = 0;      // columns per lane for keys up to 128: 1, 2, 4, or 0: the default

template <int PER, int KIND>
void launch_columns(const RecurrenceArgs& a, int columns, cudaStream_t stream) {
    if (columns == 4) launch_one<PER, 4, KIND>(a, stream);
    else if (columns == 2) launch_one<PER, 2, KIND>(a, stream);
    else launch_one<PER, 1, KIND>(a, stream);
}

template <int KIND>
void launch_kind(const RecurrenceArgs& a, cudaStream_t stream) {
    // Four columns a lane load less per multiply-add, two leave twice as many warps: with fewer than 256
    // blocks the latter win (one prompt of 2,048 tokens, 32 heads of 64: 208 against 263 us; four of them 618
    // against 607; 64 heads of 64 over a state of 128: 366 against 364 us, four prompts 1,322 against 1,171).
    const long long blocks = (long long)(padded_values(a.value_dim) / kColumns) * a.n_heads * a.n_seqs;
    const int columns = g_columns ? g_columns : blocks >= 256 ? 4 : 2;
    switch (recurrence_per_lane(a.key_dim)) {
        case 4: return launch_columns<4, KIND>(a, columns, stream);
        case 8: return launch_columns<8, KIND>(a, columns, stream);
        case 16: return launch_one<16, 2, KIND>(a, stream);
        default: return launch_one<32, 1, KIND>(a, stream);
    }
}

template <typename T>
int launch(float* o, float* state, float* prepared, const void* proj, int proj_width, int q_offset, int k_offset, int v_offset,
           const float* decay, const float* gate, int gate_width, const float* gate_bias, float inv_tau,
           const int* cu_seqlens, const int* slots, int n_rows, int n_seqs, int n_heads, int key_dim, int value_dim,
           float q_scale, int mode, int silu_inputs, cudaStream_t stream) {
    const int kp = padded_keys(key_dim), vp = padded_values(value_dim), parts = key_parts(mode), per_head = parts * kp + vp;
    const long long n = (long long)n_rows * n_heads * per_head;
    const long long blocks = ((long long)n_heads * per_head / 4 + 255) / 256;
    // (a quarter of the threads, each with four entries one behind the other: not where few rows leave the chip empty.  The whole call with
    // gated decays in us, an entry / four entries a thread: 16 heads, 1 row 3.8 / 4.2, 4 rows 5.5 / 5.6, 8 rows 7.9 / 8.0, 16 rows
    // 12.4 / 12.3; 32 heads, 4 rows 7.8 / 7.9, 8 rows 12.3 / 12.1, 64 tokens 18.1 / 14.9.  The results are the same to the bit.)
    if (sizeof(T) == 2 && (long long)n_rows * n_heads >= 256 && (key_dim | value_dim | proj_width | q_offset | k_offset | v_offset | gate_width) % 4 == 0 && blocks <= 65535 &&
        ((uintptr_t)proj & 7) == 0 && (((uintptr_t)gate | (uintptr_t)gate_bias) & 15) == 0)
        thn_launch(linear_attention_prepare_vec_kernel, dim3(n_rows, (unsigned)blocks), 256, 0, stream, prepared, (const __nv_bfloat16*)proj,
                   proj_width, q_offset, k_offset, v_offset, gate, gate_width, gate_bias, inv_tau, n_heads, key_dim, value_dim, kp, vp,
                   parts, silu_inputs);
    else
        thn_launch(linear_attention_prepare_kernel<T>, (unsigned)((n + 255) / 256), 256, 0, stream, prepared, (const T*)proj,
               proj_width, q_offset, k_offset, v_offset, gate, gate_width, gate_bias, inv_tau, n, n_heads, key_dim, value_dim, kp,
               vp, parts, silu_inputs);
    return launch_recurrence(mode, RecurrenceArgs{o, state, prepared, per_head, n_heads, prepared + parts * kp, per_head, decay,
                                                  cu_seqlens, slots, n_seqs, n_heads, key_dim, value_dim, q_scale},
                             stream);
}

}  // namespace

// How many columns of S a lane holds, for keys up to 128 (tests and measurement): 1, 2, 4, or 0: the default.
THN_API void thn_set_recurrence_columns(int columns) { g_columns = columns == 1 || columns == 2 || columns == 4 ? columns : 0; }

int launch_recurrence(int kind, const RecurrenceArgs& args, cudaStream_t stream) {
    THN_CHECK_ARG(args.key_units > 0 && args.n_heads % args.key_units == 0, "recurrence: %d heads over %d units of keys",
                  args.n_heads, args.key_units);
    THN_UNSUPPORTED_IF(args.key_dim > 512, "recurrence: keys of %d, at most 512", args.key_dim);
    THN_UNSUPPORTED_IF(args.n_heads > 65535 || args.n_seqs > 65535, "recurrence: %d heads, %d sequences", args.n_heads, args.n_seqs);
    THN_CHECK_ARG((((uintptr_t)args.keys | (uintptr_t)args.values) & 15) == 0 && args.key_stride % 4 == 0 && args.value_stride % 4 == 0,
                  "recurrence: prepared rows are not 16-byte aligned");
    switch (kind) {
        case kConstantDecay: launch_kind<kConstantDecay>(args, stream); break;
        case kChannelDecay: launch_kind<kChannelDecay>(args, stream); break;
        case kBonusRead: launch_kind<kBonusRead>(args, stream); break;
        case kSteppedDecay: launch_kind<kSteppedDecay>(args, stream); break;
        default: THN_CHECK_ARG(false, "recurrence: unknown kind %d", kind);
    }
    return thn_launch_status("recurrence");
}

// Floats of the scratch that thn_linear_attention needs for a step of n_rows rows.
THN_API long long thn_linear_attention_scratch_floats(int n_rows, int n_heads, int key_dim, int value_dim, int mode) {
    return (long long)n_rows * n_heads * ((mode == 1 ? 3 : 2) * (long long)padded_keys(key_dim) + padded_values(value_dim));
}

// o float32 [rows, heads, value_dim]; state float32 [slots, heads, value_dim, key_dim], read and
// updated; proj [rows, proj_width] of the activation type with q, k (heads * key_dim each) and v
// (heads * value_dim) from the given columns; mode 0: decay float32 [heads]; mode 1: gate float32
// [rows, gate_width] (the first heads * key_dim columns), gate_bias float32 [heads * key_dim] or
// null, tau > 0.  The tokens of sequence i are the rows [cu_seqlens[i], cu_seqlens[i + 1]) of the
// step's n_rows rows.  scratch: float32, thn_linear_attention_scratch_floats(...) entries, 16-byte aligned.
THN_API int thn_linear_attention(float* o, float* state, float* scratch, const void* proj, int proj_width, int q_offset, int k_offset,
                                 int v_offset, const float* decay, const float* gate, int gate_width,
                                 const float* gate_bias, float tau, const int* cu_seqlens, const int* slots, int n_rows,
                                 int n_seqs, int n_heads, int key_dim, int value_dim, float q_scale, int mode, int silu_inputs,
                                 int dtype, cudaStream_t stream) {
    THN_CHECK_ARG(n_seqs >= 0 && n_heads > 0 && key_dim > 0 && value_dim > 0, "linear_attention: bad sizes");
    THN_UNSUPPORTED_IF(key_dim > 512, "linear_attention: keys of %d, at most 512", key_dim);
    THN_UNSUPPORTED_IF(n_heads > 65535 || n_seqs > 65535, "linear_attention: %d heads, %d sequences", n_heads, n_seqs);
    THN_CHECK_ARG(mode == 0 ? decay != nullptr : (mode == 1 && gate != nullptr && tau > 0.f && gate_width >= n_heads * key_dim),
                  "linear_attention: decay mode %d without its operands", mode);
    THN_CHECK_ARG(q_offset >= 0 && k_offset >= 0 && v_offset >= 0 && q_offset + n_heads * key_dim <= proj_width &&
                      k_offset + n_heads * key_dim <= proj_width && v_offset + n_heads * value_dim <= proj_width,
                  "linear_attention: q, k, v do not lie inside rows of %d", proj_width);
    THN_CHECK_ARG(scratch != nullptr && ((uintptr_t)scratch & 15) == 0 && n_rows >= 0, "linear_attention: scratch missing or unaligned");
    if (n_seqs == 0 || n_rows == 0) return THN_OK;
    const float inv_tau = mode == 1 ? 1.0f / tau : 0.f;
    if (dtype == THN_F32)
        return launch<float>(o, state, scratch, proj, proj_width, q_offset, k_offset, v_offset, decay, gate, gate_width, gate_bias,
                             inv_tau, cu_seqlens, slots, n_rows, n_seqs, n_heads, key_dim, value_dim, q_scale, mode, silu_inputs,
                             stream);
    if (dtype == THN_BF16)
        return launch<__nv_bfloat16>(o, state, scratch, proj, proj_width, q_offset, k_offset, v_offset, decay, gate, gate_width,
                                     gate_bias, inv_tau, cu_seqlens, slots, n_rows, n_seqs, n_heads, key_dim, value_dim, q_scale,
                                     mode, silu_inputs, stream);
    THN_CHECK_ARG(false, "linear_attention: unknown dtype %d", dtype);
    return THN_OK;
}

// Bytes of the scratch that thn_linear_attention_chunks needs.
THN_API long long thn_linear_attention_chunks_scratch_bytes(int n_rows, int n_seqs, int n_heads) {
    return (long long)n_heads * n_rows * 3 * (2 * chunk::kKeyRow + chunk::kScoreRow) * 2 + chunk::chunk_places(n_rows, n_seqs) * n_heads * chunk::kKeys * 4;
}

// Which blocks walk the chunks (WalkCost): 1 has 16 columns and four warps, which split the keys; 2: 32, four for a group of 16; 3: 64, two; 4: as 3, two
// blocks on a multiprocessor with one buffer each, into which the warps copy themselves.  us of the whole call, 1 / 2 / 3 / 4, 16 heads of 128: one prompt of
// 2,048 tokens 125 / 149 / 215 / 285, 33 tokens beside 60 single ones 153 / 109 / 90 / 78, 512 beside 60 187 / 137 / 112 / 114, 3 x 512 91 / 85 / 74 / 92, 8 x 512
// 229 / 193 / 171 / 178; 32 heads, one prompt of 128 tokens 30 / 32 / 27 / 29.  Over 882 steps of 4 to 64 heads the chosen one takes 1.3 % longer than the best of four.
constexpr chunk::WalkCost kWalkCosts[4] = {{2.89f, 1.30f, 7.64f, 6.67f, 0.22f, 16, 1}, {3.90f, 1.60f, 5.65f, 4.09f, 0.41f, 32, 1},
                                           {4.55f, 2.51f, 4.77f, 2.96f, 0.50f, 64, 1}, {7.53f, 3.23f, 4.59f, 1.11f, 0.99f, 64, 2}};

THN_API int thn_linear_attention_walk_shape(int n_rows, int max_tokens, int n_seqs, int n_heads, int value_dim) {
    return chunk::cheapest_walk(kWalkCosts, n_rows, max_tokens, n_seqs, n_heads, value_dim);
}

// The recurrence of a step with gated decays chunk by chunk: bfloat16 rows as thn_linear_attention takes them (no silu), keys of
// 128, values of whole groups of 16; v's columns start on 16-byte boundaries, q's and k's on 8-byte ones, gate and its bias on
// 16-byte ones; max_tokens: the most rows of a sequence.  shape: 0, or which blocks walk (tests and measurement); with 16 added a brought
// walk brings nothing, so that its wait runs out (for the test of the wait only).
THN_API int thn_linear_attention_chunks(float* o, float* state, void* scratch, long long scratch_bytes, const void* proj, int proj_width,
                                        int q_offset, int k_offset, int v_offset, const float* gate, int gate_width, const float* gate_bias, float tau,
                                        const int* cu_seqlens, const int* slots, int n_rows, int max_tokens, int n_seqs, int n_heads,
                                        int key_dim, int value_dim, float q_scale, int shape, int* err, cudaStream_t stream) {
    THN_CHECK_ARG(n_seqs >= 0 && n_heads > 0 && gate != nullptr && tau > 0.f && gate_width >= n_heads * key_dim, "linear_attention_chunks: bad sizes");
    THN_UNSUPPORTED_IF(key_dim != chunk::kKeys || value_dim <= 0 || value_dim % 16 != 0 || proj_width % 8 != 0 || v_offset % 8 != 0 ||
                           (q_offset | k_offset | gate_width) % 4 != 0,
                       "linear_attention_chunks: keys of %d, values of %d, rows of %d, columns %d, %d, %d", key_dim, value_dim, proj_width,
                       q_offset, k_offset, v_offset);
    THN_CHECK_ARG(q_offset >= 0 && k_offset >= 0 && v_offset >= 0 && q_offset + n_heads * key_dim <= proj_width &&
                      k_offset + n_heads * key_dim <= proj_width && v_offset + n_heads * value_dim <= proj_width,
                  "linear_attention_chunks: q, k, v do not lie inside rows of %d", proj_width);
    THN_UNSUPPORTED_IF(n_heads > 65535 || n_seqs > 65535, "linear_attention_chunks: %d heads, %d sequences", n_heads, n_seqs);
    THN_CHECK_ARG(scratch && (((uintptr_t)state | (uintptr_t)scratch | (uintptr_t)proj | (uintptr_t)gate | (uintptr_t)gate_bias) & 15) == 0,
                  "linear_attention_chunks: operands are not 16-byte aligned");
    if (n_seqs == 0 || n_rows <= 0 || max_tokens <= 0) return THN_OK;
    const long long need = thn_linear_attention_chunks_scratch_bytes(n_rows, n_seqs, n_heads);
    THN_CHECK_ARG(scratch_bytes >= need, "linear_attention_chunks: %lld bytes of scratch, %lld needed", scratch_bytes, need);
    const int chunks = (max_tokens + chunk::kTokens - 1) / chunk::kTokens;
    const size_t plane = (size_t)n_rows * chunk::kKeyRow;
    __nv_bfloat16* queries = static_cast<__nv_bfloat16*>(scratch);
    __nv_bfloat16* keys = queries + 3 * n_heads * plane;
    __nv_bfloat16* scores = keys + 3 * n_heads * plane;
    float* decays = reinterpret_cast<float*>(scores + (size_t)3 * n_heads * n_rows * chunk::kScoreRow);
    const __nv_bfloat16* rows = static_cast<const __nv_bfloat16*>(proj);
    cudaFuncSetAttribute(linear_attention_chunk_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    thn_launch(linear_attention_chunk_kernel, dim3(chunks, n_heads, n_seqs), kChunkThreads, 0, stream, scores, queries, keys, decays, rows,
               proj_width, q_offset, k_offset, gate, gate_width, gate_bias, 1.0f / tau, cu_seqlens, n_rows, n_heads);
    chunk::WalkArgs a{};
    a.err = err;
    a.skip_loads = shape & 16;
    shape &= 15;
    a.o = o; a.state = state;
    a.q = queries; a.k = keys;
    a.key_plane = plane; a.key_unit = 3 * plane; a.key_row = chunk::kKeyRow;
    a.v = rows + v_offset; a.v_row = proj_width; a.v_head = value_dim;
    a.scores = scores; a.key_sums = decays;
    a.cu_seqlens = cu_seqlens; a.slots = slots;
    a.n_rows = n_rows; a.n_heads = n_heads; a.heads_per_unit = 1; a.value_dim = value_dim; a.scale = q_scale;
    using T = __nv_bfloat16;
    using namespace chunk;
    if (shape == 0) shape = thn_linear_attention_walk_shape(n_rows, max_tokens, n_seqs, n_heads, value_dim);
    if (value_dim % 64 != 0) shape = std::min(shape, 2);
    if (value_dim % 32 != 0) shape = 1;
    if (shape == 4) launch_walk<T, 4, 2, kPerKey, 1, false>(a, n_seqs, stream);
    else if (shape == 3) launch_brought_walk<T, 4, 2, kPerKey>(a, n_seqs, stream);
    else if (shape == 2) launch_brought_walk<T, 2, 4, kPerKey>(a, n_seqs, stream);
    else launch_brought_walk<T, 1, 4, kPerKey>(a, n_seqs, stream);
    return thn_launch_status("linear_attention_chunks");
}
