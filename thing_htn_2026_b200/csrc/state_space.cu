// State-space duality (Mamba-2): a recurrent token mixer.  Per head a matrix S [state, vdim], zero at a
// sequence's start, and for every token with an input x (vdim entries per head), B and C (state
// entries, shared by a group of neighbouring heads), one step size t and one decay a per head:
//
//     t = softplus(t_pre + bias_h)       a = exp(-rate_h t)
//     S <- a S + (t B) x^T               y = S^T C + D_h x
//
// x, B and C come out of one short causal convolution per channel with a bias and silu; the raw
// inputs of a sequence's last `taps` tokens stay in a ring [taps, channels], position p at p mod taps.
//
//   state_space_prepare   convolution, silu, step sizes and decays of a prompt's rows, into float32 rows
//                    for the shared recurrence (linear_attention.cuh, kSteppedDecay): [B | C] per row
//                    and group, [x | a, t] per row and head.  A thread takes four neighbouring
//                    channels over a run of rows, keeping the last raw inputs in registers.
//   state_space_prepare_chunks, state_space_chunk, and the walk of chunk_walk.cuh   the same for long bfloat16
//                    prompts over a state of 128, chunk by chunk.
//   state_space_decode    a single token per sequence: convolution, ring, step size, decay, recurrence
//                    and skip in one kernel, one block per (row, head).
//   gated_group_norm   y silu(z), divided by its root mean square over equal consecutive parts, times a
//                    gain: the gate comes before the norm.
//
// float32 after the loads; with float32 activations the exponentials and logarithms are computed in
// double and rounded once (exp_of, silu_of, softplus_of in common.cuh).
#include <math.h>

#include "chunk_walk.cuh"
#include "conv_run.cuh"
#include "linear_attention.cuh"

namespace {

constexpr int kRunRows = 8;          // rows per thread of the prepare kernel
constexpr int kPrepareThreads = 128;

struct SpaceShape {
    int n_heads, vdim, n_state, n_groups, taps;
    __host__ __device__ int inner() const { return n_heads * vdim; }
    __host__ __device__ int channels() const { return n_heads * vdim + 2 * n_groups * n_state; }
};

template <typename T> __device__ __forceinline__ float4 load_four(const T* p);
template <> __device__ __forceinline__ float4 load_four<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load_four<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> __device__ __forceinline__ float4 load_up_to_four(const T* p, int n, bool vec) {
    if (vec) return load_four<T>(p);
    return make_float4(n > 0 ? to_f32<T>(p[0]) : 0.f, n > 1 ? to_f32<T>(p[1]) : 0.f, n > 2 ? to_f32<T>(p[2]) : 0.f,
                       n > 3 ? to_f32<T>(p[3]) : 0.f);
}
__device__ __forceinline__ void add_scaled(float4& acc, const float4& w, const float4& v) {
    acc.x += w.x * v.x; acc.y += w.y * v.y; acc.z += w.z * v.z; acc.w += w.w * v.w;
}

// keys [rows][groups][B: kp | C: kp], values [rows][heads][x: vp | a, t, 0, 0].  Work items of a row:
// heads * vp / 4 pieces of x, groups * 2 * kp / 4 pieces of B and C, one tail per head.
// TAPS 0: any number, every raw input loaded where it is used.
template <typename T, int TAPS>
__global__ void __launch_bounds__(kPrepareThreads) state_space_prepare_kernel(
    float* __restrict__ keys, float* __restrict__ values, const T* __restrict__ proj, int proj_width, int offset,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b, const T* __restrict__ ring,
    const float* __restrict__ dt_pre, const float* __restrict__ dt_bias, const float* __restrict__ rate,
    const int* __restrict__ row_slot, const int* __restrict__ row_pos, const int* __restrict__ seq_lens, int n_rows,
    SpaceShape shape, int kp, int vp, int vec) {
    pdl_launch_dependents();
    pdl_wait();
    const int taps = TAPS > 0 ? TAPS : shape.taps;
    const int x_items = shape.n_heads * (vp / 4), bc_items = shape.n_groups * 2 * (kp / 4);
    const int item = blockIdx.x * kPrepareThreads + threadIdx.x;
    const int first_row = blockIdx.y * kRunRows, last_row = min(first_row + kRunRows, n_rows);
    const int value_stride = vp + kRecurrenceTail, channels = shape.channels();
    if (item >= x_items + bc_items + shape.n_heads) return;
    if (item >= x_items + bc_items) {                       // a head's step sizes and decays
        const int head = item - x_items - bc_items;
        const float bias = dt_bias[head], r = rate[head];
        for (int m = first_row; m < last_row; ++m) {
            const float t = softplus_of<T>(dt_pre[(size_t)m * shape.n_heads + head] + bias);
            *reinterpret_cast<float4*>(values + ((size_t)m * shape.n_heads + head) * value_stride + vp) =
                make_float4(exp_of<T>(-r * t), t, 0.f, 0.f);
        }
        return;
    }
    int channel, n;                                         // first source channel, how many of the four exist
    float* dst;
    size_t dst_stride;
    if (item < x_items) {
        const int head = item / (vp / 4), d = (item - head * (vp / 4)) * 4;
        channel = head * shape.vdim + d;
        n = shape.vdim - d;
        dst = values + (size_t)head * value_stride + d;
        dst_stride = (size_t)shape.n_heads * value_stride;
    } else {
        const int unit = (item - x_items) / (kp / 4), d = ((item - x_items) - unit * (kp / 4)) * 4;   // unit = group * 2 + which
        const int group = unit >> 1, which = unit & 1;
        channel = shape.inner() + (which * shape.n_groups + group) * shape.n_state + d;
        n = shape.n_state - d;
        dst = keys + (size_t)unit * kp + d;
        dst_stride = (size_t)shape.n_groups * 2 * kp;
    }
    dst += (size_t)first_row * dst_stride;
    if (n <= 0) {
        for (int m = first_row; m < last_row; ++m, dst += dst_stride) *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const bool whole = vec && n >= 4;
    const float4 bias = load_up_to_four<float>(conv_b + channel, n, false);
    // a channel's taps are consecutive: four channels' weights for one tap are `taps` apart
    auto weight_of = [&](int j) {
        const float* w = conv_w + (size_t)channel * taps + j;
        return make_float4(w[0], n > 1 ? w[taps] : 0.f, n > 2 ? w[2 * taps] : 0.f, n > 3 ? w[3 * taps] : 0.f);
    };
    // the raw input `back` tokens before row m: from the step's rows, from the ring, or zero
    auto raw_of = [&](int m, int pos, int local, int slot, int back) {
        if (back > pos) return make_float4(0.f, 0.f, 0.f, 0.f);
        if (back <= local) return load_up_to_four<T>(proj + (size_t)(m - back) * proj_width + offset + channel, n, whole);
        return load_up_to_four<T>(ring + ((size_t)slot * taps + (pos - back) % taps) * channels + channel, n, whole);
    };
    constexpr int HELD = TAPS > 0 ? TAPS : 1;
    float4 w[HELD], past[HELD];                              // past[j]: the raw input TAPS - 1 - j tokens back
    if (TAPS > 0) {
#pragma unroll
        for (int j = 0; j < HELD; ++j) w[j] = weight_of(j);
    }
    for (int m = first_row; m < last_row; ++m, dst += dst_stride) {
        const int slot = row_slot[m], pos = row_pos[m];
        const int local = pos - seq_lens[slot];
        float4 acc = bias;
        if (TAPS > 0) {
            if (m == first_row || local == 0) {
#pragma unroll
                for (int j = 0; j < HELD - 1; ++j) past[j] = raw_of(m, pos, local, slot, HELD - 1 - j);
            } else {
#pragma unroll
                for (int j = 0; j < HELD - 1; ++j) past[j] = past[j + 1];
            }
            past[HELD - 1] = raw_of(m, pos, local, slot, 0);
#pragma unroll
            for (int j = 0; j < HELD; ++j) add_scaled(acc, w[j], past[j]);
        } else {
            for (int j = 0; j < taps; ++j) add_scaled(acc, weight_of(j), raw_of(m, pos, local, slot, taps - 1 - j));
        }
        *reinterpret_cast<float4*>(dst) = make_float4(silu_of<T>(acc.x), n > 1 ? silu_of<T>(acc.y) : 0.f,
                                                      n > 2 ? silu_of<T>(acc.z) : 0.f, n > 3 ? silu_of<T>(acc.w) : 0.f);
    }
}

// The same for the walk in chunks (bfloat16, four taps, a state of 128, whole groups of four entries): the raw inputs
// ahead of a thread's rows are loaded together (conv_run.cuh; 4,096 rows of 10,240 channels on B200: 80 us, 130 above), B and C go out in three planes of bfloat16 (chunk_walk.cuh)
// [group][B | C][plane][rows][kKeyRow], x as [heads][rows][vdim], the step sizes as [heads][rows].
constexpr int kChunkTaps = 4;

__global__ void __launch_bounds__(kPrepareThreads, 6) state_space_prepare_chunks_kernel(
    __nv_bfloat16* __restrict__ planes, float* __restrict__ values, float* __restrict__ steps, const __nv_bfloat16* __restrict__ proj,
    int proj_width, int offset, const float* __restrict__ conv_w, const float* __restrict__ conv_b,
    const __nv_bfloat16* __restrict__ ring, const float* __restrict__ dt_pre, const float* __restrict__ dt_bias,
    const int* __restrict__ row_slot, const int* __restrict__ row_pos, const int* __restrict__ seq_lens, int n_rows, SpaceShape shape) {
    pdl_launch_dependents();
    const int item = blockIdx.x * kPrepareThreads + threadIdx.x;
    const int C = shape.channels(), c = item * 4;
    const int first = blockIdx.y * kRunRows, n_here = min(kRunRows, n_rows - first);
    if (c >= C) {
        const int head = item - C / 4;
        if (head >= shape.n_heads) return;
        pdl_wait();
        for (int r = 0; r < n_here; ++r)
            steps[(size_t)head * n_rows + first + r] = softplus_of<__nv_bfloat16>(dt_pre[(size_t)(first + r) * shape.n_heads + head] + dt_bias[head]);
        return;
    }
    float w[4][kChunkTaps], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(conv_w + (size_t)(c + i) * kChunkTaps);
        w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
        b[i] = conv_b[c + i];
    }
    pdl_wait();
    const bool is_value = c < shape.inner();
    const int kc = is_value ? 0 : c - shape.inner(), which = kc / (shape.n_groups * chunk::kKeys), in_part = kc % (shape.n_groups * chunk::kKeys);
    const long long plane = (long long)n_rows * chunk::kKeyRow;
    __nv_bfloat16* key_dst = planes + ((in_part / chunk::kKeys) * 2 + which) * 3 * plane + (long long)first * chunk::kKeyRow + in_part % chunk::kKeys;
    float* value_dst = values + ((size_t)(is_value ? c / shape.vdim : 0) * n_rows + first) * shape.vdim + (is_value ? c % shape.vdim : 0);
    const conv_run::Source source{proj + (size_t)first * proj_width + offset + c, proj_width, ring + c, C, row_slot, row_pos, seq_lens};
    conv_run::run<kRunRows, false>(source, first, n_here, w, b, [&](int r, const float (&y)[4]) {
        if (is_value) {
            *reinterpret_cast<float4*>(value_dst + (size_t)r * shape.vdim) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
            const chunk::Split lo = chunk::split(y[0], y[1]), hi = chunk::split(y[2], y[3]);
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint2*>(key_dst + p * plane + (long long)r * chunk::kKeyRow) = make_uint2(lo.part[p], hi.part[p]);
        }
    });
}

// What a chunk of 32 tokens needs beside the state, for all heads of a group: G_ij = exp(c_i - c_j) t_j C_i . B_j with
// c the sum of the chunk's log decays -rate t (in double), plus the skip's factor on the diagonal; per token
// (exp(c_i), -, t_i exp(c_last - c_i), -).  One block per (chunk, group, sequence): two warps take the products, then
// each warp's lanes are the tokens j of some of the group's heads.
constexpr int kSpaceThreads = 256;
__global__ void __launch_bounds__(kSpaceThreads) state_space_chunk_kernel(
    __nv_bfloat16* __restrict__ scores, float4* __restrict__ scalars, const __nv_bfloat16* __restrict__ planes,
    const float* __restrict__ steps, const float* __restrict__ rate, const float* __restrict__ skip, const int* __restrict__ cu_seqlens,
    int n_rows, int heads_per_group) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int C = chunk::kTokens, kPlane = C * chunk::kKeyRow;
    extern __shared__ __align__(16) unsigned char space_mem[];
    __nv_bfloat16* b_s = reinterpret_cast<__nv_bfloat16*>(space_mem);      // [3][C][kKeyRow]
    __nv_bfloat16* c_s = b_s + 3 * kPlane;                                 // [3][C][kKeyRow]
    float* dot_s = reinterpret_cast<float*>(c_s + 3 * kPlane);             // [C][C + 1]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int group = blockIdx.y, seq = blockIdx.z;
    const int begin = cu_seqlens[seq], row0 = begin + blockIdx.x * C, n_here = min(C, cu_seqlens[seq + 1] - row0);
    if (n_here <= 0) return;
    const long long plane = (long long)n_rows * chunk::kKeyRow, at0 = (long long)row0 * chunk::kKeyRow;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        chunk::copy_rows<chunk::kKeyRow, kSpaceThreads>(b_s + p * kPlane, planes + ((long long)group * 6 + p) * plane + at0, n_here);
        chunk::copy_rows<chunk::kKeyRow, kSpaceThreads>(c_s + p * kPlane, planes + ((long long)group * 6 + 3 + p) * plane + at0, n_here);
    }
    chunk::copy_commit();
    chunk::copy_wait_all();
    __syncthreads();
    if (warp < 2) {
        float dot[4][4];
        chunk::dots<3>(dot, c_s, b_s, warp, lane);
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) dot_s[(16 * warp + g + 8 * (i >> 1)) * (C + 1) + 8 * n + 2 * t + (i & 1)] = dot[n][i];
    }
    __syncthreads();
    const long long score_plane = (long long)n_rows * chunk::kScoreRow;
    for (int h = warp; h < heads_per_group; h += kSpaceThreads / 32) {
        const int head = group * heads_per_group + h;
        const bool there = lane < n_here;
        const float step = there ? steps[(size_t)head * n_rows + row0 + lane] : 0.f;
        const double log_own = there ? -(double)rate[head] * step : 0.0;      // (an infinite one, as of an infinite rate, is one of a decay of zero)
        const double c = chunk::lanes_cumulative(log_own < chunk::kLogOfNothing ? chunk::kLogOfNothing : log_own, lane);
        const double c_last = __shfl_sync(0xffffffffu, c, 31);            // (tokens beyond the step's add nothing)
        const float d = skip[head];
        if (there)
            scalars[(size_t)head * n_rows + row0 + lane] = make_float4(expf((float)c), 0.f, step * expf((float)(c_last - c)), 0.f);
        // a half warp takes a row, a lane two neighbouring tokens j of it
        const int j = 2 * (lane & 15);
        const double c0 = __shfl_sync(0xffffffffu, c, j), c1 = __shfl_sync(0xffffffffu, c, j + 1);
        const float t0 = __shfl_sync(0xffffffffu, step, j), t1 = __shfl_sync(0xffffffffu, step, j + 1);
        __nv_bfloat16* dst = scores + head * 3 * score_plane + (long long)row0 * chunk::kScoreRow + j;
#pragma unroll 4
        for (int i0 = 0; i0 < n_here; i0 += 2) {
            const int i = i0 + (lane >> 4);
            const double ci = __shfl_sync(0xffffffffu, c, i);
            if (i >= n_here) continue;
            float x = j <= i ? expf((float)(ci - c0)) * t0 * dot_s[i * (C + 1) + j] : 0.f;
            float y = j + 1 <= i ? expf((float)(ci - c1)) * t1 * dot_s[i * (C + 1) + j + 1] : 0.f;
            if (j == i) x += d;
            if (j + 1 == i) y += d;
            chunk::store_split(dst + (long long)i * chunk::kScoreRow, score_plane, x, y);
        }
    }
}
constexpr size_t kSpaceChunkBytes = (size_t)6 * chunk::kTokens * chunk::kKeyRow * 2 + chunk::kTokens * (chunk::kTokens + 1) * sizeof(float);

constexpr int kDecodeThreads = 256;
constexpr int kDecodeLanes = 8;            // lanes that share a column of S

// Shared memory: B, C [n_state] each, x [vdim].
template <typename T>
__global__ void __launch_bounds__(kDecodeThreads) state_space_decode_kernel(
    float* __restrict__ y, float* __restrict__ state, const T* __restrict__ proj, int proj_width, int offset,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b, T* __restrict__ ring, const float* __restrict__ dt_pre,
    const float* __restrict__ dt_bias, const float* __restrict__ rate, const float* __restrict__ skip,
    const int* __restrict__ row_slot, const int* __restrict__ row_pos, SpaceShape shape) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float mem[];
    const int N = shape.n_state, V = shape.vdim, taps = shape.taps, channels = shape.channels();
    const int padded = (N + 3) / 4 * 4;
    float *bs = mem, *cs = mem + padded, *xs = mem + 2 * padded;
    const int head = blockIdx.x, row = blockIdx.y;
    const int per_group = shape.n_heads / shape.n_groups, group = head / per_group;
    const int slot = row_slot[row], pos = row_pos[row];
    const T* src = proj + (size_t)row * proj_width + offset;
    T* slot_ring = ring + (size_t)slot * taps * channels;
    for (int i = threadIdx.x; i < V + 2 * N; i += kDecodeThreads) {
        const int c = i < V ? head * V + i
                            : shape.inner() + (i < V + N ? group * N + (i - V) : (shape.n_groups + group) * N + (i - V - N));
        const T raw = src[c];
        float acc = conv_b[c];
        for (int j = 0; j < taps - 1; ++j) {
            const int back = taps - 1 - j;
            if (back <= pos) acc += conv_w[(size_t)c * taps + j] * to_f32<T>(slot_ring[(size_t)((pos - back) % taps) * channels + c]);
        }
        acc += conv_w[(size_t)c * taps + taps - 1] * to_f32<T>(raw);
        // The entry that this token takes held the input of `taps` tokens ago, which no tap reads: blocks
        // that share B and C do not disturb one another.  The group's first head stores them.
        if (i < V || head == group * per_group) slot_ring[(size_t)(pos % taps) * channels + c] = raw;
        const float v = silu_of<T>(acc);
        if (i < V) xs[i] = v;
        else if (i < V + N) bs[i - V] = v;
        else cs[i - V - N] = v;
    }
    const float t = softplus_of<T>(dt_pre[(size_t)row * shape.n_heads + head] + dt_bias[head]);
    const float decay = exp_of<T>(-rate[head] * t), d_skip = skip[head];
    __syncthreads();
    float* S = state + ((size_t)slot * shape.n_heads + head) * V * N;
    const int lane = threadIdx.x % kDecodeLanes, column = threadIdx.x / kDecodeLanes;
    constexpr int kGroups = kDecodeThreads / kDecodeLanes;
    const bool vec = N % 4 == 0;
    for (int e0 = 0; e0 < V; e0 += kGroups) {
        const int e = e0 + column;
        float part = 0.f;
        if (e < V) {
            float* col = S + (size_t)e * N;
            const float tx = t * xs[e];
            if (vec) {
                for (int d = lane * 4; d < N; d += kDecodeLanes * 4) {
                    float4 s = *reinterpret_cast<const float4*>(col + d);
                    const float4 b = *reinterpret_cast<const float4*>(bs + d), c = *reinterpret_cast<const float4*>(cs + d);
                    s.x = decay * s.x + b.x * tx;
                    s.y = decay * s.y + b.y * tx;
                    s.z = decay * s.z + b.z * tx;
                    s.w = decay * s.w + b.w * tx;
                    part += s.x * c.x + s.y * c.y + s.z * c.z + s.w * c.w;
                    *reinterpret_cast<float4*>(col + d) = s;
                }
            } else {
                for (int d = lane; d < N; d += kDecodeLanes) {
                    const float s = decay * col[d] + bs[d] * tx;
                    part += s * cs[d];
                    col[d] = s;
                }
            }
        }
#pragma unroll
        for (int off = kDecodeLanes / 2; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
        if (lane == 0 && e < V) y[((size_t)row * shape.n_heads + head) * V + e] = part + d_skip * xs[e];
    }
}

// One block per (row, part), with as many threads as the part has pieces of four entries, up to 256.  The gated entries are computed twice, once for the sum of squares and
// once for the result; the second reading comes from the caches.
template <typename T>
__global__ void __launch_bounds__(256) gated_group_norm_kernel(T* __restrict__ out, const float* __restrict__ y,
                                                               const T* __restrict__ gate, long long gate_stride,
                                                               const float* __restrict__ gain, float eps, int width, int size,
                                                               int vec) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float scratch[33];
    const size_t base = (size_t)blockIdx.x * width + (size_t)blockIdx.y * size;
    const float* src = y + base;
    const T* g = gate + (size_t)blockIdx.x * gate_stride + (size_t)blockIdx.y * size;
    const float* w = gain + (size_t)blockIdx.y * size;
    T* dst = out + base;
    float ss = 0.f;
    if (vec) {
        constexpr int kKept = 4;                    // what fits stays in registers (parts up to sixteen entries a thread)
        float4 kept[kKept];
#pragma unroll
        for (int j = 0; j < kKept; ++j) {
            const int i = (j * (int)blockDim.x + (int)threadIdx.x) * 4;
            if (i < size) {
                const float4 v = *reinterpret_cast<const float4*>(src + i), z = load_four<T>(g + i);
                kept[j] = make_float4(v.x * silu_of<T>(z.x), v.y * silu_of<T>(z.y), v.z * silu_of<T>(z.z), v.w * silu_of<T>(z.w));
                ss += kept[j].x * kept[j].x + kept[j].y * kept[j].y + kept[j].z * kept[j].z + kept[j].w * kept[j].w;
            }
        }
        for (int i = (kKept * (int)blockDim.x + (int)threadIdx.x) * 4; i < size; i += (int)blockDim.x * 4) {
            const float4 v = *reinterpret_cast<const float4*>(src + i), z = load_four<T>(g + i);
            const float a = v.x * silu_of<T>(z.x), b = v.y * silu_of<T>(z.y), c = v.z * silu_of<T>(z.z), d = v.w * silu_of<T>(z.w);
            ss += a * a + b * b + c * c + d * d;
        }
        const float rstd = 1.0f / sqrtf(block_sum(ss, scratch) / (float)size + eps);
        auto store = [&](int i, const float4& v) {
            const float4 gw = *reinterpret_cast<const float4*>(w + i);
            if constexpr (sizeof(T) == 2) {
                uint2 packed;
                *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(v.x * rstd * gw.x, v.y * rstd * gw.y);
                *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(v.z * rstd * gw.z, v.w * rstd * gw.w);
                *reinterpret_cast<uint2*>(dst + i) = packed;
            } else {
                *reinterpret_cast<float4*>(dst + i) = make_float4(v.x * rstd * gw.x, v.y * rstd * gw.y, v.z * rstd * gw.z, v.w * rstd * gw.w);
            }
        };
#pragma unroll
        for (int j = 0; j < kKept; ++j) {
            const int i = (j * (int)blockDim.x + (int)threadIdx.x) * 4;
            if (i < size) store(i, kept[j]);
        }
        for (int i = (kKept * (int)blockDim.x + (int)threadIdx.x) * 4; i < size; i += (int)blockDim.x * 4) {
            const float4 v = *reinterpret_cast<const float4*>(src + i), z = load_four<T>(g + i);
            store(i, make_float4(v.x * silu_of<T>(z.x), v.y * silu_of<T>(z.y), v.z * silu_of<T>(z.z), v.w * silu_of<T>(z.w)));
        }
        return;
    }
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        const float v = src[i] * silu_of<T>(to_f32<T>(g[i]));
        ss += v * v;
    }
    const float rstd = 1.0f / sqrtf(block_sum(ss, scratch) / (float)size + eps);
    for (int i = threadIdx.x; i < size; i += blockDim.x) dst[i] = from_f32<T>(src[i] * silu_of<T>(to_f32<T>(g[i])) * rstd * w[i]);
}

// The same for bfloat16 and parts of whole groups of 128 entries, up to 1,024: a warp per (row, part), the gated entries in
// registers between the sum and the result, no barrier.  (4,096 rows of eight parts of 1,024 on B200: 61 us, 95 above.)
__global__ void __launch_bounds__(256) gated_group_norm_warp_kernel(__nv_bfloat16* __restrict__ out, const float* __restrict__ y,
                                                                    const __nv_bfloat16* __restrict__ gate, long long gate_stride,
                                                                    const float* __restrict__ gain, float eps, int rows, int width,
                                                                    int size, int parts) {
    pdl_launch_dependents();
    pdl_wait();
    using T = __nv_bfloat16;
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= (long long)rows * parts) return;
    const long long row = unit / parts;
    const int part = (int)(unit - row * parts), lane = threadIdx.x & 31;
    const float* src = y + row * width + (long long)part * size + lane * 4;
    const T* g = gate + row * gate_stride + (long long)part * size + lane * 4;
    const float* w = gain + (long long)part * size + lane * 4;
    constexpr int kGroups = 8;
    float4 kept[kGroups];
    uint2 z[kGroups];
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
        if (j * 128 < size) {
            kept[j] = *reinterpret_cast<const float4*>(src + j * 128);
            z[j] = *reinterpret_cast<const uint2*>(g + j * 128);
        }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
        if (j * 128 < size) {
            const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&z[j].x));
            const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&z[j].y));
            kept[j].x *= silu_of<T>(lo.x); kept[j].y *= silu_of<T>(lo.y); kept[j].z *= silu_of<T>(hi.x); kept[j].w *= silu_of<T>(hi.y);
            ss += kept[j].x * kept[j].x + kept[j].y * kept[j].y + kept[j].z * kept[j].z + kept[j].w * kept[j].w;
        }
    const float rstd = 1.0f / sqrtf(warp_sum(ss) / (float)size + eps);
    T* dst = out + row * width + (long long)part * size + lane * 4;
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
        if (j * 128 < size) {
            const float4 gw = *reinterpret_cast<const float4*>(w + j * 128);
            uint2 packed;
            *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(kept[j].x * rstd * gw.x, kept[j].y * rstd * gw.y);
            *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(kept[j].z * rstd * gw.z, kept[j].w * rstd * gw.w);
            *reinterpret_cast<uint2*>(dst + j * 128) = packed;
        }
}

int check_shape(const char* what, const SpaceShape& s, int proj_width, int offset) {
    THN_CHECK_ARG(s.n_heads > 0 && s.vdim > 0 && s.n_state > 0 && s.n_groups > 0 && s.n_heads % s.n_groups == 0 && s.taps > 0,
                  "%s: %d heads of %d in %d groups, state %d, %d taps", what, s.n_heads, s.vdim, s.n_groups, s.n_state, s.taps);
    THN_CHECK_ARG(offset >= 0 && offset + s.channels() <= proj_width, "%s: %d channels from column %d of rows of %d", what,
                  s.channels(), offset, proj_width);
    THN_UNSUPPORTED_IF(s.n_state > 512, "%s: a state of %d, at most 512", what, s.n_state);
    return THN_OK;
}

template <typename T>
void launch_prepare(float* keys, float* values, const void* proj, int proj_width, int offset, const float* conv_w,
                    const float* conv_b, const void* ring, const float* dt_pre, const float* dt_bias, const float* rate,
                    const int* row_slot, const int* row_pos, const int* seq_lens, int n_rows, const SpaceShape& s, cudaStream_t stream) {
    const int kp = padded_keys(s.n_state), vp = padded_values(s.vdim);
    const int items = s.n_heads * (vp / 4) + s.n_groups * 2 * (kp / 4) + s.n_heads;
    const dim3 grid((items + kPrepareThreads - 1) / kPrepareThreads, (n_rows + kRunRows - 1) / kRunRows);
    const uintptr_t piece = 4 * sizeof(T) - 1;
    const int vec = s.vdim % 4 == 0 && s.n_state % 4 == 0 && proj_width % 4 == 0 && offset % 4 == 0 &&
                    (((uintptr_t)proj | (uintptr_t)ring) & piece) == 0;
#define THN_SPACE_PREPARE(K)                                                                                            \
    thn_launch(state_space_prepare_kernel<T, K>, grid, kPrepareThreads, 0, stream, keys, values, (const T*)proj, proj_width, \
               offset, conv_w, conv_b, (const T*)ring, dt_pre, dt_bias, rate, row_slot, row_pos, seq_lens, n_rows, s, kp, vp, vec)
    if (s.taps == 4) THN_SPACE_PREPARE(4);
    else if (s.taps == 3) THN_SPACE_PREPARE(3);
    else if (s.taps == 2) THN_SPACE_PREPARE(2);
    else THN_SPACE_PREPARE(0);
#undef THN_SPACE_PREPARE
}

}  // namespace

// Floats of the scratch that thn_state_space needs for a step of n_rows rows.
THN_API long long thn_state_space_scratch_floats(int n_rows, int n_heads, int vdim, int n_state, int n_groups) {
    return (long long)n_rows * ((long long)n_groups * 2 * padded_keys(n_state) + (long long)n_heads * (padded_values(vdim) + kRecurrenceTail));
}

// Bytes of the scratch that thn_state_space_chunks needs for a step of n_rows rows.
THN_API long long thn_state_space_chunks_scratch_bytes(int n_rows, int n_heads, int vdim, int n_groups) {
    return (long long)n_rows * (6ll * n_groups * chunk::kKeyRow * 2 + (long long)n_heads * (3 * chunk::kScoreRow * 2 + 16 + vdim * 4 + 4));
}

// Whether a step's blocks are so many and short that their starts weigh more than their chunks: they then copy themselves, two to a multiprocessor.  us of
// the whole call, such blocks / the same columns brought, 64 heads of 64: 32 x 128 tokens 314 / 332, 128 beside 60 single ones 164 / 207, 512 beside 60 187 / 229,
// 12 x 300 312 / 310, 2,048 beside 60 409 / 322.
inline bool many_short(int n_rows, int n_seqs, int max_tokens) { return n_rows < 200ll * n_seqs && max_tokens < 1024; }

// Which blocks walk the chunks (WalkCost): 1 has 16 columns and four warps, which split the keys; 2: 32, four for a group of 16; 3: 64, two; 4: as 3, two
// blocks on a multiprocessor with one buffer each, into which the warps copy themselves, where blocks are many and short.  us of the whole call, 1 / 2 / 3 / 4, 64 heads
// of 64: one prompt of 2,048 tokens 236 / 184 / 286 / 356, beside 60 single ones 504 / 368 / 322 / 409, 512 tokens beside 8 112 / 90 / 94 / 112, 8 x 512
// 415 / 326 / 327 / 330; 128 heads, one prompt of 2,048 tokens 449 / 347 / 319 / 393, 512 beside 60 700 / 496 / 420 / 339.  Over 588 steps of 16 to 128 heads the
// chosen one takes 0.9 % longer than the best of four.
constexpr chunk::WalkCost kWalkCosts[3] = {{6.63f, 1.28f, 6.59f, 0.00f, 0.17f, 16, 1}, {5.32f, 1.75f, 5.74f, 0.00f, 0.06f, 32, 1}, {5.30f, 2.86f, 4.42f, 0.31f, 0.07f, 64, 1}};

THN_API int thn_state_space_walk_shape(int n_rows, int max_tokens, int n_seqs, int n_heads, int vdim) {
    if (vdim % 64 == 0 && (long long)n_seqs * n_heads * (vdim / 64) >= 384 && many_short(n_rows, n_seqs, max_tokens)) return 4;
    return chunk::cheapest_walk(kWalkCosts, n_rows, max_tokens, n_seqs, n_heads, vdim);
}

// thn_state_space chunk by chunk: bfloat16 rows in whole 8-byte pieces, four taps, a state of 128, vdim a multiple of 16;
// max_tokens: the most rows of a sequence.  On B200, us against token by token: 8 x 512 tokens of 128 heads of 64 over a
// state of 128 582 / 1,067, one prompt of 2,048 tokens of 64 heads 184 / 348, 128 tokens 34 / 32.  The error against 64 bits:
// y 1.2e-7 (1.2e-7 to 1.3e-7), the state 1.1e-7 (1.2e-7).
THN_API int thn_state_space_chunks(float* y, float* state, void* scratch, long long scratch_bytes, const void* proj, int proj_width,
                                   int offset, const float* conv_w, const float* conv_b, const void* ring, const float* dt_pre,
                                   const float* dt_bias, const float* rate, const float* skip, const int* row_slot, const int* row_pos,
                                   const int* seq_lens, const int* cu_seqlens, const int* slots, int n_rows, int max_tokens, int n_seqs,
                                   int n_heads, int vdim, int n_state, int n_groups, int taps, int* err, cudaStream_t stream) {
    const SpaceShape s{n_heads, vdim, n_state, n_groups, taps};
    if (int status = check_shape("state_space_chunks", s, proj_width, offset)) return status;
    THN_UNSUPPORTED_IF(n_state != chunk::kKeys || vdim % 16 != 0 || taps != kChunkTaps || proj_width % 4 != 0 || offset % 4 != 0,
                       "state_space_chunks: a state of %d, values of %d, %d taps, rows of %d from %d", n_state, vdim, taps, proj_width, offset);
    THN_UNSUPPORTED_IF(n_heads > 65535 || n_seqs > 65535 || (n_rows + kRunRows - 1) / kRunRows > 65535,
                       "state_space_chunks: %d heads, %d sequences, %d rows", n_heads, n_seqs, n_rows);
    THN_CHECK_ARG(scratch && (((uintptr_t)state | (uintptr_t)scratch | (uintptr_t)conv_w) & 15) == 0 &&
                      (((uintptr_t)proj | (uintptr_t)ring) & 7) == 0,
                  "state_space_chunks: operands are not aligned");
    if (n_seqs <= 0 || n_rows <= 0 || max_tokens <= 0) return THN_OK;
    const long long need = thn_state_space_chunks_scratch_bytes(n_rows, n_heads, vdim, n_groups);
    THN_CHECK_ARG(scratch_bytes >= need, "state_space_chunks: %lld bytes of scratch, %lld needed", scratch_bytes, need);
    const long long plane = (long long)n_rows * chunk::kKeyRow;
    __nv_bfloat16* planes = static_cast<__nv_bfloat16*>(scratch);
    __nv_bfloat16* scores = planes + 6 * n_groups * plane;
    float4* scalars = reinterpret_cast<float4*>(scores + (size_t)3 * n_heads * n_rows * chunk::kScoreRow);
    float* values = reinterpret_cast<float*>(scalars + (size_t)n_heads * n_rows);
    float* steps = values + (size_t)n_heads * n_rows * vdim;
    const int items = s.channels() / 4 + n_heads;
    thn_launch(state_space_prepare_chunks_kernel, dim3((items + kPrepareThreads - 1) / kPrepareThreads, (n_rows + kRunRows - 1) / kRunRows),
               kPrepareThreads, 0, stream, planes, values, steps, (const __nv_bfloat16*)proj, proj_width, offset, conv_w, conv_b,
               (const __nv_bfloat16*)ring, dt_pre, dt_bias, row_slot, row_pos, seq_lens, n_rows, s);
    cudaFuncSetAttribute(state_space_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpaceChunkBytes);
    thn_launch(state_space_chunk_kernel, dim3((max_tokens + chunk::kTokens - 1) / chunk::kTokens, n_groups, n_seqs), kSpaceThreads, kSpaceChunkBytes,
               stream, scores, scalars, planes, steps, rate, skip, cu_seqlens, n_rows, n_heads / n_groups);
    chunk::WalkArgs a{};
    a.err = err;
    a.o = y; a.state = state;
    a.k = planes; a.q = planes + 3 * plane;
    a.key_plane = plane; a.key_unit = 6 * plane; a.key_row = chunk::kKeyRow;
    a.v = values; a.v_row = vdim; a.v_head = (long long)n_rows * vdim;
    a.scores = scores; a.scalars = scalars;
    a.cu_seqlens = cu_seqlens; a.slots = slots;
    a.n_rows = n_rows; a.n_heads = n_heads; a.heads_per_unit = n_heads / n_groups; a.value_dim = vdim; a.scale = 1.f;
    using namespace chunk;
    switch (thn_state_space_walk_shape(n_rows, max_tokens, n_seqs, n_heads, vdim)) {
        case 4: launch_walk<float, 4, 2, kPlain, 1, false>(a, n_seqs, stream); break;
        case 3: launch_brought_walk<float, 4, 2, kPlain>(a, n_seqs, stream); break;
        case 2: launch_brought_walk<float, 2, 4, kPlain>(a, n_seqs, stream); break;
        default: launch_brought_walk<float, 1, 4, kPlain>(a, n_seqs, stream);
    }
    return thn_launch_status("state_space_chunks");
}

// y float32 [rows, heads, vdim]; state float32 [slots, heads, vdim, n_state], read and updated; the raw
// inputs [x: heads * vdim | B: groups * n_state | C: groups * n_state] are the columns from `offset` of
// proj [rows, proj_width]; conv_w float32 [channels, taps] (the last tap is the current token's), conv_b
// float32 [channels]; ring [slots, taps, channels] of the activation type (read only: the step's inputs
// go in by thn_conv_ring_update afterwards); dt_pre float32 [rows, heads]; dt_bias, rate (the decay is
// exp(-rate * step)), skip float32 [heads]; seq_lens: the tokens each slot held before the step.
THN_API int thn_state_space(float* y, float* state, float* scratch, const void* proj, int proj_width, int offset,
                            const float* conv_w, const float* conv_b, const void* ring, const float* dt_pre,
                            const float* dt_bias, const float* rate, const float* skip, const int* row_slot,
                            const int* row_pos, const int* seq_lens, const int* cu_seqlens, const int* slots, int n_rows,
                            int n_seqs, int n_heads, int vdim, int n_state, int n_groups, int taps, int dtype,
                            cudaStream_t stream) {
    const SpaceShape s{n_heads, vdim, n_state, n_groups, taps};
    const int bad = check_shape("state_space", s, proj_width, offset);
    if (bad) return bad;
    THN_CHECK_ARG(scratch != nullptr && ((uintptr_t)scratch & 15) == 0 && n_rows >= 0 && n_seqs >= 0, "state_space: scratch missing or unaligned");
    THN_UNSUPPORTED_IF(n_rows > 65535 * kRunRows, "state_space: %d rows", n_rows);
    if (n_rows == 0 || n_seqs == 0) return THN_OK;
    const int kp = padded_keys(n_state), vp = padded_values(vdim);
    float* keys = scratch;
    float* values = scratch + (size_t)n_rows * n_groups * 2 * kp;
    if (dtype == THN_F32)
        launch_prepare<float>(keys, values, proj, proj_width, offset, conv_w, conv_b, ring, dt_pre, dt_bias, rate, row_slot,
                              row_pos, seq_lens, n_rows, s, stream);
    else if (dtype == THN_BF16)
        launch_prepare<__nv_bfloat16>(keys, values, proj, proj_width, offset, conv_w, conv_b, ring, dt_pre, dt_bias, rate,
                                      row_slot, row_pos, seq_lens, n_rows, s, stream);
    else
        THN_CHECK_ARG(false, "state_space: unknown dtype %d", dtype);
    return launch_recurrence(kSteppedDecay, RecurrenceArgs{y, state, keys, 2 * kp, n_groups, values, vp + kRecurrenceTail, skip,
                                                           cu_seqlens, slots, n_seqs, n_heads, n_state, vdim, 1.0f}, stream);
}

// One token per sequence: the same, and the token's raw inputs go into the ring.
THN_API int thn_state_space_decode(float* y, float* state, const void* proj, int proj_width, int offset, const float* conv_w,
                                   const float* conv_b, void* ring, const float* dt_pre, const float* dt_bias,
                                   const float* rate, const float* skip, const int* row_slot, const int* row_pos, int n_rows,
                                   int n_heads, int vdim, int n_state, int n_groups, int taps, int dtype, cudaStream_t stream) {
    const SpaceShape s{n_heads, vdim, n_state, n_groups, taps};
    const int bad = check_shape("state_space_decode", s, proj_width, offset);
    if (bad) return bad;
    const size_t smem = (size_t)(2 * ((n_state + 3) / 4 * 4) + vdim) * sizeof(float);
    THN_UNSUPPORTED_IF(n_rows > 65535 || smem > 48 * 1024, "state_space_decode: %d rows, values of %d", n_rows, vdim);
    if (n_rows <= 0) return THN_OK;
    const dim3 grid(n_heads, n_rows);
    if (dtype == THN_F32)
        thn_launch(state_space_decode_kernel<float>, grid, kDecodeThreads, smem, stream, y, state, (const float*)proj, proj_width,
                   offset, conv_w, conv_b, (float*)ring, dt_pre, dt_bias, rate, skip, row_slot, row_pos, s);
    else if (dtype == THN_BF16)
        thn_launch(state_space_decode_kernel<__nv_bfloat16>, grid, kDecodeThreads, smem, stream, y, state,
                   (const __nv_bfloat16*)proj, proj_width, offset, conv_w, conv_b, (__nv_bfloat16*)ring, dt_pre, dt_bias, rate,
                   skip, row_slot, row_pos, s);
    else
        THN_CHECK_ARG(false, "state_space_decode: unknown dtype %d", dtype);
    return thn_launch_status("state_space_decode");
}

// y float32 [rows, width]; gate of the activation type, rows gate_stride elements apart; gain float32
// [width]; out [rows, width] of the activation type; `parts` equal consecutive parts of a row.
THN_API int thn_gated_group_norm(void* out, const float* y, const void* gate, long long gate_stride, const float* gain,
                                 float eps, int rows, int width, int parts, int dtype, cudaStream_t stream) {
    THN_CHECK_ARG(rows >= 0 && width > 0 && parts > 0 && width % parts == 0 && parts <= 65535 && gate_stride >= width && eps > 0.f,
                  "gated_group_norm: rows of %d in %d parts", width, parts);
    if (rows == 0) return THN_OK;
    const int size = width / parts;
    const size_t element = dtype == THN_BF16 ? 2 : 4;
    const int vec = size % 4 == 0 && gate_stride % 4 == 0 && (((uintptr_t)y | (uintptr_t)gain) & 15) == 0 &&
                    (((uintptr_t)gate | (uintptr_t)out) & (4 * element - 1)) == 0;
    // Few parts are faster with a block each, the more so the longer they are.  In us, a block / a warp each, back to back: parts of
    // 1,024: 1,184 of them 4.3 / 4.6, 2,048 6.3 / 6.7, 3,072 8.9 / 6.7; of 512: 1,184 2.9 / 3.0, 2,048 4.1 / 3.9; of 256: 1,184 2.9 / 2.4.
    const long long units = (long long)rows * parts;
    const long long enough = 3ll * size < 1184 ? 1184 : 3ll * size;
    if (dtype == THN_BF16 && vec && size % 128 == 0 && size <= 1024 && units >= enough) {
        thn_launch(gated_group_norm_warp_kernel, (unsigned)((units + 7) / 8), 256, 0, stream, (__nv_bfloat16*)out, y,
                   (const __nv_bfloat16*)gate, gate_stride, gain, eps, rows, width, size, parts);
        return thn_launch_status("gated_group_norm");
    }
    const dim3 grid(rows, parts);
    const int threads = size >= 1024 ? 256 : (size / 4 + 31) / 32 * 32 < 32 ? 32 : (size / 4 + 31) / 32 * 32;
    if (dtype == THN_F32)
        thn_launch(gated_group_norm_kernel<float>, grid, threads, 0, stream, (float*)out, y, (const float*)gate, gate_stride, gain, eps,
                   width, size, vec);
    else if (dtype == THN_BF16)
        thn_launch(gated_group_norm_kernel<__nv_bfloat16>, grid, threads, 0, stream, (__nv_bfloat16*)out, y, (const __nv_bfloat16*)gate,
                   gate_stride, gain, eps, width, size, vec);
    else
        THN_CHECK_ARG(false, "gated_group_norm: unknown dtype %d", dtype);
    return thn_launch_status("gated_group_norm");
}
