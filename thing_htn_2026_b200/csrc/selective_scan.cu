// The selective scan (Mamba): per channel c a state vector S[c, 0..N-1], zero at a sequence's
// start, and for every token
//
//     dt_c = softplus(dt_pre[c] + dt_bias[c])
//     S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n
//     y_c = (sum_n S[c, n] C_n + D_c x_c) * silu(z_c)
//
// with A < 0 a constant matrix, x the convolved input, B and C vectors of the token shared by
// all channels, z the token's gate.  Ahead of it a short causal convolution per channel with
// silu:  x_c[t] = silu(bias_c + sum_j w[c, j] raw_c[t - (taps - 1) + j]),  zeros before the
// sequence's start.
//
//   causal_conv   one thread per (row, channel).  A token's predecessors come from the step's own
//                 rows or, before the step's first row, from the ring: the last `taps` raw inputs
//                 of the sequence, position p at p mod taps.
//   conv_ring_update   after every reader of the ring has ended: the step's last raw inputs go in.
//   selective_scan     a channel's state is held by 4 lanes (8 for states above 32; entry n by lane
//                 n mod lanes); one block per (sequence, 64 or 32 channels) walks the sequence's tokens of the step in order;
//                 the tokens come through shared memory, sixteen at a time in two buffers.
//   selective_scan_walk     the same for bfloat16 prompts with states up to 32 (walk_pays): some of a block's warps walk the
//                 state, the others load, transform and write beside them.
//
// float32 after the loads: the step size with its softplus, the decay with its exponential, the
// state, the sums, the gate.  The convolution is summed in float32 and rounded once after silu.
// With float32 activations the exponentials and logarithms are computed in double and rounded once
// (exp_of, silu_of, softplus_of in common.cuh).
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "conv_run.cuh"

namespace {



template <typename T>
__global__ void causal_conv_kernel(T* __restrict__ out, const T* __restrict__ proj, int proj_width, int offset,
                                   const float* __restrict__ weight, const float* __restrict__ bias,
                                   const T* __restrict__ ring, const int* __restrict__ row_slot,
                                   const int* __restrict__ row_pos, const int* __restrict__ seq_lens, long long n,
                                   int channels, int taps) {
    pdl_launch_dependents();
    pdl_wait();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const long long row = e / channels;
    const int c = (int)(e - row * channels);
    const int slot = row_slot[row], pos = row_pos[row];
    const int local = pos - seq_lens[slot];          // index of the row among its sequence's rows of this step
    float acc = bias ? bias[c] : 0.f;
    for (int j = 0; j < taps; ++j) {
        const int back = taps - 1 - j;               // how many tokens before this one
        if (back > pos) continue;                    // before the sequence's start: zero
        float v;
        if (back <= local) v = to_f32<T>(proj[(size_t)(row - back) * proj_width + offset + c]);
        else v = to_f32<T>(ring[((size_t)slot * taps + (pos - back) % taps) * channels + c]);
        acc += weight[(size_t)c * taps + j] * v;
    }
    out[e] = from_f32<T>(silu_of<T>(acc));
}

// The same for bfloat16 rows of 8-byte pieces and four taps: a thread takes four neighbouring channels of
// kConvRows rows, with the raw inputs ahead of a row in registers, so that an input is loaded once for
// its four uses.  2,048 rows of 4,096 channels on B200: 22 us against 78 with a thread per entry (2-byte
// accesses, two divisions an entry); the inputs once and the outputs once take 5.  (Eight channels a
// thread need 114 registers and leave too few warps to cover the loads: 29 us.)
constexpr int kConvTaps = 4;
constexpr int kConvRows = 8;

template <bool FEW>
__global__ void __launch_bounds__(128) causal_conv_vec_kernel(
    __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ proj, int proj_width, int offset,
    const float* __restrict__ weight, const float* __restrict__ bias, const __nv_bfloat16* __restrict__ ring,
    const int* __restrict__ row_slot, const int* __restrict__ row_pos, const int* __restrict__ seq_lens, int n_rows,
    int channels) {
    pdl_launch_dependents();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const int first = blockIdx.y * kConvRows, n_here = min(kConvRows, n_rows - first);
    if (c >= channels) return;
    float w[4][kConvTaps], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(weight + (size_t)(c + i) * kConvTaps);
        w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
        b[i] = bias ? bias[c + i] : 0.f;
    }
    pdl_wait();
    __nv_bfloat16* dst = out + (size_t)first * channels + c;
    const conv_run::Source source{proj + (size_t)first * proj_width + offset + c, proj_width, ring + c, channels, row_slot, row_pos, seq_lens};
    conv_run::run<kConvRows, FEW>(source, first, n_here, w, b, [&](int t, const float (&y)[4]) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
        *reinterpret_cast<uint2*>(dst + (size_t)t * channels) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    });
}

template <typename T>
__global__ void conv_ring_update_kernel(T* __restrict__ ring, const T* __restrict__ proj, int proj_width, int offset,
                                        const int* __restrict__ cu_seqlens, const int* __restrict__ slots,
                                        const int* __restrict__ seq_lens, int channels, int taps) {
    pdl_launch_dependents();
    pdl_wait();
    const int seq = blockIdx.y;
    const int row0 = cu_seqlens[seq], row1 = cu_seqlens[seq + 1], slot = slots[seq];
    const int held = seq_lens[slot];
    const int first = max(row0, row1 - taps);
    const int total = (row1 - first) * channels;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int r = first + e / channels, c = e % channels;
        const int pos = held + (r - row0);
        ring[((size_t)slot * taps + pos % taps) * channels + c] = proj[(size_t)r * proj_width + offset + c];
    }
}

// The decay exp(dt * A).  With bfloat16 activations A is held times log2(e) and the exponential is
// the hardware's base-2 one (two ulp; four full ones a token are a third of the scan's instructions
// otherwise); on the 32-bit path it is computed in double and rounded once.
template <typename T> struct Decay {
    static __device__ __forceinline__ float hold(float a) { return a * 1.4426950408889634f; }
    static __device__ __forceinline__ float of(float dt, float held) { return exp2f(dt * held); }
};
template <> struct Decay<float> {
    static __device__ __forceinline__ float hold(float a) { return a; }
    static __device__ __forceinline__ float of(float dt, float held) { return exp_of<float>(dt * held); }
};

// LANES lanes hold a channel's state, PER entries each; NP = LANES * PER: the padded state size of a
// staged token's B and C.  A block of 256 threads takes 256 / LANES channels: 64 with four lanes
// (states up to 32), so that a token's step sizes, inputs and gates are runs of 128 to 256 bytes.
// A staged token is [B | C | dt of the block's channels | x | silu(z)]; FETCH values per thread
// and stage.  Every thread fetches its part of the next stage into registers, the block works
// through the current one, then the fetched values are transformed once per block (the step size
// with its bias and softplus, the gate with its silu) and stored for all lanes to read.
constexpr int kStage = 16;
constexpr int kScanThreads = 256;

// A value as it was loaded, untouched: turning it into a float is a use, and a use makes the thread
// wait for the load.  The stage's loads are all issued first and turned into floats when they are stored.
template <typename T> __device__ __forceinline__ uint32_t raw_load(const T* p);
template <> __device__ __forceinline__ uint32_t raw_load<float>(const float* p) { return *reinterpret_cast<const uint32_t*>(p); }
template <> __device__ __forceinline__ uint32_t raw_load<__nv_bfloat16>(const __nv_bfloat16* p) {
    return *reinterpret_cast<const unsigned short*>(p);
}
template <typename T> __device__ __forceinline__ float from_raw(uint32_t bits);
template <> __device__ __forceinline__ float from_raw<float>(uint32_t bits) { return __uint_as_float(bits); }
template <> __device__ __forceinline__ float from_raw<__nv_bfloat16>(uint32_t bits) { return __uint_as_float(bits << 16); }

template <typename T, int LANES, int PER, int FETCH>
__global__ void __launch_bounds__(kScanThreads) selective_scan_kernel(
    T* __restrict__ y, float* __restrict__ state, const T* __restrict__ x, const float* __restrict__ dt_pre,
    const float* __restrict__ dt_bias, const T* __restrict__ bc, int bc_width, const float* __restrict__ A,
    const float* __restrict__ D, const T* __restrict__ z, int z_stride, const int* __restrict__ cu_seqlens,
    const int* __restrict__ slots, int channels, int n_state) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kLanes = LANES, kChannels = kScanThreads / LANES, kThreads = kScanThreads;
    constexpr int NP = kLanes * PER, ROW = 2 * NP + 3 * kChannels;
    __shared__ float stage_mem[2 * kStage * ROW];
    __shared__ float bias_mem[kChannels];
    const int seq = blockIdx.y;
    const int c0 = blockIdx.x * kChannels;
    const int group = threadIdx.x / kLanes, lane = threadIdx.x % kLanes;
    const int channel = c0 + group;
    const bool live = channel < channels;
    const int c = live ? channel : channels - 1;
    const int row0 = cu_seqlens[seq], row1 = cu_seqlens[seq + 1];
    const int slot = slots[seq];
    float* S = state + ((size_t)slot * channels + c) * n_state;

    float s[PER], a[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int n = lane + kLanes * i;
        s[i] = n < n_state ? S[n] : 0.f;
        a[i] = n < n_state ? Decay<T>::hold(A[(size_t)c * n_state + n]) : 0.f;
    }
    const float skip = D[c];
    if (threadIdx.x < kChannels) bias_mem[threadIdx.x] = dt_bias[min(c0 + (int)threadIdx.x, channels - 1)];

    uint32_t fetched[FETCH];
    auto fetch = [&](int first_row) {
#pragma unroll
        for (int j = 0; j < FETCH; ++j) {
            const int e = threadIdx.x + j * kThreads;
            const int t = e / ROW, k = e - t * ROW;
            const int row = first_row + t;
            uint32_t v = 0;
            if (row < row1) {
                if (k < 2 * NP) {
                    const int which = k / NP, n = k - which * NP;
                    if (n < n_state) v = raw_load<T>(bc + (size_t)row * bc_width + which * n_state + n);
                } else {
                    const int which = (k - 2 * NP) / kChannels, ch = min(c0 + (k - 2 * NP) % kChannels, channels - 1);
                    if (which == 0) v = raw_load<float>(dt_pre + (size_t)row * channels + ch);
                    else if (which == 1) v = raw_load<T>(x + (size_t)row * channels + ch);
                    else v = raw_load<T>(z + (size_t)row * z_stride + ch);
                }
            }
            fetched[j] = v;
        }
    };
    auto publish = [&](int buf, int n) {
        float* dst = stage_mem + buf * kStage * ROW;
#pragma unroll
        for (int j = 0; j < FETCH; ++j) {
            const int e = threadIdx.x + j * kThreads;
            if (e >= n * ROW) continue;          // what lies beyond the step's tokens is neither transformed nor read
            const int k = e % ROW;
            float v;
            if (k >= 2 * NP + 2 * kChannels) v = silu_of<T>(from_raw<T>(fetched[j]));
            else if (k >= 2 * NP + kChannels) v = from_raw<T>(fetched[j]);
            else if (k >= 2 * NP) v = softplus_of<T>(__uint_as_float(fetched[j]) + bias_mem[k - 2 * NP]);
            else v = from_raw<T>(fetched[j]);
            dst[e] = v;
        }
    };

    if (row1 - row0 == 1) {
        // a single token: straight from global memory, no stage and no barrier
        const float dt = softplus_of<T>(dt_pre[(size_t)row0 * channels + c] + dt_bias[c]);     // (bias_mem is not read here)
        const float xv = to_f32<T>(x[(size_t)row0 * channels + c]);
        const float dx = dt * xv;
        float part = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int n = lane + kLanes * i;
            const bool in = n < n_state;
            const float b = in ? to_f32<T>(bc[(size_t)row0 * bc_width + n]) : 0.f;
            const float cc = in ? to_f32<T>(bc[(size_t)row0 * bc_width + n_state + n]) : 0.f;
            s[i] = Decay<T>::of(dt, a[i]) * s[i] + dx * b;
            part += s[i] * cc;
            if (in && live) S[n] = s[i];
        }
#pragma unroll
        for (int off = kLanes / 2; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
        if (lane == 0 && live)
            y[(size_t)row0 * channels + c] = from_f32<T>((part + skip * xv) * silu_of<T>(to_f32<T>(z[(size_t)row0 * z_stride + c])));
        return;
    }
    if (row0 < row1) fetch(row0);
    __syncthreads();                                   // the channels' biases are in place
    if (row0 < row1) publish(0, min(kStage, row1 - row0));
    __syncthreads();
    for (int first = row0, buf = 0; first < row1; first += kStage, buf ^= 1) {
        const bool more = first + kStage < row1;
        if (more) fetch(first + kStage);
        // the loads stay here, ahead of the stage's work: sunk to where their values are stored, each
        // would wait for memory in its turn
        asm volatile("" ::: "memory");
        const float* src = stage_mem + buf * kStage * ROW;
        const int n_tokens = min(kStage, row1 - first);
        // (unrolled: only the state's multiply-add links one token to the next; the loads, the
        // exponentials and the shuffles of several tokens then overlap)
#pragma unroll 4
        for (int t = 0; t < n_tokens; ++t) {
            const float* tok = src + t * ROW;
            const float dt = tok[2 * NP + group], xv = tok[2 * NP + kChannels + group];
            const float dx = dt * xv;
            float part = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int n = lane + kLanes * i;
                s[i] = Decay<T>::of(dt, a[i]) * s[i] + dx * tok[n];
                part += s[i] * tok[NP + n];
            }
#pragma unroll
            for (int off = kLanes / 2; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
            if (lane == 0 && live)
                y[(size_t)(first + t) * channels + c] = from_f32<T>((part + skip * xv) * tok[2 * NP + 2 * kChannels + group]);
        }
        if (more) publish(buf ^ 1, min(kStage, row1 - first - kStage));
        __syncthreads();
    }
    if (live && row0 < row1) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int n = lane + kLanes * i;
            if (n < n_state) S[n] = s[i];
        }
    }
}

// ---------------------------------------------------------------- several tokens, bfloat16, states up to 32
//
// What a token costs a channel beside its state (loads, the softplus of the step size, the silu of the gate,
// the write) is more work than the state itself, and none of it waits for the token before.  So four warps
// of a block walk the state and nothing else, and eight (or four) others run ahead of and behind them: they load a
// stage of tokens, leave (step size, step size * input) and B, C in shared memory a stage ahead, and add up,
// gate and write the read-outs of the stage before.  LANES lanes hold a channel's state, PER neighbouring
// entries each, in pairs for the two-wide multiply-add; a lane leaves its share of a token's sum in shared
// memory for the other warps to add.  One barrier per stage, two buffers of everything.
// Either side is a chain of latencies: with four helping warps and the walk a token at a time, one prompt of 2,048 tokens and 4,096 channels
// took 141 us, the helpers alone 134, the walk alone 107.  The walk takes GROUP tokens' loads and exponentials ahead of their chain
// through the state, the helpers are twice as many: 118.  What bounds it now is shared memory (69 % of its cycles) and issue.  B200,
// against the kernel above, us: one prompt of 2,048 tokens, 4,096 channels 118 / 763, 8,192 channels 165 / 770; 8 x 512
// tokens of 4,096 153 / 447; 100 tokens 13 / 46.  (One set of warps for everything took 211 for the first; cutting
// the tokens into segments that run side by side doubles the exponentials; step sizes once instead of twice in shared memory 124; loads
// two stages ahead 137.)
constexpr int kWalkThreads = 128;          // threads of each of the two halves of a block
constexpr int kWalkStage = 16;

// the hardware's base-2 exponential (as Decay above; what would be below 2^-126 is zero)
__device__ __forceinline__ float decay_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A in base 2.  An infinite one (a decay of zero) becomes the largest number: times the step size of zero of the tokens that
// fill up a stage it must be zero, not a NaN.
__device__ __forceinline__ float bounded_rate(float a) {
    const float x = a * 1.4426950408889634f;
    return x < -3.4e38f ? -3.4e38f : x;
}

// The barrier at which the two halves of a block meet.  They wait for one another at different places of the program, which
// __syncthreads() does not allow: a numbered barrier of all the block's threads does.
template <int THREADS>
__device__ __forceinline__ void halves_meet() { asm volatile("barrier.cta.sync 1, %0;" ::"n"(THREADS) : "memory"); }

template <int LANES, int PER, int HELPERS, int GROUP>
__global__ void __launch_bounds__(kWalkThreads + HELPERS, HELPERS > 128 ? 2 : 3) selective_scan_walk_kernel(
    __nv_bfloat16* __restrict__ y, float* __restrict__ state, const __nv_bfloat16* __restrict__ x,
    const float* __restrict__ dt_pre, const float* __restrict__ dt_bias, const __nv_bfloat16* __restrict__ bc, int bc_width,
    const float* __restrict__ A, const float* __restrict__ D, const __nv_bfloat16* __restrict__ z, int z_stride,
    const int* __restrict__ cu_seqlens, const int* __restrict__ slots, int channels, int n_state) {
    pdl_launch_dependents();
    pdl_wait();
    using T = __nv_bfloat16;
    constexpr int N = LANES * PER, ST = kWalkStage, PAIRS = PER / 2, CH = kWalkThreads / LANES;
    using ull = unsigned long long;
    // a staged token: per lane its entries of B, then of C; per channel the step size twice, then its product with the input twice
    __shared__ __align__(16) float bc_mem[2][ST][2 * N];
    __shared__ __align__(16) float4 step_mem[2][ST][CH];
    __shared__ __align__(16) float share_mem[2][ST][CH * LANES];
    const int seq = blockIdx.y;
    const int row0 = cu_seqlens[seq], n_tokens = cu_seqlens[seq + 1] - row0;
    if (n_tokens <= 0) return;
    const int n_stages = (n_tokens + ST - 1) / ST;
    const int c0 = blockIdx.x * CH;

    if (threadIdx.x < kWalkThreads) {
        const int lane = threadIdx.x % LANES, group = threadIdx.x / LANES;
        const bool live = c0 + group < channels;
        const int c = live ? c0 + group : channels - 1;
        float* S = state + ((size_t)slots[seq] * channels + c) * n_state;
        ull s[PAIRS], a[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const int n = lane * PER + 2 * i;
            s[i] = pack2(n < n_state ? S[n] : 0.f, n + 1 < n_state ? S[n + 1] : 0.f);
            a[i] = pack2(n < n_state ? bounded_rate(A[(size_t)c * n_state + n]) : 0.f,
                         n + 1 < n_state ? bounded_rate(A[(size_t)c * n_state + n + 1]) : 0.f);
        }
        halves_meet<kWalkThreads + HELPERS>();                       // the first stage is in place
        for (int stage = 0; stage < n_stages; ++stage) {
            const int buf = stage & 1;
            // (tokens beyond the step's have a step size of zero and leave the state as it is)
#pragma unroll
            for (int t0 = 0; t0 < ST; t0 += GROUP) {
                ulonglong2 step[GROUP];
                ull b[GROUP][2 * PAIRS], decay[GROUP][PAIRS];
#pragma unroll
                for (int t = 0; t < GROUP; ++t) {
                    step[t] = *reinterpret_cast<const ulonglong2*>(&step_mem[buf][t0 + t][group]);
#pragma unroll
                    for (int i = 0; i < 2 * PAIRS; i += 2) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(bc_mem[buf][t0 + t] + lane * 2 * PER + 2 * i);
                        b[t][i] = v.x;
                        b[t][i + 1] = v.y;
                    }
                }
                if (GROUP > 1) asm volatile("" ::: "memory");
#pragma unroll
                for (int t = 0; t < GROUP; ++t)
#pragma unroll
                    for (int i = 0; i < PAIRS; ++i) {
                        float e0, e1;
                        unpack2(mul2(step[t].x, a[i]), e0, e1);
                        decay[t][i] = pack2(decay_exp2(e0), decay_exp2(e1));
                        b[t][i] = mul2(step[t].y, b[t][i]);
                    }
                float part[GROUP];
#pragma unroll
                for (int t = 0; t < GROUP; ++t) {
                    ull sum = 0;
#pragma unroll
                    for (int i = 0; i < PAIRS; ++i) {
                        s[i] = fma2(decay[t][i], s[i], b[t][i]);
                        sum = i == 0 ? mul2(s[i], b[t][PAIRS + i]) : fma2(s[i], b[t][PAIRS + i], sum);
                    }
                    float s0, s1;
                    unpack2(sum, s0, s1);
                    part[t] = s0 + s1;
                }
#pragma unroll
                for (int t = 0; t < GROUP; ++t) share_mem[buf][t0 + t][threadIdx.x] = part[t];
            }
            halves_meet<kWalkThreads + HELPERS>();
        }
        if (!live) return;
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const int n = lane * PER + 2 * i;
            float s0, s1;
            unpack2(s[i], s0, s1);
            if (n < n_state) S[n] = s0;
            if (n + 1 < n_state) S[n + 1] = s1;
        }
        return;
    }

    // the other half: a thread serves one channel and every (kWalkThreads / CH)-th token of a stage
    const int tid = threadIdx.x - kWalkThreads;
    constexpr int STRIDE = HELPERS / CH, OWN = ST / STRIDE;
    const int group = tid % CH, t0 = tid / CH;
    const bool live = c0 + group < channels;
    const int c = live ? c0 + group : channels - 1;
    const float skip = D[c], bias = dt_bias[c];
    constexpr int kShare = ST * 2 * N / HELPERS, kShareStep = HELPERS / (2 * N);
    static_assert(ST * 2 * N % HELPERS == 0 && HELPERS % (2 * N) == 0 && ST % STRIDE == 0, "whole shares");
    // this thread's column of the staged B and C: lane, B or C, entry
    const int share_col = tid % (2 * N), share_t = tid / (2 * N);
    const int share_n = share_col / (2 * PER) * PER + share_col % PER, share_which = share_col % (2 * PER) / PER;
    const bool share_in = share_n < n_state;
    const T* bc_src = bc + (size_t)(row0 + share_t) * bc_width + share_which * n_state + (share_in ? share_n : 0);
    const size_t first_row = row0 + t0, own_step = (size_t)STRIDE * channels, z_step = (size_t)STRIDE * z_stride;
    const float* dt_src = dt_pre + first_row * channels + c;
    const T* x_src = x + first_row * channels + c;
    const T* z_src = z + first_row * z_stride + c;
    T* y_dst = y + first_row * channels + c;
    uint32_t bc_raw[kShare] = {}, x_raw[OWN] = {}, z_raw[OWN] = {};
    float dt_raw[OWN] = {};
    float skipped[2][OWN], gate[2][OWN];
    auto fetch = [&](int stage) {
        const int left = n_tokens - stage * ST;
#pragma unroll
        for (int j = 0; j < kShare; ++j)
            if (share_in && share_t + j * kShareStep < left) bc_raw[j] = raw_load<T>(bc_src + (size_t)(j * kShareStep) * bc_width);
        bc_src += (size_t)ST * bc_width;
#pragma unroll
        for (int j = 0; j < OWN; ++j)
            if (t0 + j * STRIDE < left) {
                dt_raw[j] = dt_src[j * own_step];
                x_raw[j] = raw_load<T>(x_src + j * own_step);
                z_raw[j] = raw_load<T>(z_src + j * z_step);
            }
        dt_src += OWN * own_step;
        x_src += OWN * own_step;
        z_src += OWN * z_step;
    };
    auto transform = [&](int stage, int buf, float (&skipped_)[OWN], float (&gate_)[OWN]) {
        const int left = n_tokens - stage * ST;
#pragma unroll
        for (int j = 0; j < kShare; ++j) (&bc_mem[buf][0][0])[tid + j * HELPERS] = from_raw<T>(bc_raw[j]);
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const float d = t0 + j * STRIDE < left ? softplus_of<T>(dt_raw[j] + bias) : 0.f;
            const float in = from_raw<T>(x_raw[j]), din = d * in;
            step_mem[buf][t0 + j * STRIDE][group] = make_float4(d, d, din, din);
            skipped_[j] = skip * in;
            gate_[j] = silu_of<T>(from_raw<T>(z_raw[j]));
        }
    };
    auto finish = [&](int stage, int buf, const float (&skipped_)[OWN], const float (&gate_)[OWN]) {
        const int left = n_tokens - stage * ST;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const float4* share = reinterpret_cast<const float4*>(&share_mem[buf][t0 + j * STRIDE][group * LANES]);
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < LANES / 4; ++l) {
                const float4 v = share[l];
                sum += (v.x + v.y) + (v.z + v.w);
            }
            if (live && t0 + j * STRIDE < left) y_dst[j * own_step] = from_f32<T>((sum + skipped_[j]) * gate_[j]);
        }
        y_dst += OWN * own_step;
    };
    // (two stages a turn, so that the buffers' numbers are constants)
    fetch(0);
    transform(0, 0, skipped[0], gate[0]);
    if (1 < n_stages) fetch(1);
    halves_meet<kWalkThreads + HELPERS>();
    for (int stage = 0; stage < n_stages; stage += 2) {
        // the walk is at `stage`: read out the one before, prepare the one after
        if (stage > 0) finish(stage - 1, 1, skipped[1], gate[1]);
        if (stage + 1 < n_stages) transform(stage + 1, 1, skipped[1], gate[1]);
        if (stage + 2 < n_stages) fetch(stage + 2);
        halves_meet<kWalkThreads + HELPERS>();
        if (stage + 1 >= n_stages) break;
        finish(stage, 0, skipped[0], gate[0]);
        if (stage + 2 < n_stages) transform(stage + 2, 0, skipped[0], gate[0]);
        if (stage + 3 < n_stages) fetch(stage + 3);
        halves_meet<kWalkThreads + HELPERS>();
    }
    if (n_stages & 1) finish(n_stages - 1, 0, skipped[0], gate[0]);
    else finish(n_stages - 1, 1, skipped[1], gate[1]);
}

int launch_walk(void* y, float* state, const void* x, const float* dt_pre, const float* dt_bias, const void* bc, int bc_width,
                const float* A, const float* D, const void* z, int z_stride, const int* cu_seqlens, const int* slots, int n_rows, int max_tokens, int n_seqs,
                int channels, int n_state, cudaStream_t stream) {
    using T = __nv_bfloat16;
#define THN_WALK_LAUNCH(L, P, H, G)                                                                                               \
    thn_launch_ordered(selective_scan_walk_kernel<L, P, H, G>, dim3((channels + kWalkThreads / L - 1) / (kWalkThreads / L), n_seqs), \
                       kWalkThreads + H, 0, stream, (T*)y, state, (const T*)x, dt_pre, dt_bias, (const T*)bc, bc_width, A, D, \
                       (const T*)z, z_stride, cu_seqlens, slots, channels, n_state)
    // Eight lanes a channel put twice as many warps on the chip and issue more for the same sums: they win while the
    // blocks of four lanes (32 channels) do not fill it once.  Eight warps beside the four that walk: with four, these were what the
    // walk waited for.  But two blocks of twelve warps share a multiprocessor where three of eight do, and a wave of two takes three
    // quarters of the time of one of three: few waves that come out worse so take four, and so do very short sequences, which
    // have little to walk.  So do blocks that are many for the time of the longest sequence: they fill the chip either way, and with eight
    // issue more.  us, eight lanes and eight warps / four and eight / four and four, 16 entries: one prompt of 2,048 tokens, 4,096
    // channels 118 / 132 / 177, 8,192 channels 241 / 165 / 199; 2 x 700 tokens of 4,096 channels 89 / 62 / 75; 3 x 512 85 / 78 / 68;
    // 8 x 512 185 / 153 / 164; 64 x 16 101 / 75 / 70; 64 x 128 - / 300 / 287.  32 entries, eight / four warps: 2 x 700 150 / 181, 3 x 512 163 / 161,
    // 4 x 512 193 / 212, 64 x 16 171 / 133, 64 x 128 742 / 716.  8 entries: 64 x 128 278 / 252.
    auto blocks = [&](int lanes) { return ((long long)channels * lanes + kWalkThreads - 1) / kWalkThreads * n_seqs; };
    auto four = [&](int lanes) {
        const long long n = blocks(lanes);
        return n_rows < 64ll * n_seqs || (n <= 6 * 148 && (n + 295) / 296 * 3 > (n + 443) / 444 * 4) ||
               n * std::min(1.0, (double)n_rows / n_seqs / max_tokens) > (lanes == 4 ? 10 : 16) * 148;
    };
    if (n_state <= 8) {
        if (four(4)) THN_WALK_LAUNCH(4, 2, 128, 1);
        else THN_WALK_LAUNCH(4, 2, 256, 8);
    } else if (n_state <= 16 && blocks(4) <= 148) {
        THN_WALK_LAUNCH(8, 2, 256, 2);
    } else if (n_state <= 16) {
        if (four(4)) THN_WALK_LAUNCH(4, 4, 128, 1);
        else THN_WALK_LAUNCH(4, 4, 256, 8);
    } else {
        if (four(8)) THN_WALK_LAUNCH(8, 4, 128, 1);
        else THN_WALK_LAUNCH(8, 4, 256, 2);
    }
#undef THN_WALK_LAUNCH
    return thn_launch_status("selective_scan");
}

// Whether a step's rows are walked by the kernel above.  It takes a sequence's tokens sixteen at a time, so that one token
// costs as much as sixteen: a few prompts among many single tokens are cheaper token by token.  What the two take, in us on
// B200, to within a fifth of what was measured (4,096 channels, 16 entries, token by token / walked):
// two tokens of one sequence 6.3 / 4.8, beside 8 single tokens 7.7 / 11.9; 16 beside 8 10.4 / 12.3, beside 60 39 / 61; 128 beside
// 8 55 / 21, beside 60 57 / 66; 2,048 beside 60 770 / 205; 64 sequences of 2 59 / 66, of 4 70 / 66, of 16 133 / 70.
bool walk_pays(int n_rows, int max_tokens, int n_seqs, int channels) {
    const float width = channels / 4096.f;
    const long long longest = (max_tokens + kWalkStage - 1) / kWalkStage;
    const long long stages = std::min((long long)n_seqs * longest, n_rows / kWalkStage + (long long)n_seqs);      // at most
    const float by_token = 0.5f + std::max(0.37f * max_tokens, (0.09f * n_rows + 0.6f * n_seqs) * width);
    const float walked = std::max(1.1f * longest, 0.95f * stages * width);
    return max_tokens > 1 && walked <= by_token;
}

template <typename T>
int launch_scan(void* y, float* state, const void* x, const float* dt_pre, const float* dt_bias, const void* bc,
                int bc_width, const float* A, const float* D, const void* z, int z_stride, const int* cu_seqlens,
                const int* slots, int n_seqs, int channels, int n_state, cudaStream_t stream) {
#define THN_SCAN_LAUNCH(L, P)                                                                                           \
    thn_launch_ordered(selective_scan_kernel<T, L, P, (kStage * (2 * L * P + 3 * (kScanThreads / L)) + kScanThreads - 1) / kScanThreads>, \
                       dim3((channels + kScanThreads / L - 1) / (kScanThreads / L), n_seqs), kScanThreads, 0, stream, (T*)y, state, \
                       (const T*)x, dt_pre, dt_bias, (const T*)bc, bc_width, A, D, (const T*)z, z_stride, cu_seqlens, slots, \
                       channels, n_state)
    if (n_state <= 4) THN_SCAN_LAUNCH(4, 1);
    else if (n_state <= 8) THN_SCAN_LAUNCH(4, 2);
    else if (n_state <= 16) THN_SCAN_LAUNCH(4, 4);
    else if (n_state <= 32) THN_SCAN_LAUNCH(4, 8);
    else if (n_state <= 64) THN_SCAN_LAUNCH(8, 8);
    else THN_SCAN_LAUNCH(8, 16);
#undef THN_SCAN_LAUNCH
    return thn_launch_status("selective_scan");
}

}  // namespace

// out [rows, channels] of the activation type; the raw inputs are the columns [offset, offset +
// channels) of proj [rows, proj_width]; weight float32 [channels, taps] (the last tap is the
// current token's), bias float32 [channels] or null; ring [slots, taps, channels] of the
// activation type; seq_lens int32 [slots]: the tokens each slot held before the step.
THN_API int thn_causal_conv(void* out, const void* proj, int proj_width, int offset, const float* weight,
                            const float* bias, const void* ring, const int* row_slot, const int* row_pos,
                            const int* seq_lens, int n_rows, int channels, int taps, int dtype, cudaStream_t stream) {
    THN_CHECK_ARG(n_rows >= 0 && channels > 0 && taps > 0 && offset >= 0 && offset + channels <= proj_width,
                  "causal_conv: bad sizes");
    const long long n = (long long)n_rows * channels;
    if (n == 0) return THN_OK;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    const bool pieces = channels % 4 == 0 && offset % 4 == 0 && proj_width % 4 == 0 &&
                        (((uintptr_t)out | (uintptr_t)proj | (uintptr_t)ring) & 7) == 0 && ((uintptr_t)weight & 15) == 0;
    if (dtype == THN_BF16 && taps == kConvTaps && pieces && (n_rows + kConvRows - 1) / kConvRows <= 65535)
        thn_launch(conv_run::few_entries(n_rows, channels) ? causal_conv_vec_kernel<true> : causal_conv_vec_kernel<false>,
                   dim3((unsigned)((channels / 4 + 127) / 128), (unsigned)((n_rows + kConvRows - 1) / kConvRows)),
                   128, 0, stream, (__nv_bfloat16*)out, (const __nv_bfloat16*)proj, proj_width, offset, weight, bias,
                   (const __nv_bfloat16*)ring, row_slot, row_pos, seq_lens, n_rows, channels);
    else if (dtype == THN_F32)
        thn_launch(causal_conv_kernel<float>, blocks, 256, 0, stream, (float*)out, (const float*)proj, proj_width, offset,
                   weight, bias, (const float*)ring, row_slot, row_pos, seq_lens, n, channels, taps);
    else if (dtype == THN_BF16)
        thn_launch(causal_conv_kernel<__nv_bfloat16>, blocks, 256, 0, stream, (__nv_bfloat16*)out,
                   (const __nv_bfloat16*)proj, proj_width, offset, weight, bias, (const __nv_bfloat16*)ring, row_slot,
                   row_pos, seq_lens, n, channels, taps);
    else
        THN_CHECK_ARG(false, "causal_conv: unknown dtype %d", dtype);
    return thn_launch_status("causal_conv");
}

// The step's last raw inputs (at most taps per sequence) go into the ring, position p at p mod taps.
THN_API int thn_conv_ring_update(void* ring, const void* proj, int proj_width, int offset, const int* cu_seqlens,
                                 const int* slots, const int* seq_lens, int n_seqs, int channels, int taps, int dtype,
                                 cudaStream_t stream) {
    THN_CHECK_ARG(n_seqs >= 0 && channels > 0 && taps > 0 && offset >= 0 && offset + channels <= proj_width,
                  "conv_ring_update: bad sizes");
    THN_UNSUPPORTED_IF(n_seqs > 65535, "conv_ring_update: %d sequences", n_seqs);
    if (n_seqs == 0) return THN_OK;
    const dim3 grid((unsigned)min((long long)(((long long)taps * channels + 255) / 256), 64ll), n_seqs);
    if (dtype == THN_F32)
        thn_launch(conv_ring_update_kernel<float>, grid, 256, 0, stream, (float*)ring, (const float*)proj, proj_width,
                   offset, cu_seqlens, slots, seq_lens, channels, taps);
    else if (dtype == THN_BF16)
        thn_launch(conv_ring_update_kernel<__nv_bfloat16>, grid, 256, 0, stream, (__nv_bfloat16*)ring,
                   (const __nv_bfloat16*)proj, proj_width, offset, cu_seqlens, slots, seq_lens, channels, taps);
    else
        THN_CHECK_ARG(false, "conv_ring_update: unknown dtype %d", dtype);
    return thn_launch_status("conv_ring_update");
}

// y, x [rows, channels] of the activation type; state float32 [slots, channels, n_state], read and
// updated; dt_pre float32 [rows, channels], dt_bias float32 [channels]; bc [rows, bc_width] of the
// activation type: B in the first n_state columns, C in the next; A float32 [channels, n_state]
// (negative); D float32 [channels]; z of the activation type, rows z_stride apart.
THN_API int thn_selective_scan(void* y, float* state, const void* x, const float* dt_pre, const float* dt_bias,
                               const void* bc, int bc_width, const float* A, const float* D, const void* z, int z_stride,
                               const int* cu_seqlens, const int* slots, int n_rows, int max_tokens, int n_seqs, int channels, int n_state, int dtype,
                               cudaStream_t stream) {
    THN_CHECK_ARG(n_seqs >= 0 && channels > 0 && n_state > 0 && bc_width >= 2 * n_state && z_stride >= channels,
                  "selective_scan: bad sizes");
    THN_UNSUPPORTED_IF(n_state > 128, "selective_scan: a state of %d per channel, at most 128", n_state);
    THN_UNSUPPORTED_IF(n_seqs > 65535, "selective_scan: %d sequences", n_seqs);
    if (n_seqs == 0) return THN_OK;
    if (dtype == THN_F32)
        return launch_scan<float>(y, state, x, dt_pre, dt_bias, bc, bc_width, A, D, z, z_stride, cu_seqlens, slots, n_seqs,
                                  channels, n_state, stream);
    if (dtype == THN_BF16 && n_state <= 32 && walk_pays(n_rows, max_tokens, n_seqs, channels))
        return launch_walk(y, state, x, dt_pre, dt_bias, bc, bc_width, A, D, z, z_stride, cu_seqlens, slots, n_rows, max_tokens, n_seqs,
                           channels, n_state, stream);
    if (dtype == THN_BF16)
        return launch_scan<__nv_bfloat16>(y, state, x, dt_pre, dt_bias, bc, bc_width, A, D, z, z_stride, cu_seqlens, slots,
                                          n_seqs, channels, n_state, stream);
    THN_CHECK_ARG(false, "selective_scan: unknown dtype %d", dtype);
    return THN_OK;
}
