// Shared device helpers for the sm_100a kernels of this library.
//
// Activation type T is float (the true 32-bit path) or __nv_bfloat16 (serving).
// rnd<T>(x) rounds a float to T's precision and returns it as float: the identity for
// float, round-to-nearest-even for bfloat16.  The kernels place it exactly where the
// reference rounds (engine/kernels/torch_ref.py:16-29).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define THN_API extern "C" __attribute__((visibility("default")))

enum ThnDtype { THN_F32 = 0, THN_BF16 = 1 };

// Error codes returned by the launchers (0 = ok, 1..999 = cudaError_t of the launch).
enum ThnStatus {
    THN_OK = 0,
    THN_BAD_ARGUMENT = 1001,
    THN_UNSUPPORTED = 1002,
};

// Bits set by kernels in the caller's device error word.
enum ThnDeviceError {
    THN_ERR_TOKEN_RANGE = 1,     // a token id outside [0, vocab)
    THN_ERR_PAGE_UNMAPPED = 2,   // a cache position whose page is not mapped
    THN_ERR_POSITION_RANGE = 4,  // a position beyond the rotary table
    THN_ERR_WAIT_TIMEOUT = 8,    // a bounded wait on a barrier gave up
};

void thn_set_error(const char* fmt, ...);

#define THN_CHECK_ARG(cond, ...)              \
    do {                                      \
        if (!(cond)) {                        \
            thn_set_error(__VA_ARGS__);       \
            return THN_BAD_ARGUMENT;          \
        }                                     \
    } while (0)

#define THN_UNSUPPORTED_IF(cond, ...)         \
    do {                                      \
        if (cond) {                           \
            thn_set_error(__VA_ARGS__);       \
            return THN_UNSUPPORTED;           \
        }                                     \
    } while (0)

static inline int thn_launch_status(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        thn_set_error("%s: launch failed: %s", what, cudaGetErrorString(e));
        return (int)e;
    }
    return THN_OK;
}

// Programmatic dependent launch.  Every kernel of this library says at its start that the
// next kernel in the stream may be scheduled (pdl_launch_dependents), and waits for the
// kernels before it to finish (pdl_wait) before it reads anything they wrote or writes
// anything at all.  What a kernel does between the two must depend on nothing but constant
// data (weights): it runs while the previous kernel is still at work.  Without the launch
// attribute both are no-ops.  Neither is a spin: the wait is the hardware's own.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

extern int g_thn_pdl;   // 1: launch with programmatic stream serialization (elementwise.cu)

template <typename... Params, typename... Args>
inline void thn_launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                       Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = g_thn_pdl ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);   // the caller reads cudaGetLastError
}

// A launch in plain stream order, whatever the switch says: for kernels whose time is set by how
// evenly their blocks are spread over the SMs.  Blocks of a kernel that is scheduled while its
// predecessor still runs go wherever that one leaves room, several to an SM; a kernel with
// about a block per SM and a long chain of dependent steps in each then takes twice as long.
template <typename... Params, typename... Args>
inline void thn_launch_ordered(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                               Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = nullptr;
    config.numAttrs = 0;
    cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);   // the caller reads cudaGetLastError
}

// The same with the blocks grouped into thread-block clusters of the given shape.
template <typename... Params, typename... Args>
inline void thn_launch_cluster(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                               dim3 cluster, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = cluster.x;
    attribute[0].val.clusterDim.y = cluster.y;
    attribute[0].val.clusterDim.z = cluster.z;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = g_thn_pdl ? 2 : 1;
    cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);   // the caller reads cudaGetLastError
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T> __device__ __forceinline__ float rnd(float v) { return to_f32<T>(from_f32<T>(v)); }

// Transcendentals of the recurrent layers.  On the true 32-bit path (T = float) they are computed
// in double and rounded once: a float32 expf leans one way by a fraction of an ulp, and a decay
// that multiplies a state a thousand times over carries that lean into the logits.  With
// bfloat16 activations the float32 functions are exact enough by a wide margin.
template <typename T> __device__ __forceinline__ float exp_of(float x) { return expf(x); }
template <> __device__ __forceinline__ float exp_of<float>(float x) { return (float)exp((double)x); }
template <typename T> __device__ __forceinline__ float silu_of(float x) { return x / (1.0f + expf(-x)); }
template <> __device__ __forceinline__ float silu_of<float>(float x) { return (float)((double)x / (1.0 + exp(-(double)x))); }
// softplus(x) = ln(1 + e^x)
template <typename T> __device__ __forceinline__ float softplus_of(float x) { return x > 20.f ? x : log1pf(expf(x)); }
template <> __device__ __forceinline__ float softplus_of<float>(float x) {
    return x > 40.f ? x : (float)log1p(exp((double)x));
}

// Two floats in a 64-bit register and the two-wide float32 operations on them (each half rounded as alone).
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result.  The order of
// additions depends only on blockDim, never on the data or the grid.
__device__ __forceinline__ float block_sum(float v, float* scratch /* >= 33 floats */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int n_warps = (blockDim.x + 31) >> 5;
        float t = lane < n_warps ? scratch[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// The clock of the bounded waits on mbarriers: time by the global timer, in which a step from one
// look at the timer to the next counts for kWaitStepCapNs at most.  Looks are microseconds apart
// while a kernel runs; a longer step means that the GPU ran another process in between (time
// slicing), and that time is not waiting: a wait that took it for such would give up with its
// copies and products still in flight.
constexpr unsigned long long kWaitStepCapNs = 100ull * 1000;
struct WaitClock {
    unsigned long long last = 0, waited = 0;
    // One look at the timer.  True once the waiting seen so far exceeds limit_ns.
    __device__ __forceinline__ bool ran_out(unsigned long long limit_ns) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (last != 0) {
            const unsigned long long step = now - last;
            waited += step < kWaitStepCapNs ? step : kWaitStepCapNs;
        }
        last = now;
        return waited > limit_ns;
    }
};
// What a block does ahead of its end where one of its waits has run out: copies and products that it has started are given a
// millisecond to land, for what lands later lands in the shared memory of the multiprocessor's next block.
__device__ __forceinline__ void let_copies_land() {
    WaitClock clock;
    while (!clock.ran_out(1000 * 1000)) __nanosleep(1000);
}

// How attention scores are shaped between q . k and the softmax, beyond the plain scale:
//   temperature  the scores of the query at position p are multiplied by
//                1 + temp_coef * ln(floor((p + 1) / temp_every) + 1)       (temp_every 0: none)
//   cap          score <- cap * tanh(score / cap)                           (cap 0: none)
// in this order, after the scale.  float32 throughout.
struct ScoreShape {
    float cap;
    float temp_coef;
    int temp_every;
    __host__ __device__ bool active() const { return cap > 0.f || temp_every > 0; }
    // the factor on the scores of the row at position pos
    __device__ __forceinline__ float row_factor(int pos) const {
        return temp_every > 0 ? 1.0f + temp_coef * logf((float)((pos + 1) / temp_every) + 1.0f) : 1.0f;
    }
    // the cap, with the library's tanh: for the kernels that compute a score at a time
    __device__ __forceinline__ float capped(float s) const { return cap > 0.f ? cap * tanhf(s / cap) : s; }
};

// tanh from one exponential and one division, both of the fast kind: absolute error about
// 2e-7 everywhere (it saturates to +-1 exactly), which is what the tensor-core attention
// kernels need of a capped score.
__device__ __forceinline__ float tanh_by_exp2(float x) {
    const float e = exp2f(x * 2.8853900817779268f);      // e^(2x)
    return 1.0f - __fdividef(2.0f, 1.0f + e);
}

// Geometry of one cache entry: pages of page_size tokens; inside a page K then V, each
// [n_kv][page_size][head_dim] (V: [n_kv][page_size][value_dim] where values have a size of
// their own; kernels that take such entries address them with kv_offset_sized).
struct PagedKV {
    const void* base;      // first byte of this entry's pool
    const int* block_table;  // [max_slots][bt_stride] physical page of (slot, logical page), -1 = unmapped
    int bt_stride;
    int n_kv;
    int page_size;
    int head_dim;
    int value_dim;         // size of a value where it differs from a key's; 0: the same (head_dim)
};

__device__ __forceinline__ long long kv_offset(const PagedKV& kv, int page, int which, int kvh, int in_page) {
    return ((((long long)page * 2 + which) * kv.n_kv + kvh) * kv.page_size + in_page) * (long long)kv.head_dim;
}

// The same for entries whose values may have a size of their own: element offset of key
// (which = 0) or value (which = 1) `in_page` of kv head `kvh` in `page`.
__device__ __forceinline__ long long kv_offset_sized(const PagedKV& kv, int page, int which, int kvh, int in_page) {
    const long long dv = kv.value_dim > 0 ? kv.value_dim : kv.head_dim;
    const long long k_block = (long long)kv.n_kv * kv.page_size * kv.head_dim;
    const long long page_base = (long long)page * (k_block + (long long)kv.n_kv * kv.page_size * dv);
    if (which == 0) return page_base + ((long long)kvh * kv.page_size + in_page) * kv.head_dim;
    return page_base + k_block + ((long long)kvh * kv.page_size + in_page) * dv;
}
