// Recurrences over a matrix state S [128 keys, values] whose decay is one number per head and token, or one
// per head, token and key, walked a chunk of 32 tokens at a time, for prompts with bfloat16 activations.  Token by token such a
// kernel is a chain of thousands of dependent steps.  Inside a chunk the sums can be taken in any order:
//
//     o_i  = alpha_i S0^T q_i + beta_i sum_{j <= i} G_ij v_j
//     S    = alpha_last S0 + beta_last sum_j w_j k_j v_j^T
//
// with S0 the state ahead of the chunk.  A kernel of the mixer works out, for all chunks at once, G (the
// products q_i . k_j with the decays between the two tokens, zero for j > i) and the numbers per token;
// what is left to walk is three products per chunk.  The delta rule's values are v = u - W S0 with rows u
// and W that its kernel has worked out too.  The gated matrix memory keeps the logarithms' running maximum
// m, a number that only the walk knows: alpha and beta come from it, and a vector n beside S.  With a decay
// per key the mixer's kernel has multiplied it into the queries, the keys and G, and S is decayed by a number per key.
//
// The products run on the tensor cores in bfloat16 with operands split into three parts, x = h + m + l exactly (24
// bits), and the six products of parts that reach 2^-24: h h; and, in an accumulator of their own, h m, m h, m m,
// h l, l h (operands that come in bfloat16 are exact in one part, and the products fewer).  The tensor core's
// accumulation rounds towards zero, so every step of 16 along the sum's axis has a fresh accumulator and
// the steps meet in float32 additions.  (tf32 in two parts costs the same and is off by 2.4e-7 where the
// token-by-token delta rule is off by 1.3e-7 and this by 1.4e-7.)  The mixer's kernels leave their operands split, as
// planes of bfloat16 in rows that ldmatrix reads without bank conflicts: split in the walk they were half
// of its instructions (177 us for 2,048 tokens of 16 heads of the delta rule, 157 with planes).
//
// A block walks one sequence, head and 16 CG columns of values.  S^T lives in the accumulator registers of
// its warps: warp (cg, ks) holds 16 columns and 128 / KS keys; the accumulator layout of two groups of eight
// keys is the A operand's layout, so S never moves.  With KS > 1 the warps' shares of W S0 and S0^T q meet in
// shared memory, each warp then finishes some of the tokens.  The next chunk's operands travel into the other of STAGES
// buffers (with one buffer, other blocks of the multiprocessor cover the wait); rows beyond the sequence's are zeros.
//
// Who brings them: the warps themselves, by asynchronous copies of 16 bytes, or (BROUGHT, where the operands lie in planes) four more
// warps, by bulk copies of whole planes.  The first hold every warp up for as long as a chunk takes to come from L2 (1,765 of a chunk's
// 4,630 clocks for the delta rule of 16 heads, 1,225 of 3,700 for 32 heads with a decay per key), but start sooner and leave room for more
// blocks: they stay where blocks are many and short.  (One more warp takes 1,200 clocks to start a chunk's bulk copies, most of the time that the others
// need for it.)  Blocks of 16 and 32 columns are brought however short the sequences: over 370 steps, 33 tokens and more, copying was never faster by more than
// 2 %, but for linear attention's 33 tokens beside 8 single ones (29.4 / 32.0 us); us of the whole call, copying / brought, 16 columns: one prompt of 33 tokens, delta rule of 8 heads
// 35 / 27, linear attention of 16 heads 18.0 / 17.1, 128 tokens, state-space duality of 64 heads 51 / 46.  The wait for what is brought is bounded: after kWaitLimitNs by the global timer the block sets
// THN_ERR_WAIT_TIMEOUT, lets what is on its way land and returns; its results and state are then not written, those of other blocks may be.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace chunk {

constexpr int kTokens = 32;           // tokens per chunk
constexpr int kKeys = 128;
// rows of the planes, in bfloat16: eight rows of 16 bytes lie on distinct banks
constexpr int kKeyRow = kKeys + 8, kScoreRow = kTokens + 8;

// Where the chunks of a sequence stand among the chunks of all, counted from its first row on; chunk_places: how many places
// there are.  (A sequence of n rows from row0 on takes (n + 31) / 32 places, never more than lie ahead of the next one's.)
__host__ __device__ inline size_t chunk_place(int row0, int seq) { return (size_t)row0 / kTokens + seq; }
inline long long chunk_places(int n_rows, int n_seqs) { return n_rows / kTokens + (long long)n_seqs; }

struct WalkArgs {
    float* o;                  // [rows, heads, value_dim]
    float* state;              // [slots, heads, value_dim, kKeys], read and updated
    // planes of bfloat16 (three, or one where q, k and v are bfloat16): plane p, unit u, row m from
    // q + p * key_plane + u * key_unit + m * key_row (elements); k likewise
    const __nv_bfloat16* q;
    const __nv_bfloat16* k;
    long long key_plane, key_unit, key_row;
    const void* v;             // float32 or bfloat16; row m, head h: v + m * v_row + h * v_head
    long long v_row, v_head;
    const __nv_bfloat16* w;    // delta: [heads][3][rows][kKeyRow]
    const __nv_bfloat16* scores;   // G: [heads][3][rows][kScoreRow]
    const float4* scalars;     // [heads][rows]: (alpha, -, w, -); gated: (sum of log f, maximum, w, sum of the row of G)
    const int* cu_seqlens;
    const int* slots;
    int n_rows, n_heads, heads_per_unit, value_dim;
    float scale;               // on every read-out
    // the gated matrix memory
    float* normaliser;         // [slots, heads, value_dim / 16, kKeys + 1]: copies of n, then m
    const float* key_sums;     // [chunk_place, heads, kKeys]: sum_j w_j k_j of every chunk; a decay per key: the chunk's decay of S
    float floor_;
    int* err;                  // the caller's error word, or null: walks that are brought need one
    int skip_loads;            // the test of the bounded wait: nothing is brought
};

__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "r"(there ? 16 : 0));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// kTokens rows of ROW elements that lie one behind the other, to shared memory as they are; zeros beyond
// `there` rows (the addresses of those are not read).
template <int ROW, int THREADS>
__device__ __forceinline__ void copy_rows(__nv_bfloat16* smem, const __nv_bfloat16* gmem, int there) {
    static_assert(ROW % 8 == 0, "whole pieces");
    constexpr int kPieces = kTokens * ROW / 8;
    const int end = there * (ROW / 8);
#pragma unroll
    for (int e = 0; e < kPieces; e += THREADS) {
        const int i = e + (int)threadIdx.x;
        if (kPieces % THREADS == 0 || i < kPieces) copy16(smem + i * 8, gmem + (i < end ? i * 8 : 0), i < end);
    }
}

constexpr unsigned long long kWaitLimitNs = 20ull * 1000 * 1000;
__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_addr(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase with the given parity.  Returns false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    WaitClock clock;
    for (int spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(shared_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spin & 15) == 15 && clock.ran_out(kWaitLimitNs)) return false;
    }
}
// 16-byte aligned on both sides, whole pieces of 16 bytes; counted by `bar`.
__device__ __forceinline__ void copy_bulk(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(shared_addr(smem)), "l"(gmem), "r"(bytes), "r"(shared_addr(bar)) : "memory");
}
// The other way; the thread that starts such stores waits for them with stores_wait.
__device__ __forceinline__ void store_bulk(void* gmem, const void* smem, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\ncp.async.bulk.commit_group;"
                 ::"l"(gmem), "r"(shared_addr(smem)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void stores_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// The barrier hears of this thread's copies of 16 bytes when they have landed.
__device__ __forceinline__ void copies_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(shared_addr(bar)) : "memory");
}
__device__ __forceinline__ void barrier_sync(int id, int threads) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// Whether all threads of the block say yes, and a barrier.
__device__ __forceinline__ bool all_agree(bool yes) {
    uint32_t all;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %1, 0;\n"
        "barrier.cta.red.and.pred q, 0, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(all)
        : "r"((uint32_t)yes)
        : "memory");
    return all != 0;
}
// What threads have written to shared memory stands ahead of the bulk copies that are started behind the next barrier.
__device__ __forceinline__ void writes_ahead_of_copies() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// Nonzero where one of the two halves is an infinity or a NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t two) { return ((two & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }
__device__ __forceinline__ bool finite(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ float not_a_number() { return __uint_as_float(0x7fffffffu); }
__device__ __forceinline__ float low_half(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_half(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// two floats in three parts each: part[0] + part[1] + part[2], exactly
struct Split {
    uint32_t part[3];
};
__device__ __forceinline__ Split split(float x, float y) {
    Split s;
    s.part[0] = pack_bf16(x, y);
    x -= low_half(s.part[0]);
    y -= high_half(s.part[0]);
    s.part[1] = pack_bf16(x, y);
    x -= low_half(s.part[1]);
    y -= high_half(s.part[1]);
    s.part[2] = pack_bf16(x, y);
    return s;
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// four 8 x 8 matrices of bfloat16; lane l gives the address of row l % 8 of matrix l / 8
__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
// Where a lane's address lies inside a 16 x 16 tile of rows of `row` elements:
// an A operand [m][k], or B operands of two neighbouring groups of n stored [k][n] (loaded transposed)
__device__ __forceinline__ int a_tile(int lane, int row) { return ((lane & 7) + (lane >> 3 & 1) * 8) * row + (lane >> 4) * 8; }
// B operands of two neighbouring groups of n stored [n][k], or an A operand stored [k][m] (loaded transposed)
__device__ __forceinline__ int b_tile(int lane, int row) { return ((lane & 7) + (lane >> 4) * 8) * row + (lane >> 3 & 1) * 8; }

// The A operand of a step of 16 along the sum's axis, in parts.
struct Parts {
    uint32_t part[3][4];
};
// from rows g and g + 8 at k = 2t, 2t + 1 and at k = 2t + 8, 2t + 9
__device__ __forceinline__ Parts parts_of(float2 g_lo, float2 g8_lo, float2 g_hi, float2 g8_hi) {
    Parts p;
    const Split s[4] = {split(g_lo.x, g_lo.y), split(g8_lo.x, g8_lo.y), split(g_hi.x, g_hi.y), split(g8_hi.x, g8_hi.y)};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) p.part[j][i] = s[i].part[j];
    return p;
}
// The B operands of two neighbouring groups of eight columns, in parts: part[p][2 n + half of k]
template <int PARTS>
struct Columns {
    uint32_t part[PARTS][4];
};
template <int PARTS>
__device__ __forceinline__ Columns<PARTS> columns_of(const __nv_bfloat16* p, int plane) {
    Columns<PARTS> c;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) load_matrices(c.part[i], p + i * plane);
    return c;
}
template <int PARTS>
__device__ __forceinline__ Columns<PARTS> columns_transposed(const __nv_bfloat16* p, int plane) {
    Columns<PARTS> c;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) load_matrices_transposed(c.part[i], p + i * plane);
    return c;
}
// large += h h, small += the other products, over PAIRS pairs of groups of columns: product by product, so that
// neighbouring instructions have accumulators of their own.  A_PARTS 1: A is exact in one part.
template <int A_PARTS = 3, int PARTS, int PAIRS>
__device__ __forceinline__ void multiply(float (&large)[2 * PAIRS][4], float (&small)[2 * PAIRS][4], const Parts& a,
                                         const Columns<PARTS> (&b)[PAIRS]) {
    auto all = [&](float (&d)[2 * PAIRS][4], int x, int y) {
#pragma unroll
        for (int n = 0; n < 2 * PAIRS; ++n) mma(d[n], a.part[x], b[n / 2].part[y % PARTS][2 * (n & 1)], b[n / 2].part[y % PARTS][2 * (n & 1) + 1]);
    };
    if (A_PARTS == 3) all(small, 2, 0);
    if (PARTS == 3) all(small, 0, 2);
    if (A_PARTS == 3 && PARTS == 3) all(small, 1, 1);
    all(large, 0, 0);
    if (A_PARTS == 3) all(small, 1, 0);
    if (PARTS == 3) all(small, 0, 1);
}
// One step's sum.  The accumulation rounds towards zero; kLean of the result is put back in the finer units of
// the small products (the factor of least error: 0 and 4.3e-8 are both worse by a tenth).
constexpr float kLean = 2.2e-8f;
__device__ __forceinline__ float joined(float large, float small) { return large + fmaf(large, kLean, small); }
template <int N>
__device__ __forceinline__ void clear(float (&d)[N][4]) {
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) d[n][i] = 0.f;
}
__device__ __forceinline__ float2 pair_of(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 pair_of(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

// Of a chunk's values as A operands (columns by tokens), those that are not finite become zero; from[0], from[1]: the first
// token of columns g and g + 8 that had one.
template <int PARTS>
__device__ __forceinline__ void leave_out(Parts (&values)[kTokens / 16], int (&from)[2], int t) {
    from[0] = from[1] = kTokens;
#pragma unroll
    for (int j = 0; j < kTokens / 16; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t which = not_finite(values[j].part[0][i]);
            const int token = 16 * j + 8 * (i >> 1) + 2 * t;
            if (which & 0x80000000u) from[i & 1] = min(from[i & 1], token + 1);
            if (which & 0x00008000u) from[i & 1] = min(from[i & 1], token);
            const uint32_t kept = (which & 0x80000000u ? 0u : 0xffff0000u) | (which & 0x00008000u ? 0u : 0x0000ffffu);
#pragma unroll
            for (int p = 0; p < (PARTS == 1 ? 1 : 3); ++p) values[j].part[p][i] &= kept;
        }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        from[c] = min(from[c], __shfl_xor_sync(0xffffffffu, from[c], 1));
        from[c] = min(from[c], __shfl_xor_sync(0xffffffffu, from[c], 2));
    }
}

// What the mixer's recurrence is.
enum Kind {
    kPlain,        // a decay per token
    kDelta,        // values less what the state holds
    kGated,        // a running maximum beside it, read-outs divided
    kPerKey        // a decay per token and key, already in the queries, the keys and G
};

template <typename T, int CG, int KS, Kind KIND, int STAGES, bool BROUGHT>
struct Layout {
    static constexpr bool DELTA = KIND == kDelta;
    static constexpr int kParts = sizeof(T) == 2 && KIND != kPerKey ? 1 : 3;      // of queries and keys
    static constexpr int kThreads = 32 * CG * KS, kColumns = 16 * CG;
    static constexpr int kBringers = BROUGHT ? 128 : 0;            // threads that bring the operands
    static_assert(!BROUGHT || (kParts == 3 && STAGES == 2), "planes, two buffers");
    static constexpr int kValueRow = kColumns + (sizeof(T) == 2 ? 8 : 4);
    static constexpr int kKeyPlane = kTokens * kKeyRow, kScorePlane = kTokens * kScoreRow;      // elements
    static constexpr int kQ = 0;
    static constexpr int kK = kQ + kParts * kKeyPlane * 2;
    static constexpr int kW = kK + kParts * kKeyPlane * 2;
    static constexpr int kG = kW + (DELTA ? 3 * kKeyPlane * 2 : 0);
    static constexpr int kV = kG + 3 * kScorePlane * 2;
    static constexpr int kScalars = kV + kTokens * kValueRow * (int)sizeof(T);
    static constexpr int kSums = kScalars + kTokens * 16;                                    // gated: the chunk's sum of keys
    static constexpr int kStage = kSums + (KIND == kGated || KIND == kPerKey ? kKeys * 4 : 0);
    static constexpr int kShares = KS > 1 ? KS * CG * (DELTA ? 2 : 1) * 4 * 32 * 16 : 0;    // [ks][cg][which][8 tokens][lane] float4
    static constexpr int kBytes = STAGES * kStage + kShares + (kTokens * 3 + kKeys + 4) * 4 + STAGES * 8;
};

template <typename T, int CG, int KS, Kind KIND, int STAGES, bool BROUGHT>
__global__ void __launch_bounds__(32 * CG * KS + (BROUGHT ? 128 : 0), STAGES == 1 ? 512 / (32 * CG * KS) : 1) walk_kernel(WalkArgs a) {
    using L = Layout<T, CG, KS, KIND, STAGES, BROUGHT>;
    constexpr bool DELTA = KIND == kDelta, GATED = KIND == kGated, PER_KEY = KIND == kPerKey;
    constexpr int PARTS = L::kParts, VALUE_PARTS = sizeof(T) == 2 ? 1 : 3;
    constexpr int KT = kKeys / KS / 8;               // groups of 8 keys of a warp
    constexpr int GROUPS = kTokens / 8;              // groups of 8 tokens
    constexpr int OWN = GROUPS / KS;                 // groups that a warp finishes
    static_assert(KT % 4 == 0 && OWN >= 1, "whole steps");
    static_assert(!DELTA || KS > 1, "the barrier ahead of the shares frees the chunk's queries and W");
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char mem[];
    float4* shares = reinterpret_cast<float4*>(mem + STAGES * L::kStage);
    float* alpha_s = reinterpret_cast<float*>(mem + STAGES * L::kStage + L::kShares);     // gated: per token
    float* beta_s = alpha_s + kTokens;
    float* under_s = beta_s + kTokens;
    float* n_s = under_s + kTokens;
    int* lost_s = reinterpret_cast<int*>(n_s + kKeys);      // delta: a value was not finite, in this chunk or ahead of it
    uint64_t* full = reinterpret_cast<uint64_t*>(lost_s + 4);        // [STAGES] a chunk has landed
    const int slab = blockIdx.x, head = blockIdx.y, seq = blockIdx.z;
    if (DELTA && threadIdx.x == 0) *lost_s = 0;
    if (BROUGHT && threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) mbar_init(full + i, L::kBringers + 1);      // their copies, and the bytes' announcement
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (BROUGHT) __syncthreads();
    const int row0 = a.cu_seqlens[seq], n_tokens = a.cu_seqlens[seq + 1] - row0;
    if (n_tokens <= 0) return;
    const int slot = a.slots[seq], unit = head / a.heads_per_unit, n_chunks = (n_tokens + kTokens - 1) / kTokens;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int cg = warp / KS, ks = warp % KS, key0 = ks * (kKeys / KS);
    const int group0 = ks * OWN;                     // the first group of tokens that this warp finishes
    const int col0 = slab * L::kColumns;
    const __nv_bfloat16* q_src = a.q + unit * a.key_unit + row0 * a.key_row;
    const __nv_bfloat16* k_src = a.k + unit * a.key_unit + row0 * a.key_row;
    const long long w_plane = (long long)a.n_rows * kKeyRow, g_plane = (long long)a.n_rows * kScoreRow;
    const __nv_bfloat16* w_src = DELTA ? a.w + head * 3 * w_plane + (long long)row0 * kKeyRow : nullptr;
    const __nv_bfloat16* g_src = a.scores + head * 3 * g_plane + (long long)row0 * kScoreRow;
    const T* v_src = static_cast<const T*>(a.v) + row0 * a.v_row + head * a.v_head + col0;
    const float4* scalar_src = a.scalars + (long long)head * a.n_rows + row0;

    if (BROUGHT && warp >= CG * KS) {
        // ---- the warps that bring the operands: W, the queries, the keys and G, a plane a lane, and the values' rows
        const int bringer = threadIdx.x - L::kThreads, p = min(lane, 2);
        auto bring = [&](int chunk) {
            if (a.skip_loads) return;
            unsigned char* dst = mem + (chunk % STAGES) * L::kStage;
            uint64_t* bar = full + chunk % STAGES;
            const int first = chunk * kTokens, n_here = min(kTokens, n_tokens - first);
            constexpr uint32_t kRowBytes = (DELTA ? 9 : 6) * kKeyRow * 2 + 3 * kScoreRow * 2 + (PER_KEY ? 0 : 16);
            if (bringer == 0) mbar_expect(bar, n_here * kRowBytes + (PER_KEY ? kKeys * 4 : 0));
            const uint32_t key_bytes = n_here * kKeyRow * 2;
            const long long key_at = (long long)first * kKeyRow;
            if (bringer < 32) {
                if (DELTA && lane < 3) copy_bulk(dst + L::kW + p * L::kKeyPlane * 2, w_src + p * w_plane + key_at, key_bytes, bar);
                if (PER_KEY && lane == 0)
                    copy_bulk(dst + L::kSums, a.key_sums + ((chunk_place(row0, seq) + chunk) * a.n_heads + head) * kKeys, kKeys * 4, bar);
            } else if (bringer < 64) {
                if (lane < 3) copy_bulk(dst + L::kQ + p * L::kKeyPlane * 2, q_src + p * a.key_plane + key_at, key_bytes, bar);
            } else if (bringer < 96) {
                if (lane < 3) copy_bulk(dst + L::kK + p * L::kKeyPlane * 2, k_src + p * a.key_plane + key_at, key_bytes, bar);
            } else {
                if (lane < 3)
                    copy_bulk(dst + L::kG + p * L::kScorePlane * 2, g_src + p * g_plane + (long long)first * kScoreRow, n_here * kScoreRow * 2, bar);
                else if (!PER_KEY && lane == 3)
                    copy_bulk(dst + L::kScalars, scalar_src + first, n_here * 16, bar);
            }
            constexpr int kPer16 = 16 / (int)sizeof(T), kValueCopies = L::kColumns / kPer16;
#pragma unroll
            for (int e = bringer; e < kTokens * kValueCopies; e += L::kBringers) {
                const int i = e / kValueCopies, c = e % kValueCopies * kPer16;
                const bool there = i < n_here;
                copy16(dst + L::kV + (i * L::kValueRow + c) * (int)sizeof(T), v_src + (there ? first + i : 0) * a.v_row + c, there);
            }
            copies_arrive(bar);
        };
        bring(0);
        if (n_chunks > 1) bring(1);
        for (int chunk = 0; chunk < n_chunks; ++chunk) {
            if (!all_agree(true)) {
                let_copies_land();
                return;
            }
            if (chunk > 0 && chunk + 1 < n_chunks) bring(chunk + 1);      // (the chunk ahead of this one is through: its buffer is free)
        }
        return;
    }
    auto issue = [&](int chunk) {
        unsigned char* dst = mem + (chunk % STAGES) * L::kStage;
        const int first = chunk * kTokens, n_here = min(kTokens, n_tokens - first);
        __nv_bfloat16* q_dst = reinterpret_cast<__nv_bfloat16*>(dst + L::kQ);
        __nv_bfloat16* k_dst = reinterpret_cast<__nv_bfloat16*>(dst + L::kK);
        if (PARTS == 3) {
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                copy_rows<kKeyRow, L::kThreads>(q_dst + p * L::kKeyPlane, q_src + p * a.key_plane + (long long)first * kKeyRow, n_here);
                copy_rows<kKeyRow, L::kThreads>(k_dst + p * L::kKeyPlane, k_src + p * a.key_plane + (long long)first * kKeyRow, n_here);
            }
        } else {
            // (a thread copies the same column of some rows, the same distance apart in every chunk)
            constexpr int kRowsApart = L::kThreads / (kKeys / 8);
            const int i0 = threadIdx.x / (kKeys / 8), c = threadIdx.x % (kKeys / 8) * 8;
            const __nv_bfloat16* q_from = q_src + c + (first + i0) * a.key_row;
            const __nv_bfloat16* k_from = k_src + c + (first + i0) * a.key_row;
#pragma unroll
            for (int u = 0; u < kTokens / kRowsApart; ++u) {
                const bool there = i0 + u * kRowsApart < n_here;
                copy16(q_dst + (i0 + u * kRowsApart) * kKeyRow + c, there ? q_from : q_src, there);
                copy16(k_dst + (i0 + u * kRowsApart) * kKeyRow + c, there ? k_from : k_src, there);
                q_from += kRowsApart * a.key_row;
                k_from += kRowsApart * a.key_row;
            }
        }
        if ((GATED || PER_KEY) && threadIdx.x < kKeys / 4)
            copy16(dst + L::kSums + threadIdx.x * 16,
                   a.key_sums + ((chunk_place(row0, seq) + chunk) * a.n_heads + head) * kKeys + threadIdx.x * 4, true);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            if (DELTA)
                copy_rows<kKeyRow, L::kThreads>(reinterpret_cast<__nv_bfloat16*>(dst + L::kW) + p * L::kKeyPlane,
                                                w_src + p * w_plane + (long long)first * kKeyRow, n_here);
            copy_rows<kScoreRow, L::kThreads>(reinterpret_cast<__nv_bfloat16*>(dst + L::kG) + p * L::kScorePlane,
                                              g_src + p * g_plane + (long long)first * kScoreRow, n_here);
        }
        constexpr int kPer16 = 16 / (int)sizeof(T), kValueCopies = L::kColumns / kPer16;
        for (int e = threadIdx.x; e < kTokens * kValueCopies; e += L::kThreads) {
            const int i = e / kValueCopies, c = e % kValueCopies * kPer16;
            const bool there = i < n_here;
            copy16(dst + L::kV + (i * L::kValueRow + c) * (int)sizeof(T), v_src + (there ? first + i : 0) * a.v_row + c, there);
        }
        for (int i = threadIdx.x; !PER_KEY && i < kTokens; i += L::kThreads)
            copy16(dst + L::kScalars + i * 16, scalar_src + (i < n_here ? first + i : 0), i < n_here);
        copy_commit();
    };
    if (!BROUGHT) issue(0);

    // S^T: s[j][0], s[j][1]: column g, keys 8j + 2t and the one after; s[j][2], s[j][3]: column g + 8
    float s[KT][4];
    float* S = a.state + (((size_t)slot * a.n_heads + head) * a.value_dim + col0 + cg * 16) * kKeys + key0;
#pragma unroll
    for (int j = 0; j < KT; ++j) {
        const float2 x = *reinterpret_cast<const float2*>(S + g * kKeys + 8 * j + 2 * t);
        const float2 y = *reinterpret_cast<const float2*>(S + (g + 8) * kKeys + 8 * j + 2 * t);
        s[j][0] = x.x; s[j][1] = x.y; s[j][2] = y.x; s[j][3] = y.y;
    }
    float m = 0.f;
    float* nm = nullptr;
    if (GATED) {
        nm = a.normaliser + (((size_t)slot * a.n_heads + head) * (a.value_dim / 16) + slab * CG) * (kKeys + 1);
        for (int d = threadIdx.x; d < kKeys; d += L::kThreads) n_s[d] = nm[d];
        m = nm[kKeys];
    }
    const int key_at = b_tile(lane, kKeyRow) + key0;          // this lane's address in a tile of 16 tokens and 16 keys
    const int key_at_transposed = a_tile(lane, kKeyRow) + key0;

    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        // this chunk is in place; the other buffer, and the shares, are free again
        if constexpr (BROUGHT) {
            if (!all_agree(mbar_wait(full + chunk % STAGES, chunk / STAGES & 1))) {
                if (threadIdx.x == 0) atomicOr(a.err, THN_ERR_WAIT_TIMEOUT);
                let_copies_land();
                return;
            }
        } else {
            if (STAGES == 1 && chunk > 0) {
                __syncthreads();           // the only stage is free again
                issue(chunk);
            }
            copy_wait_all();
            __syncthreads();
            if (STAGES > 1 && chunk + 1 < n_chunks) issue(chunk + 1);
        }
        unsigned char* stage = mem + (chunk % STAGES) * L::kStage;
        const __nv_bfloat16* q_s = reinterpret_cast<const __nv_bfloat16*>(stage + L::kQ);
        const __nv_bfloat16* k_s = reinterpret_cast<const __nv_bfloat16*>(stage + L::kK);
        const __nv_bfloat16* w_s = reinterpret_cast<const __nv_bfloat16*>(stage + L::kW);
        const __nv_bfloat16* g_s = reinterpret_cast<const __nv_bfloat16*>(stage + L::kG);
        T* v_s = reinterpret_cast<T*>(stage + L::kV) + cg * 16;
        const float4* scalars = reinterpret_cast<const float4*>(stage + L::kScalars);
        const int first = chunk * kTokens, n_here = min(kTokens, n_tokens - first);
        if (BROUGHT && n_here < kTokens) {
            // the sequence's last chunk: zeros where rows beyond it would enter the state (queries and G's rows enter their own read-outs
            // alone, and G's columns behind a row's token are zero)
            auto clear_rows = [&](int at, int row_bytes) {
                for (int e = n_here * row_bytes / 16 + threadIdx.x; e < kTokens * row_bytes / 16; e += L::kThreads)
                    *reinterpret_cast<uint4*>(stage + at + e * 16) = make_uint4(0, 0, 0, 0);
            };
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                clear_rows(L::kK + p * L::kKeyPlane * 2, kKeyRow * 2);
                if (DELTA) clear_rows(L::kW + p * L::kKeyPlane * 2, kKeyRow * 2);
            }
            if (!PER_KEY) clear_rows(L::kScalars, 16);
            barrier_sync(1, L::kThreads);
        }

        if (GATED) {
            // alpha, beta and the denominators of the chunk's tokens; four threads share a token's n . q
            static_assert(!GATED || L::kThreads >= kTokens * 4, "four threads per token");
            if (threadIdx.x < kTokens * 4) {
                const int i = threadIdx.x >> 2, part = threadIdx.x & 3;
                const float4 sc = scalars[i];
                const float top = fmaxf(sc.x + m, sc.y);
                const float alpha = expf(sc.x + m - top), beta = expf(sc.y - top);
                float dot0 = 0.f, dot1 = 0.f;
#pragma unroll
                for (int d = 0; d < kKeys / 8; ++d) {
                    const float2 q = pair_of(q_s + i * kKeyRow + 2 * (part + 4 * d));
                    const float2 n = pair_of(n_s + 2 * (part + 4 * d));
                    dot0 = fmaf(q.x, n.x, dot0);
                    dot1 = fmaf(q.y, n.y, dot1);
                }
                float dot = dot0 + dot1;
                dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                dot += __shfl_xor_sync(0xffffffffu, dot, 2);
                if (part == 0) {
                    alpha_s[i] = alpha;
                    beta_s[i] = beta;
                    under_s[i] = fmaxf(fabsf((alpha * dot + beta * sc.w) * a.scale), expf(-top)) + a.floor_;
                }
            }
        }

        // this warp's keys of S0^T q (and W S0): over the chunk's tokens, columns 16 cg ..
        float read[4][4], fixed[4][4];
#pragma unroll
        for (int j = 0; j < KT; j += 2) {
            const Parts p = parts_of(make_float2(s[j][0], s[j][1]), make_float2(s[j][2], s[j][3]),
                                     make_float2(s[j + 1][0], s[j + 1][1]), make_float2(s[j + 1][2], s[j + 1][3]));
            const int at = key_at + 8 * j;
            auto share = [&](float (&sum)[4][4], const auto& columns) {
                float large[4][4], small[4][4];
                clear(large);
                clear(small);
                multiply(large, small, p, columns);
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[n][i] = j == 0 ? joined(large[n][i], small[n][i]) : sum[n][i] + joined(large[n][i], small[n][i]);
            };
            if constexpr (DELTA) {
                const Columns<3> w[2] = {columns_of<3>(w_s + at, L::kKeyPlane), columns_of<3>(w_s + at + 16 * kKeyRow, L::kKeyPlane)};
                share(fixed, w);
            }
            const Columns<PARTS> q[2] = {columns_of<PARTS>(q_s + at, L::kKeyPlane), columns_of<PARTS>(q_s + at + 16 * kKeyRow, L::kKeyPlane)};
            share(read, q);
        }
        constexpr int WHICH = DELTA ? 2 : 1;
        if (KS > 1) {
            float4* own = shares + (size_t)(ks * CG + cg) * WHICH * 4 * 32 + lane;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                own[n * 32] = make_float4(read[n][0], read[n][1], read[n][2], read[n][3]);
                if (DELTA) own[(4 + n) * 32] = make_float4(fixed[n][0], fixed[n][1], fixed[n][2], fixed[n][3]);
            }
        }
        if (KS > 1 || GATED) barrier_sync(1, L::kThreads);
        if (KS > 1) {
            // (the sums are taken in the order of the keys, whoever takes them)
#pragma unroll
            for (int n = 0; n < OWN; ++n) {
#pragma unroll
                for (int which = 0; which < WHICH; ++which) {
                    float (&dst)[4] = which == 0 ? read[n] : fixed[n];
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int other = 0; other < KS; ++other) {
                        const float4 x = shares[((size_t)(other * CG + cg) * WHICH * 4 + which * 4 + group0 + n) * 32 + lane];
                        sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
                    }
                    dst[0] = sum.x; dst[1] = sum.y; dst[2] = sum.z; dst[3] = sum.w;
                }
            }
        }
        // The delta rule's values v = u - W S0, as they are and times w, go out as planes [column][token] over the chunk's queries
        // and W, which no warp reads any more: split by the warps that finish them, once (one prompt of 2,048 tokens of 32
        // heads 397 -> 362 us against every warp splitting them).
        constexpr int kSplitRow = kTokens + 8, kSplitPlane = 16 * kSplitRow;
        __nv_bfloat16* plain_s = reinterpret_cast<__nv_bfloat16*>(stage + L::kQ) + cg * 3 * kSplitPlane;
        __nv_bfloat16* scaled_s = reinterpret_cast<__nv_bfloat16*>(stage + L::kW) + cg * 3 * kSplitPlane;
        if constexpr (DELTA) {
            uint32_t own_lost = 0;
#pragma unroll
            for (int n = 0; n < OWN; ++n) {
                const int i = 8 * (group0 + n) + 2 * t;
                const T* u = v_s + i * L::kValueRow + g;
                const float w0 = scalars[i].z, w1 = scalars[i + 1].z;
                const float v[4] = {u[0] - fixed[n][0], u[L::kValueRow] - fixed[n][1], u[8] - fixed[n][2], u[L::kValueRow + 8] - fixed[n][3]};
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int at = (g + 8 * half) * kSplitRow + i;
                    const Split as_is = split(v[2 * half], v[2 * half + 1]), by_w = split(v[2 * half] * w0, v[2 * half + 1] * w1);
                    own_lost |= not_finite(as_is.part[0]);
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        *reinterpret_cast<uint32_t*>(plain_s + p * kSplitPlane + at) = as_is.part[p];
                        *reinterpret_cast<uint32_t*>(scaled_s + p * kSplitPlane + at) = by_w.part[p];
                    }
                }
            }
            if (own_lost) *lost_s = 1;
            if (BROUGHT) writes_ahead_of_copies();
            barrier_sync(1, L::kThreads);
        }
        // the chunk's values as A operands: columns by tokens, as they are and times w
        Parts plain[kTokens / 16], scaled[kTokens / 16];
#pragma unroll
        for (int j = 0; j < kTokens / 16; ++j) {
            if constexpr (DELTA) {
                const int at = a_tile(lane, kSplitRow) + 16 * j;
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    load_matrices(scaled[j].part[p], scaled_s + p * kSplitPlane + at);
                    load_matrices(plain[j].part[p], plain_s + p * kSplitPlane + at);
                }
                continue;
            }
            float2 v[4];        // column g, g + 8 at tokens 2t, 2t + 1; the same at 2t + 8, 2t + 9
            if constexpr (VALUE_PARTS == 1) {
                load_matrices_transposed(plain[j].part[0], v_s + 16 * j * L::kValueRow + b_tile(lane, L::kValueRow));
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = make_float2(low_half(plain[j].part[0][i]), high_half(plain[j].part[0][i]));
            } else {
                const T* src = v_s + (16 * j + 2 * t) * L::kValueRow + g;
                v[0] = make_float2(src[0], src[L::kValueRow]);
                v[1] = make_float2(src[8], src[L::kValueRow + 8]);
                src += 8 * L::kValueRow;
                v[2] = make_float2(src[0], src[L::kValueRow]);
                v[3] = make_float2(src[8], src[L::kValueRow + 8]);
                plain[j] = parts_of(v[0], v[1], v[2], v[3]);
            }
            if constexpr (PER_KEY) continue;
            const float4* sc = scalars + 16 * j + 2 * t;
            const float w0 = sc[0].z, w1 = sc[1].z, w8 = sc[8].z, w9 = sc[9].z;
            scaled[j] = parts_of(make_float2(v[0].x * w0, v[0].y * w1), make_float2(v[1].x * w0, v[1].y * w1),
                                 make_float2(v[2].x * w8, v[2].y * w9), make_float2(v[3].x * w8, v[3].y * w9));
        }
        // the state behind the chunk
        const float keep = PER_KEY ? 1.f : GATED ? alpha_s[n_here - 1] : scalars[n_here - 1].x, take = GATED ? beta_s[n_here - 1] : 1.f;
        constexpr int KP = 2;                        // pairs of groups of keys at a time
#pragma unroll
        for (int n = 0; n < KT; n += 2 * KP) {
            float sum[2 * KP][4];
#pragma unroll
            for (int j = 0; j < kTokens / 16; ++j) {
                const __nv_bfloat16* p = k_s + key_at_transposed + 16 * j * kKeyRow + 8 * n;
                Columns<PARTS> k[KP];
#pragma unroll
                for (int o = 0; o < KP; ++o) k[o] = columns_transposed<PARTS>(p + 16 * o, L::kKeyPlane);
                float large[2 * KP][4], small[2 * KP][4];
                clear(large);
                clear(small);
                if constexpr (PER_KEY) multiply<VALUE_PARTS>(large, small, plain[j], k);
                else multiply(large, small, scaled[j], k);
#pragma unroll
                for (int o = 0; o < 2 * KP; ++o)
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[o][i] = j == 0 ? joined(large[o][i], small[o][i]) : sum[o][i] + joined(large[o][i], small[o][i]);
            }
#pragma unroll
            for (int o = 0; o < 2 * KP; ++o) {
                float2 by_key = make_float2(keep, keep);
                if constexpr (PER_KEY) by_key = pair_of(reinterpret_cast<const float*>(stage + L::kSums) + key0 + 8 * (n + o) + 2 * t);
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n + o][i] = fmaf(i & 1 ? by_key.y : by_key.x, s[n + o][i], take * sum[o][i]);
            }
        }
        // sum_j G_ij v_j for this warp's tokens, and the read-outs
        // (G's rows are loaded for 16 tokens at a time; with one group of tokens a warp, two warps share them)
        constexpr int kPairs = OWN >= 2 ? OWN / 2 : 1;
        float inner[kPairs][2][4];
        const int pair0 = group0 / 2;
        auto take_inner = [&] {
#pragma unroll
            for (int pair = 0; pair < kPairs; ++pair) {
                clear(inner[pair]);
#pragma unroll
                for (int j = 0; j < kTokens / 16; ++j) {
                    if (j > pair0 + pair) continue;
                    const Columns<3> row[1] = {columns_of<3>(g_s + b_tile(lane, kScoreRow) + 16 * (pair0 + pair) * kScoreRow + 16 * j, L::kScorePlane)};
                    float large[2][4], small[2][4];
                    clear(large);
                    clear(small);
                    multiply<VALUE_PARTS>(large, small, plain[j], row);
#pragma unroll
                    for (int o = 0; o < 2; ++o)
#pragma unroll
                        for (int i = 0; i < 4; ++i) inner[pair][o][i] += joined(large[o][i], small[o][i]);
                }
            }
        };
        take_inner();
        // Where G is zero the products multiply all the same, and zero times an infinity or a NaN is NaN: such a value would
        // reach the tokens ahead of its own.  Where a warp has one, the products are taken again without it, and the column's
        // sums are NaN from its token on.  (The state has taken it as it is.)  The delta rule's values are looked at by the warps that
        // finish them.
        bool lost;
        if constexpr (DELTA) {
            lost = *reinterpret_cast<volatile int*>(lost_s) != 0;
        } else {
            uint32_t own = 0;
#pragma unroll
            for (int j = 0; j < kTokens / 16; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) own |= not_finite(plain[j].part[0][i]);
            lost = __any_sync(0xffffffffu, own != 0);
        }
        if (lost) {
            int from[2];
            leave_out<VALUE_PARTS>(plain, from, t);
            take_inner();
#pragma unroll
            for (int pair = 0; pair < kPairs; ++pair)
#pragma unroll
                for (int o = 0; o < 2; ++o)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (16 * (pair0 + pair) + 8 * o + 2 * t + (i & 1) >= from[i >> 1]) inner[pair][o][i] = not_a_number();
        }
#pragma unroll
        for (int n = 0; n < OWN; ++n) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = 8 * (group0 + n) + 2 * t + half;
                if (i >= n_here) continue;
                const int o = OWN == 1 ? group0 & 1 : n & 1;
                const float in0 = o ? inner[n / 2][1][half] : inner[n / 2][0][half];
                const float in1 = o ? inner[n / 2][1][2 + half] : inner[n / 2][0][2 + half];
                const float alpha = PER_KEY ? 1.f : GATED ? alpha_s[i] : scalars[i].x, beta = GATED ? beta_s[i] : 1.f;
                float y0 = (alpha * read[n][half] + beta * in0) * a.scale;
                float y1 = (alpha * read[n][2 + half] + beta * in1) * a.scale;
                if (GATED) {
                    y0 /= under_s[i];
                    y1 /= under_s[i];
                }
                float* dst = a.o + ((size_t)(row0 + first + i) * a.n_heads + head) * a.value_dim + col0 + cg * 16 + g;
                dst[0] = y0;
                dst[8] = y1;
            }
        }
        if (GATED) {
            const float4 sc = scalars[n_here - 1];
            m = fmaxf(sc.x + m, sc.y);
            // (every n . q of the chunk was taken ahead of the barrier above; the next chunk's wait behind one too)
            const float* sums = reinterpret_cast<const float*>(stage + L::kSums);
            for (int d = threadIdx.x; d < kKeys; d += L::kThreads) n_s[d] = fmaf(keep, n_s[d], take * sums[d]);
        }
    }
#pragma unroll
    for (int j = 0; j < KT; ++j) {
        *reinterpret_cast<float2*>(S + g * kKeys + 8 * j + 2 * t) = make_float2(s[j][0], s[j][1]);
        *reinterpret_cast<float2*>(S + (g + 8) * kKeys + 8 * j + 2 * t) = make_float2(s[j][2], s[j][3]);
    }
    if (GATED) {
        for (int copy = 0; copy < CG; ++copy) {       // (a thread stores the entries of n that it holds)
            for (int d = threadIdx.x; d < kKeys; d += L::kThreads) nm[copy * (kKeys + 1) + d] = n_s[d];
            if (threadIdx.x == 0) nm[copy * (kKeys + 1) + kKeys] = m;
        }
    }
}

template <typename T, int CG, int KS, Kind KIND, int STAGES, bool BROUGHT>
void launch_walk(const WalkArgs& a, int n_seqs, cudaStream_t stream) {
    using L = Layout<T, CG, KS, KIND, STAGES, BROUGHT>;
    static_assert(L::kBytes <= 227 * 1024, "what a block may have");
    auto kernel = walk_kernel<T, CG, KS, KIND, STAGES, BROUGHT>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes);
    thn_launch_ordered(kernel, dim3(a.value_dim / L::kColumns, a.n_heads, n_seqs), L::kThreads + L::kBringers, L::kBytes, stream, a);
}

// The walk whose operands are brought, where the caller has an error word in which its wait can say that it ran out; otherwise the warps copy
// themselves, with the same results to the bit.
template <typename T, int CG, int KS, Kind KIND>
void launch_brought_walk(const WalkArgs& a, int n_seqs, cudaStream_t stream) {
    if (a.err) launch_walk<T, CG, KS, KIND, 2, true>(a, n_seqs, stream);
    else launch_walk<T, CG, KS, KIND, 2, false>(a, n_seqs, stream);
}

// What a step's walk takes in blocks of one shape, in us: a time to start; the longest sequence's chain of chunks, as often as its blocks must queue,
// `per_sm` of them to a multiprocessor (0: any number), which is a whole number where all sequences are as long; what all chunks and sequences take
// together, per hundred heads of 128 values; and how much of the shorter of both stays beside the longer.  The mixers' tables are fitted to measured
// times of hundreds of steps: by pairs of sequence and head alone, single tokens beside a prompt count as much as the prompt, and blocks are too wide for its chain.
struct WalkCost {
    float start, chain, chunk, sequence, side;
    int columns, per_sm;
};
constexpr int kMultiprocessors = 148;

// The shape of the least such time, from 1 on; the first one's columns divide all values.
template <int N>
int cheapest_walk(const WalkCost (&costs)[N], int n_rows, int max_tokens, int n_seqs, int n_heads, int value_dim) {
    const long long longest = (max_tokens + kTokens - 1) / kTokens;
    const long long chunks = std::min(n_seqs * longest, n_rows / kTokens + (long long)n_seqs);      // at most
    const double heads = (double)n_heads * value_dim / 128, together = heads * std::min((double)n_seqs, (double)n_rows / max_tokens);
    const bool same = (long long)n_seqs * max_tokens == n_rows;
    int best = 1;
    double least = 0;
    for (int i = 0; i < N; ++i) {
        const WalkCost& c = costs[i];
        if (value_dim % c.columns != 0) continue;
        double waves = c.per_sm ? together * 128 / c.columns / (kMultiprocessors * c.per_sm) : 1.0;
        waves = std::max(1.0, same ? std::ceil(waves) : waves);
        const double chain = c.chain * longest * waves, all = (c.chunk * chunks + c.sequence * n_seqs) * heads / 100;
        const double us = c.start + std::max(chain, all) + c.side * std::min(chain, all);
        if (i == 0 || us < least) {
            best = i + 1;
            least = us;
        }
    }
    return best;
}

// ---------------------------------------------------------------- what the mixers' own kernels share

// Inclusive sum over the lanes of a warp.
__device__ __forceinline__ double lanes_cumulative(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    return v;
}
// The logarithm of a decay in [0, 1]; a decay of zero gets one whose exponential is zero in float32, so that differences of
// sums of logarithms stay numbers.  A NaN stays one.
constexpr double kLogOfNothing = -200.0;
__device__ __forceinline__ double log_decay(float a) { return a <= 0.f ? kLogOfNothing : log((double)a); }

// Rows 16 m_tile .. of x times all 32 rows of y, both planes of kKeys in shared memory: out[n][..] are
// the products of rows (g, g, g + 8, g + 8) with rows 8n + (2t, 2t + 1, 2t, 2t + 1); groups of y that lie
// behind all of x's rows are left out (zero).
template <int PARTS>
__device__ __forceinline__ void dots(float (&out)[4][4], const __nv_bfloat16* x, const __nv_bfloat16* y, int m_tile, int lane) {
    constexpr int kPlane = kTokens * kKeyRow;
    const __nv_bfloat16* xa = x + 16 * m_tile * kKeyRow + a_tile(lane, kKeyRow);
    const __nv_bfloat16* yb = y + b_tile(lane, kKeyRow);
    clear(out);
#pragma unroll
    for (int j = 0; j < kKeys / 16; ++j) {
        Parts p;
#pragma unroll
        for (int i = 0; i < PARTS; ++i) load_matrices(p.part[i], xa + i * kPlane + 16 * j);
#pragma unroll
        for (int pair = 0; pair < 2; ++pair) {
            if (pair > m_tile) continue;
            float large[2][4], small[2][4];
            clear(large);
            clear(small);
            const Columns<PARTS> c[1] = {columns_of<PARTS>(yb + 16 * pair * kKeyRow + 16 * j, kPlane)};
            multiply<PARTS>(large, small, p, c);
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int i = 0; i < 4; ++i) out[2 * pair + o][i] += joined(large[o][i], small[o][i]);
        }
    }
}

// Two neighbouring entries of a row, in three planes.
__device__ __forceinline__ void store_split(__nv_bfloat16* p, long long plane, float x, float y) {
    const Split s = split(x, y);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(p + i * plane) = s.part[i];
}

}  // namespace chunk
