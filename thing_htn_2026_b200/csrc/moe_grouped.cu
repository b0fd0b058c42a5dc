// A mixture of experts over many rows as products of the chosen experts alone, on Blackwell's
// fifth-generation tensor cores.  (The dense form, every expert over every row, multiplies eight experts
// where two are chosen.)
//
//   moe_sort_kernel    the (row, choice) pairs in the order of their experts, and among one expert's in
//                      the order of the rows; one block per expert.
//   moe_gather_kernel  the rows of x in that order.
//   pair_gemm_kernel   the products.  kGlu, kGelu: up-projections with the experts' activation and the
//                      routing weight as the epilogue, the sorted rows of all experts and the shared
//                      expert's (all rows, as they are) in one launch.  kPartial: the experts' down-projections,
//                      a float32 row per pair.  kCombine: the shared expert's down-projection, to which the
//                      epilogue adds the row's float32 partial sums, in the order in which its experts were
//                      chosen; one rounding.
//   moe_combine_kernel the same sum where there is no shared expert.
//
// The products are of pairs of blocks on neighbouring multiprocessors (tcgen05 with cta_group::2): a tile is
// 256 rows of the weight by up to 256 rows of x, of which each block holds half of either operand, so that a
// step of 64 along the sum brings 32 KB to a multiprocessor for 512 clocks of products.  (One block
// per tile of 128 x 256 brings 48 KB for as many, more than the L2 cache delivers: 1.0-1.19 PFLOP/s.)
// The weight is the wide operand (the accumulator's lanes) and the rows of x are its columns, because the
// instruction takes any multiple of 32 columns: an expert's rows are cut into equal tiles of at most 256, and the
// last one costs what it holds.  For kGlu a block's 128 weight rows are 64 gates and the 64 ups that belong to them;
// the warps that read them from tensor memory hand each other half of their columns through shared memory.
//
// The rows of a pair's tile do not touch one another: a row's result depends on its own entries alone.
//
// B200, 2,048 rows of 2,048, eight experts of 1,024 of which two are chosen, a shared one, gated: sort 6 us, gather 5, up-projections 56 (51 GFLOP: 0.92
// PFLOP/s; 196 tiles are 2.6 a pair, and the last one's epilogue stands alone), down-projections 27 and 20; the layer 125 us, 207 in the
// dense form.  The up-projections keep the tensor pipe 50 % busy, the L2 cache 32 % and the issue slots 34 %: what is left is the tail.  Sixteen epilogue warps: with eight the up-projections took 62 us.
//
// Every wait on an mbarrier is bounded: after kWaitLimitNs by the global timer the waiter sets
// THN_ERR_WAIT_TIMEOUT in the caller's error word and goes on to the common exit, where
// tensor memory is given back.  A pair's two blocks are one cluster and always resident together; no wait depends on
// another pair.
#include <cuda.h>
#include <math.h>

#include "common.cuh"

namespace {

constexpr int kFeatures = 256, kRows = 256, BK = 64, UMMA_K = 16;    // a pair's tile
constexpr int kStages = 6;
constexpr int kEpilogueGroups = 4, kEpilogueWarps = 4 * kEpilogueGroups;      // (a group reads all 128 lanes of a chunk of 32 columns)
constexpr int kThreads = 64 + 32 * kEpilogueWarps;       // warp 0: TMA, warp 1: products and tensor memory, the others: epilogue
constexpr int kTmemCols = 512;                           // two accumulators of 256 columns
constexpr uint32_t kABytes = kFeatures / 2 * BK * 2, kBBytes = kRows / 2 * BK * 2;     // of one block
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr int kMaxGroups = 256;                          // experts
constexpr int kHandBytes = kEpilogueGroups * 16 * 128 * 4;     // kGlu: [group][16 columns][128 lanes]
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + kHandBytes + (kMaxGroups + 2) * 4 + 1024 /* alignment */ + 256 /* barriers */;
constexpr unsigned long long kWaitLimitNs = 20ull * 1000 * 1000;

enum Mode { kGlu, kGelu, kPartial, kCombine };
// rows of x in a tile: a chunk of columns per group of warps where a thread keeps its columns' partial sums in registers
constexpr int tile_rows(int mode) { return mode == kCombine ? 32 * kEpilogueGroups : kRows; }

struct PairArgs {
    int n_experts;               // groups of sorted rows (kCombine: 0)
    const int* offsets;          // [n_experts + 1] where they begin
    const int* sorted_row;       // kGlu, kGelu: the row of a sorted position
    const float* sorted_weight;  // and its weight
    int n_rows;                  // rows of the shared expert (0: none)
    int n_features, shared_features;     // outputs of an expert (kPartial, kCombine: of all)
    int up_row;                  // kGlu: how many weight rows the ups lie behind the gates
    int k;                       // entries of a sum
    void* out;                   // [sorted positions, n_features]: bfloat16; kPartial: float32
    __nv_bfloat16* shared_out;   // [rows, shared_features]
    float limit, shared_limit, alpha, up_shift;
    int weight_output;
    const float* shared_logit;   // the rows' gate logits of the shared expert, logit_stride apart, or null
    long long logit_stride;
    const float* partial;        // kCombine: [sorted positions, n_features]
    const int* place;            // [rows, top]: the sorted position of a row's choices
    int top;
    int* err;
    int skip_loads;              // the test of the bounded waits: nothing is loaded
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t block_in_pair() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the address, as a cluster sees it, of the leading block's copy of something in shared memory
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_addr(p)));
    return a;
}
__device__ __forceinline__ void pair_barrier() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase with the given parity.  Returns false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_addr(bar);
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
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spin & 15) == 15 && clock.ran_out(kWaitLimitNs)) return false;
    }
}
// Whether all threads of a named barrier say yes.
__device__ __forceinline__ bool all_of(bool yes, int barrier, int threads) {
    uint32_t all;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %1, 0;\n"
        "barrier.cta.red.and.pred q, %2, %3, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(all)
        : "r"((uint32_t)yes), "r"(barrier), "r"(threads)
        : "memory");
    return all != 0;
}
// A tile to this block's shared memory, its bytes counted by the leading block's barrier.
__device__ __forceinline__ void load_tile(void* dst, const CUtensorMap* map, uint32_t leader_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(leader_bar), "r"(x), "r"(y)
        : "memory");
}
// Shared-memory matrix descriptor of a K-major tile in rows of 128 bytes with the 128-byte swizzle (see gemm_tcgen05.cu).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// Instruction descriptor, kind::f16: float32 from bfloat16, both K-major, M = 256 over the pair, N = columns.
__device__ __forceinline__ uint32_t instruction(int columns) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns >> 3) << 17) | ((uint32_t)(kFeatures >> 4) << 24);
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t instr, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(instr), "r"(accumulate)
        : "memory");
}
// The barrier at this place in both blocks hears of the products issued so far.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_addr(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tmem_load_32(uint32_t taddr, float (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
          "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
          "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]),
          "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One tile: rows [row0, row0 + here) of its group's operand (sorted positions, or rows for the shared expert)
// by a pair's share of features from `feature` on; `columns`: the rows rounded up to what the instruction takes.
struct Tile {
    int group, row0, here, columns, feature;
    bool shared;
};

template <int N>
struct Number {
    static constexpr int value = N;
};

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) pair_gemm_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_sorted,
    const __grid_constant__ CUtensorMap map_x, PairArgs a) {
    pdl_launch_dependents();
    constexpr int kTileFeatures = MODE == kGlu ? kFeatures / 2 : kFeatures, kTileRows = tile_rows(MODE);
    constexpr uint32_t kLoaded = kABytes + kTileRows / 2 * BK * 2;      // bytes of a step, per block
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* hand = reinterpret_cast<float*>(tiles + (size_t)kStages * kStageBytes);
    int* first_tile = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(hand) + kHandBytes);     // [groups + 1]
    uint64_t* full = reinterpret_cast<uint64_t*>(first_tile + kMaxGroups + 2);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;      // [2] accumulator ready for the epilogue
    uint64_t* acc_empty = acc_full + 2;        // [2] accumulator drained by both blocks (the leader's counts)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* give_up = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)block_in_pair(), pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_k = (a.k + BK - 1) / BK;
    const int n_groups = a.n_experts + (a.n_rows > 0 && MODE != kPartial ? 1 : 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full + i, 1);
            mbar_init(acc_empty + i, 2 * kEpilogueWarps);
        }
        *give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {   // the same warp of both blocks allocates both accumulators' columns
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    // how many tiles the groups have, summed: warp 0, a group a lane and turn
    if (warp == 0) {
        int sum = 0;
        for (int base = 0; base <= n_groups; base += 32) {
            const int e = base + lane;
            int n = 0;
            if (e < n_groups) {
                const bool shared = e >= a.n_experts;
                const int row0 = shared ? 0 : a.offsets[e], rows = shared ? a.n_rows : a.offsets[e + 1] - row0;
                const int features = shared ? a.shared_features : a.n_features;
                n = (rows + kTileRows - 1) / kTileRows * ((features + kTileFeatures - 1) / kTileFeatures);
            }
            int upto = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += x;
            }
            if (e <= n_groups) first_tile[e] = sum + upto - n;
            sum += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_barrier();                            // both blocks' barriers stand
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const int n_tiles = first_tile[n_groups];

    // Neighbouring tiles share their weight rows: the tiles of rows run fastest.
    auto tile_of = [&](int i) {
        int lo = 0, hi = n_groups - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first_tile[mid] <= i) lo = mid; else hi = mid - 1;
        }
        Tile t;
        t.group = lo;
        t.shared = lo >= a.n_experts;
        const int row0 = t.shared ? 0 : a.offsets[lo], rows = t.shared ? a.n_rows : a.offsets[lo + 1] - row0;
        const int cuts = (rows + kTileRows - 1) / kTileRows, j = i - first_tile[lo];
        const int size = ((rows + cuts - 1) / cuts + 31) / 32 * 32;        // equal tiles, of whole columns
        const int cut = j % cuts;
        t.row0 = row0 + cut * size;
        t.here = max(0, min(size, rows - cut * size));
        t.columns = max(32, (t.here + 31) / 32 * 32);
        t.feature = j / cuts * kTileFeatures;
        return t;
    };

    if (warp == 0 && lane == 0) {
        // ---- TMA producer
        int it = 0;
        for (int i = pair; i < n_tiles && !*give_up; i += n_pairs) {
            const Tile t = tile_of(i);
            const CUtensorMap* rows = t.shared || MODE == kCombine ? &map_x : &map_sorted;
            const int b_row = t.row0 + rank * (t.columns / 2);
            int a0, a1, k0 = 0;                // the block's weight rows, 64 and 64
            if (MODE == kGlu) {
                a0 = t.group * a.n_features + t.feature + rank * 64;
                a1 = a0 + a.up_row;
            } else {
                a0 = (MODE == kGelu ? t.group * a.n_features : 0) + t.feature + rank * 128;
                a1 = a0 + 64;
                if (MODE == kPartial) k0 = t.group * a.k;
                if (MODE == kCombine) k0 = a.up_row;        // (where the shared expert's columns begin)
            }
            for (int kb = 0; kb < n_k && !a.skip_loads; ++kb, ++it) {
                const int s = it % kStages;
                if (!mbar_wait(empty + s, ((it / kStages) & 1) ^ 1)) {
                    if (a.err) atomicOr(a.err, THN_ERR_WAIT_TIMEOUT);
                    *give_up = 1;
                    break;
                }
                unsigned char* dst = tiles + (size_t)s * kStageBytes;
                const uint32_t bar = leader_addr(full + s);
                if (rank == 0) mbar_expect_tx(full + s, 2 * kLoaded);
                load_tile(dst, &map_w, bar, k0 + kb * BK, a0);
                load_tile(dst + kABytes / 2, &map_w, bar, k0 + kb * BK, a1);
                load_tile(dst + kABytes, rows, bar, kb * BK, b_row);
            }
        }
    } else if (warp == 1 && lane == 0 && rank == 0) {
        // ---- the leading block issues the pair's products
        int it = 0, local = 0;
        for (int i = pair; i < n_tiles && !*give_up; i += n_pairs, ++local) {
            const Tile t = tile_of(i);
            const uint32_t instr = instruction(t.columns);
            const int buf = local & 1;
            bool ok = mbar_wait(acc_empty + buf, ((local >> 1) & 1) ^ 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + buf * kRows;
            for (int kb = 0; kb < n_k && ok; ++kb, ++it) {
                const int s = it % kStages;
                ok = mbar_wait(full + s, (it / kStages) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = smem_addr(tiles + (size_t)s * kStageBytes);
                const uint64_t a_desc = smem_desc(at), b_desc = smem_desc(at + kABytes);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k)      // 32 bytes further along K: + 2 in the address field
                    pair_mma(tmem_d, a_desc + 2 * k, b_desc + 2 * k, instr, (kb | k) != 0);
                pair_commit(empty + s);                    // the stage is free in both blocks when these products are done
            }
            pair_commit(acc_full + buf);
            if (!ok) {
                if (a.err) atomicOr(a.err, THN_ERR_WAIT_TIMEOUT);
                *give_up = 1;
            }
        }
    } else if (warp >= 2) {
        // ---- epilogue: a warp reads tensor-memory lanes 32 * (warp % 4) .. + 31 (= features), its group every fourth chunk of
        // 32 columns (= rows)
        const int quarter = warp & 3, group = (warp - 2) >> 2;
        int local = 0;
        for (int i = pair; i < n_tiles; i += n_pairs, ++local) {
            const Tile t = tile_of(i);
            const int buf = local & 1;
            const int features = t.shared ? a.shared_features : a.n_features;
            const int feature = t.feature + (MODE == kGlu ? rank * 64 + (quarter & 1) * 32 : rank * 128 + quarter * 32) + lane;
            const bool there = feature < features;

            // kCombine: the rows' partial sums are on their way while the products run
            float sum[MODE == kCombine ? 32 : 1];
            if constexpr (MODE == kCombine) {
#pragma unroll
                for (int j = 0; j < 32; ++j) sum[j] = 0.f;
                const float* partial = a.partial + min(feature, features - 1);
                // (columns behind the last row read that row's sums)
                const int* places = a.place + (long long)(t.row0 + min(32 * group + lane, t.here - 1)) * a.top;
#pragma unroll 1
                for (int pick = 0; pick < a.top; ++pick) {
                    const int at = places[pick];
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = partial[(long long)__shfl_sync(0xffffffffu, at, j) * features];
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[j] += v[j];
                }
            }
            const bool ready = !*give_up && mbar_wait(acc_full + buf, (local >> 1) & 1);
            if (!all_of(ready, 1 + group, 128)) {      // the four warps that meet below go on, or stop, together
                if (lane == 0 && a.err) atomicOr(a.err, THN_ERR_WAIT_TIMEOUT);
                *give_up = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_base + buf * kRows + ((uint32_t)(quarter * 32) << 16);
            // calls put(j, value) for the chunk's columns j that are rows: the usual chunk has them all
            auto rows_of = [&](int first, auto n, auto put) {
                if (!there) return;
                if (first + n.value <= t.here) {
#pragma unroll
                    for (int j = 0; j < n.value; ++j) put(j);
                } else {
#pragma unroll
                    for (int j = 0; j < n.value; ++j)
                        if (first + j < t.here) put(j);
                }
            };
            // the weight of lane's row of the chunk's: what a row's activation is multiplied by
            auto weight_of = [&](int column) {
                const int pos = t.row0 + min(column, t.here - 1);
                if (!t.shared) return a.sorted_weight[pos];
                return a.shared_logit ? 1.0f / (1.0f + expf(-a.shared_logit[pos * a.logit_stride])) : 1.0f;
            };
            auto drain = [&](int c) {
                float v[32];
                if constexpr (MODE == kGlu) {
                    // warps of quarters 0, 1 hold gates, 2, 3 the ups of the same features: the first finish columns 0-15 of
                    // the chunk, the second 16-31, with what the others hold of them
                    const bool ups = quarter >= 2;
                    const int from = c + (ups ? 16 : 0);
                    const float weight = weight_of(from + (lane & 15));
                    tmem_load_32(taddr + c, v);
                    float* place = hand + group * 16 * 128 + lane;
                    float* mine = place + quarter * 32;
                    const float* theirs = place + (quarter ^ 2) * 32;
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");      // what was handed over before has been read
#pragma unroll
                    for (int j = 0; j < 16; ++j) mine[j * 128] = ups ? v[j] : v[16 + j];
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
                    const float lim = t.shared ? a.shared_limit : a.limit;
                    const bool scales_input = !t.shared && !a.weight_output;
                    float y[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float other = theirs[j * 128], w = __shfl_sync(0xffffffffu, weight, j);
                        const float before = scales_input ? w : 1.0f, after = scales_input ? 1.0f : w;
                        const float g = fminf(before * (ups ? other : v[j]), lim);
                        const float u = fminf(fmaxf(before * (ups ? v[16 + j] : other), -lim), lim);
                        // (The fast division is off by up to two units in the last place of float32, 2^-15 of the rounding to bfloat16 that follows; the
                        // layer's error against 64 bits is 2.3e-3 with either.  The exact one, whose slow path every lane may take, costs the layer 2 to 5 %: 16
                        // experts of 1,024 over 2,048, 512 rows 75 / 78 us, 8 of 2,048 over 4,096, 2,048 rows 318 / 333.)
                        y[j] = __fdividef(g, 1.0f + expf(-a.alpha * g)) * (u + a.up_shift) * after;
                        if (w == 0.f && !t.shared) y[j] = 0.f;
                    }
                    __nv_bfloat16* out = (t.shared ? a.shared_out : static_cast<__nv_bfloat16*>(a.out)) + (long long)(t.row0 + from) * features + feature;
                    rows_of(from, Number<16>{}, [&](int j) {
                        *out = __float2bfloat16_rn(y[j]);
                        out += features;
                    });
                } else if constexpr (MODE == kGelu) {
                    const float weight = weight_of(c + lane);
                    tmem_load_32(taddr + c, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float w = __shfl_sync(0xffffffffu, weight, j);
                        v[j] = 0.5f * v[j] * (1.0f + erff(v[j] * 0.70710678118654752f)) * w;
                        if (w == 0.f && !t.shared) v[j] = 0.f;
                    }
                    __nv_bfloat16* out = (t.shared ? a.shared_out : static_cast<__nv_bfloat16*>(a.out)) + (long long)(t.row0 + c) * features + feature;
                    rows_of(c, Number<32>{}, [&](int j) {
                        *out = __float2bfloat16_rn(v[j]);
                        out += features;
                    });
                } else if constexpr (MODE == kPartial) {
                    tmem_load_32(taddr + c, v);
                    float* out = static_cast<float*>(a.out) + (long long)(t.row0 + c) * features + feature;
                    rows_of(c, Number<32>{}, [&](int j) {
                        *out = v[j];
                        out += features;
                    });
                } else {
                    tmem_load_32(taddr + c, v);
                    __nv_bfloat16* out = a.shared_out + (long long)(t.row0 + c) * features + feature;
                    rows_of(c, Number<32>{}, [&](int j) {
                        *out = __float2bfloat16_rn(v[j] + sum[j]);
                        out += features;
                    });
                }
            };
#pragma unroll 1
            for (int c = 32 * group; c < t.columns; c += 32 * kEpilogueGroups) drain(c);
            // this warp has read its share of the accumulator: the leader may fill it again
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr(acc_empty + buf)) : "memory");
        }
    }
    if (*give_up) let_copies_land();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_barrier();                            // neither block leaves while the other may reach into it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

constexpr int kSortThreads = 1024;

// Block e: where expert e's pairs begin (all pairs of the experts ahead of it), and its pairs in the order of the rows.
// A choice that a row has made before (only where logits are no numbers) weighs nothing the second time.
__global__ void __launch_bounds__(kSortThreads) moe_sort_kernel(int* __restrict__ offsets, int* __restrict__ sorted_row,
                                                                float* __restrict__ sorted_weight, int* __restrict__ place,
                                                                const int* __restrict__ chosen, const float* __restrict__ dense,
                                                                int n, int top, int n_experts) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ int counts[kSortThreads / 32], ahead[kSortThreads / 32];
    const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // a thread counts a run of neighbouring pairs, eight loads at a time
    const int per = (n + kSortThreads - 1) / kSortThreads, i0 = min(n, (int)threadIdx.x * per), i1 = min(n, i0 + per);
    auto eight = [&](int i, int (&c)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = i + j < i1 ? chosen[i + j] : n_experts;
    };
    int own = 0, less = 0;
    for (int i = i0; i < i1; i += 8) {
        int c[8];
        eight(i, c);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            own += c[j] == e;
            less += c[j] < e;
        }
    }
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
        less += __shfl_xor_sync(0xffffffffu, less, o);
    }
    if (lane == 31) counts[warp] = upto;
    if (lane == 0) ahead[warp] = less;
    __syncthreads();
    int at = upto - own, all = 0;
    for (int w = 0; w < kSortThreads / 32; ++w) {
        at += ahead[w] + (w < warp ? counts[w] : 0);
        all += ahead[w] + counts[w];
    }
    if (threadIdx.x == 0) {
        if (e == 0) offsets[0] = 0;
        offsets[e + 1] = all;
    }
    for (int i = i0; own > 0 && i < i1; i += 8) {
        int c[8];
        eight(i, c);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (c[j] != e) continue;
            const int row = (i + j) / top;
            float w = dense[(long long)row * n_experts + e];
            for (int k = row * top; k < i + j; ++k)
                if (chosen[k] == e) w = 0.f;
            sorted_row[at] = row;
            sorted_weight[at] = w;
            place[i + j] = at;
            ++at;
        }
    }
}

// 16 bytes a thread and turn: rows of x in the sorted order.
__global__ void __launch_bounds__(256) moe_gather_kernel(uint4* __restrict__ out, const uint4* __restrict__ x,
                                                         const int* __restrict__ sorted_row, int n, int pieces) {
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = blockIdx.x * 8 + warp;
    if (pos >= n) return;
    const uint4* src = x + (long long)sorted_row[pos] * pieces;
    uint4* dst = out + (long long)pos * pieces;
    int c = lane;
    for (; c + 224 < pieces; c += 256) {
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = src[c + 32 * j];
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[c + 32 * j] = v[j];
    }
    for (; c < pieces; c += 32) dst[c] = src[c];
}

// out [rows, size] = the sum of the rows' partial sums, in the order of the choices; four entries a thread.
__global__ void __launch_bounds__(256) moe_combine_kernel(__nv_bfloat16* __restrict__ out, const float* __restrict__ partial,
                                                          const int* __restrict__ place, int size, int top) {
    pdl_launch_dependents();
    pdl_wait();
    const int c = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (c >= size) return;
    const long long row = blockIdx.x;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int pick = 0; pick < top; ++pick) {
        const float4 v = *reinterpret_cast<const float4*>(partial + (long long)place[row * top + pick] * size + c);
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(sum.x, sum.y), hi = __floats2bfloat162_rn(sum.z, sum.w);
    *reinterpret_cast<uint2*>(out + row * size + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiled)p;
    }();
    return fn;
}

// A row-major [rows, width] bfloat16 matrix as a 2-D tensor map with boxes of 64 entries x box_rows.
bool make_map(CUtensorMap* map, const void* base, long long rows, int width, int box_rows) {
    const EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)width * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// most_tiles: no fewer than the launch can have
template <int MODE>
int launch_pairs(const CUtensorMap& w, const CUtensorMap& sorted, const CUtensorMap& x, const PairArgs& args, long long most_tiles,
                 cudaStream_t stream) {
    auto kernel = pair_gemm_kernel<MODE>;
    static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (configured != cudaSuccess) {
        thn_set_error("moe_grouped: cannot reserve %zu bytes of shared memory: %s", kSmemBytes, cudaGetErrorString(configured));
        return (int)configured;
    }
    int device = 0, n_sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, device);
    const long long pairs = most_tiles < n_sms / 2 ? most_tiles : n_sms / 2;
    thn_launch(kernel, dim3((unsigned)(2 * (pairs > 0 ? pairs : 1))), kThreads, kSmemBytes, stream, w, sorted, x, args);
    return thn_launch_status("moe_grouped");
}

// no fewer than the tiles of `rows` rows in all, in `groups` groups
long long tiles_of(long long rows, int groups, int features, int tile, int mode) {
    return (rows / tile_rows(mode) + groups) * ((features + tile - 1) / tile);
}

}  // namespace

// 1 if the grouped products take a mixture of these sizes.
THN_API int thn_moe_grouped_supported(int hidden, int n_experts, int ff, int shared_ff) {
    return hidden >= 64 && hidden % 64 == 0 && n_experts >= 1 && n_experts <= kMaxGroups && ff >= 64 && ff % 64 == 0 && shared_ff >= 0 &&
           shared_ff % 64 == 0;
}

// out bfloat16 [rows, hidden]: the weighted sum of the chosen experts' outputs and the shared expert's.
//   x            bfloat16 [rows, hidden]
//   chosen       int32 [rows, top], dense float32 [rows, experts]: thn_moe_route's
//   glu != 0     w_up [2 * (experts * ff + shared_ff), hidden]: the gates of all columns, then the ups; the activation of
//                thn_routed_clamped_glu (limit ... weight_output).  glu == 0: w_up [experts * ff + shared_ff, hidden], gelu.
//   w_down       [hidden, experts * ff + shared_ff]
//   shared_logit the rows' gate logits of the shared expert, logit_stride apart (null: no gate)
//   sorted_x, act, shared_act bfloat16 [rows * top, hidden], [rows * top, ff], [rows, shared_ff]; partial float32
//                [rows * top, hidden]; ints int32 [2 * rows * top + experts + 1]; floats float32 [rows * top]: scratch
// All matrices 16-byte aligned.  err: device error word (THN_ERR_WAIT_TIMEOUT if a pipeline wait gave up).  skip_loads: 0; otherwise no
// operand is loaded, so that the products' waits run out (for the test of the waits only).
THN_API int thn_moe_grouped_bf16(void* out, const void* x, const int* chosen, const float* dense, const void* w_up, const void* w_down,
                                 const float* shared_logit, long long logit_stride, void* sorted_x, void* act, void* shared_act,
                                 float* partial, int* ints, float* floats, int n_rows, int hidden, int n_experts, int top, int ff,
                                 int shared_ff, int glu, float limit, float shared_limit, float alpha, float up_shift, int weight_output,
                                 int skip_loads, int* err, cudaStream_t stream) {
    THN_UNSUPPORTED_IF(!thn_moe_grouped_supported(hidden, n_experts, ff, shared_ff), "moe_grouped: %d experts of %d (and %d) over rows of %d not supported",
                       n_experts, ff, shared_ff, hidden);
    THN_CHECK_ARG(n_rows >= 0 && top > 0 && top <= n_experts, "moe_grouped: %d rows, top %d of %d experts", n_rows, top, n_experts);
    THN_CHECK_ARG((((uintptr_t)out | (uintptr_t)x | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)sorted_x | (uintptr_t)act |
                    (uintptr_t)shared_act | (uintptr_t)partial) & 15) == 0, "moe_grouped: operands must be 16-byte aligned");
    THN_CHECK_ARG(!glu || (limit > 0.f && (shared_ff == 0 || shared_limit > 0.f)), "moe_grouped: limits must be positive");
    THN_UNSUPPORTED_IF((long long)n_rows * top > (1 << 30), "moe_grouped: %d rows", n_rows);
    if (n_rows == 0) return THN_OK;
    const int n = n_rows * top, width = n_experts * ff + shared_ff;
    int* offsets = ints;
    int* sorted_row = ints + n_experts + 1;
    int* place = sorted_row + n;
    thn_launch(moe_sort_kernel, n_experts, kSortThreads, 0, stream, offsets, sorted_row, floats, place, chosen, dense, n, top, n_experts);
    thn_launch(moe_gather_kernel, (n + 7) / 8, 256, 0, stream, (uint4*)sorted_x, (const uint4*)x, sorted_row, n, hidden / 8);
    // (a launch's maps are made just ahead of it: the host works while the device sorts, gathers and multiplies)
    auto no_map = [&] {
        thn_set_error("moe_grouped: cuTensorMapEncodeTiled failed for %d rows of %d, %d experts of %d", n_rows, hidden, n_experts, ff);
        return THN_BAD_ARGUMENT;
    };
    CUtensorMap map_up, map_down, map_sorted, map_x, map_act, map_shared;
    if (!make_map(&map_up, w_up, (glu ? 2LL : 1LL) * width, hidden, 64) || !make_map(&map_sorted, sorted_x, n, hidden, kRows / 2) ||
        !make_map(&map_x, x, n_rows, hidden, kRows / 2))
        return no_map();
    PairArgs up = {};
    up.n_experts = n_experts;
    up.offsets = offsets;
    up.sorted_row = sorted_row;
    up.sorted_weight = floats;
    up.n_rows = shared_ff ? n_rows : 0;
    up.n_features = ff;
    up.shared_features = shared_ff;
    up.up_row = width;
    up.k = hidden;
    up.out = act;
    up.shared_out = (__nv_bfloat16*)shared_act;
    up.limit = limit;
    up.shared_limit = shared_limit;
    up.alpha = alpha;
    up.up_shift = up_shift;
    up.weight_output = weight_output;
    up.shared_logit = shared_logit;
    up.logit_stride = logit_stride;
    up.err = err;
    up.skip_loads = skip_loads;
    const int up_tile = glu ? kFeatures / 2 : kFeatures;
    const long long up_tiles = tiles_of(n, n_experts, ff, up_tile, kGlu) + (shared_ff ? tiles_of(n_rows, 1, shared_ff, up_tile, kGlu) : 0);
    int status = glu ? launch_pairs<kGlu>(map_up, map_sorted, map_x, up, up_tiles, stream)
                     : launch_pairs<kGelu>(map_up, map_sorted, map_x, up, up_tiles, stream);
    if (status != THN_OK) return status;
    if (!make_map(&map_down, w_down, hidden, width, 64) || !make_map(&map_act, act, n, ff, kRows / 2)) return no_map();
    PairArgs down = {};
    down.n_experts = n_experts;
    down.offsets = offsets;
    down.n_features = hidden;
    down.k = ff;
    down.out = partial;
    down.err = err;
    down.skip_loads = skip_loads;
    status = launch_pairs<kPartial>(map_down, map_act, map_act, down, tiles_of(n, n_experts, hidden, kFeatures, kPartial), stream);
    if (status != THN_OK) return status;
    if (shared_ff == 0) {
        thn_launch(moe_combine_kernel, dim3(n_rows, (hidden / 4 + 255) / 256), 256, 0, stream, (__nv_bfloat16*)out, partial, place, hidden, top);
        return thn_launch_status("moe_combine");
    }
    if (!make_map(&map_shared, shared_act, n_rows, shared_ff, tile_rows(kCombine) / 2)) return no_map();
    PairArgs sum = {};
    sum.n_rows = n_rows;
    sum.n_features = sum.shared_features = hidden;
    sum.up_row = n_experts * ff;
    sum.k = shared_ff;
    sum.shared_out = (__nv_bfloat16*)out;
    sum.partial = partial;
    sum.place = place;
    sum.top = top;
    sum.err = err;
    sum.skip_loads = skip_loads;
    return launch_pairs<kCombine>(map_down, map_shared, map_shared, sum, tiles_of(n_rows, 1, hidden, kFeatures, kCombine), stream);
}
