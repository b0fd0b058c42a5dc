// C[M, N] = A[M, K] @ W[N, K]^T in true float32 on the CUDA cores (FFMA only: no
// tensor cores, no TF32).  It is the matrix product of the 32-bit path, where the
// reference calls a library product with TF32 disabled (engine/engine.py:113-114,
// :341-350).  Every output element accumulates k = 0, 1, 2, ... in one accumulator, so a
// row's result does not depend on how many other rows the call has.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

__global__ void __launch_bounds__(256) gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A,
                                                       const float* __restrict__ W, int M, int N, int K) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 x 16 elements per operand, 256 threads: 4 each; consecutive threads walk k.
        for (int e = tid; e < BM * BK; e += 256) {
            const int r = e / BK, c = e % BK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
            As[c][r] = (gm < M && gk < K) ? A[(size_t)gm * K + gk] : 0.f;
            Ws[c][r] = (gn < N && gk < K) ? W[(size_t)gn * K + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn < N) C[(size_t)gm * N + gn] = acc[i][j];
        }
    }
}
}  // namespace

THN_API int thn_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    THN_CHECK_ARG(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return THN_OK;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    THN_UNSUPPORTED_IF(grid.y > 65535, "gemm_f32: %d rows exceed the grid limit", M);
    thn_launch(gemm_f32_kernel, grid, 256, 0, stream, C, A, W, M, N, K);
    return thn_launch_status("gemm_f32");
}

// ------------------------------------------------------------------ a few outputs per row, float32 out
//
// C[M, N] float32 = A[M, K] bfloat16 @ W[N, K]^T bfloat16 for a weight of few rows (a router, a
// gate of one number per token): the products that vendor libraries serve worst, since N is
// neither large nor a multiple of eight.  A block takes 16 rows and 8 TILES columns; its sixteen warps deal out
// K in steps of 32 on the tensor cores, each product of 16 into a fresh accumulator (the tensor core's accumulation
// rounds towards zero; the sum over the products is float32 additions, over the warps double ones).  A sum that float32
// holds exactly comes out exactly.  A lane loads its operands straight from memory, 16 bytes of a row at k = 32 s + 8 t: which
// k a lane's pair stands for does not matter as long as both operands agree; the loads of four or eight steps are
// issued together.  The warps' sums meet in shared memory in a fixed order, so a row's result depends on nothing but K,
// whatever M, N and TILES are.  K is a multiple of eight and both operands are 16-byte aligned.
// B200, against a warp's float32 multiply-adds over four rows and four columns at a time, which it took the place of: 2,251
// rows, 32 columns over 2,048 5.8 us / 27.4, 4,096 rows, 64 columns over 4,096 30 / 143; few rows the same with the weight
// in HBM (8 rows, 32 columns over 4,096: 8.2 / 10.2), 0.1 to 1.1 us more back to back with everything in L2 (2.2 / 1.8 for 8
// rows, 32 columns over 2,048; the number of rows may not choose the kernel, since a row's bits would follow it).  Error against 64 bits,
// 2-norms: 5.8e-8 to 7.3e-8 / 7.9e-8 to 9.2e-8 over 2,048 and 4,096 normal entries, 2.8e-8 / 4.8e-8 where all are positive,
// 7.3e-8 / 9.1e-8 where they spread over forty powers of two.  (Scaling the result up by the
// accumulation's mean loss, 4.3e-8, changes sums that were exact.)
namespace {
constexpr int kSkinnyThreads = 512;

__device__ __forceinline__ void skinny_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int TILES>
__global__ void __launch_bounds__(kSkinnyThreads) linear_skinny_kernel(float* __restrict__ C,
                                                                       const __nv_bfloat16* __restrict__ A,
                                                                       const __nv_bfloat16* __restrict__ W, int M, int N,
                                                                       int vecs) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kWarps = kSkinnyThreads / 32, kBatch = TILES == 1 ? 8 : 4;
    __shared__ __align__(16) float part[kWarps][TILES][32][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.x * 16, n0 = blockIdx.y * 8 * TILES;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    // (rows and columns beyond the last repeat it; their results are not stored)
    const uint4* a_lo = reinterpret_cast<const uint4*>(A) + (size_t)min(m0 + g, M - 1) * vecs;
    const uint4* a_hi = reinterpret_cast<const uint4*>(A) + (size_t)min(m0 + g + 8, M - 1) * vecs;
    const uint4* w[TILES];
#pragma unroll
    for (int n = 0; n < TILES; ++n) w[n] = reinterpret_cast<const uint4*>(W) + (size_t)min(n0 + 8 * n + g, N - 1) * vecs;
    float acc[TILES][4];
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
    const int steps = (vecs + 3) / 4;
    for (int s0 = warp; s0 < steps; s0 += kBatch * kWarps) {
        uint4 x[kBatch], y[kBatch], z[kBatch][TILES];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (s0 + u * kWarps >= steps) continue;
            const int v = 4 * (s0 + u * kWarps) + t, at = min(v, vecs - 1);      // this lane's 16 bytes of a row
            x[u] = a_lo[at];
            y[u] = a_hi[at];
#pragma unroll
            for (int n = 0; n < TILES; ++n) z[u][n] = v < vecs ? __ldg(w[n] + at) : zero;
            if (v >= vecs) x[u] = y[u] = zero;
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (s0 + u * kWarps >= steps) continue;
#pragma unroll
            for (int n = 0; n < TILES; ++n) {
                float one[4] = {0.f, 0.f, 0.f, 0.f}, two[4] = {0.f, 0.f, 0.f, 0.f};
                skinny_mma(one, x[u].x, y[u].x, x[u].y, y[u].y, z[u][n].x, z[u][n].y);
                skinny_mma(two, x[u].z, y[u].z, x[u].w, y[u].w, z[u][n].z, z[u][n].w);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n][i] += one[i] + two[i];
            }
        }
    }
#pragma unroll
    for (int n = 0; n < TILES; ++n) *reinterpret_cast<float4*>(part[warp][n][lane]) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
    __syncthreads();
    for (int e = threadIdx.x; e < TILES * 128; e += kSkinnyThreads) {
        const int n = e >> 7, l = e >> 2 & 31, i = e & 3;
        double sum[4] = {0.0, 0.0, 0.0, 0.0};            // (four short chains)
#pragma unroll
        for (int k = 0; k < kWarps; ++k) sum[k & 3] += (double)part[k][n][l][i];
        const double total = (sum[0] + sum[1]) + (sum[2] + sum[3]);
        const int row = m0 + (l >> 2) + 8 * (i >> 1), col = n0 + 8 * n + 2 * (l & 3) + (i & 1);
        if (row < M && col < N) C[(size_t)row * N + col] = (float)total;
    }
}
}  // namespace

THN_API int thn_linear_skinny_supported(int N, int K) { return N >= 1 && N <= 64 && K >= 8 && K % 8 == 0; }

THN_API int thn_linear_skinny_bf16(float* C, const void* A, const void* W, int M, int N, int K, cudaStream_t stream) {
    THN_CHECK_ARG(M >= 0 && thn_linear_skinny_supported(N, K), "linear_skinny: bad sizes M=%d N=%d K=%d", M, N, K);
    THN_CHECK_ARG((((uintptr_t)A | (uintptr_t)W) & 15) == 0, "linear_skinny: operands must be 16-byte aligned (M=%d)", M);
    if (M == 0) return THN_OK;
    // two tiles of columns a block read A half as often; one tile a block where that leaves multiprocessors idle
    const int row_blocks = (M + 15) / 16, tiles = (N + 7) / 8;
    if (row_blocks * ((tiles + 1) / 2) >= 120)
        thn_launch(linear_skinny_kernel<2>, dim3(row_blocks, (tiles + 1) / 2), kSkinnyThreads, 0, stream, C, (const __nv_bfloat16*)A,
                   (const __nv_bfloat16*)W, M, N, K / 8);
    else
        thn_launch(linear_skinny_kernel<1>, dim3(row_blocks, tiles), kSkinnyThreads, 0, stream, C, (const __nv_bfloat16*)A,
                   (const __nv_bfloat16*)W, M, N, K / 8);
    return thn_launch_status("linear_skinny");
}
