// The two GEMM rows that have no tcgen05 kind: fp32 on the CUDA cores (small products and sums of less than 64 numbers;
// the others are gemm_f32_kernel's) and fp64 on the warp-level DMMA path.  They take the place of the reference's cuBLASLt "fp32" and
// "fp64" rows (src/cuda/cuda_blas.cpp:567-581) behind the same clpk_gemm entry point:
// C[M][N] = alpha * A[M][K] * B[N][K]^T, both operands K-contiguous, C row-major in the
// operand type.
//
// fp32 (sgemm_kernel).  128 x 128 x 16 tile per CTA of 128 threads = 4 warps in a 2 x 2
// grid, two CTAs per SM, 8 rows x 16 columns of outputs per thread.  The multiply is
// sm_100's packed fma.rn.f32x2 (two FMAs per issued instruction) on accumulator pairs of
// neighbouring columns, the row value duplicated into a fresh register pair just before
// its eight FMAs.  Which shape the packed FMA likes was measured from registers alone: 8
// rows x 8 pairs with that duplication runs at 71 of 74 TFLOPS with 8 warps per SM, 16
// rows x 4 pairs at 51, pairs over two neighbouring k (no duplication at all) at 52 --
// the operand pairs collide in the register banks.  Operands are transposed into shared
// memory ([k][row]) so that both fragments are 128-bit loads: global -> staging buffer by
// asynchronous 16-byte copies two k blocks ahead, staging -> registers -> tile by the
// thread that copied them, one barrier per k block.  Fragment loads are laid out for two
// passes of the shared-memory data pipe per 128-bit load (see the kernel).  Bound: the
// fp32 pipe, 128 FMA / clock / SM (B200: 148 SMs x 128 x 2 x 1.965 GHz = 74.4 TFLOPS).
// Measured 62.6 TFLOPS at 8192^3 (0.84 of the pipe, 0.95 of cuBLAS) and 60.8 at 4096^3
// (1.07 of cuBLAS: 1024 tiles are 3.5 waves of 296 CTAs, and a CTA alone on its SM runs
// twice as fast).  The same loop runs at 68.4 without the transposition, 65.2 without the
// fragment loads and 69.6 with neither; moving the transposition under the multiplies
// (with or without a branch) and 128-bit tile stores changed nothing; leaving A as it lies
// in memory (fragments of four k per row, only B transposed) ran at 53.5.  Earlier shapes:
// 256 threads x (8 x 8) with the next k block held in registers across the multiply,
// 54.0 (the warps stood at the tile stores waiting for the global loads); the same through
// the staging buffer, 58.9.
//
// fp64 (dgemm_kernel).  64 x 64 x 16 tile per CTA of 128 threads = 4 warps in a 2 x 2 grid, four CTAs per SM, 32 x 32
// outputs per warp = 4 x 4 m8n8k4 accumulator tiles, multiplied two at a time (m16n8k4).  Operands go global -> shared with
// cp.async (16 bytes), three stages; a row's chunks are permuted so that the fragment reads (lane -> row lane/4, k lane%4)
// fall in 16 distinct 8-byte banks per half warp.  Bound: the DMMA pipe, 64 fp64 FMA / clock / SM, the same rate as the scalar
// DFMA pipe (37.2 TFLOPS at 1.965 GHz).  Measured 34.6 TFLOPS at 4096^3 and 8192 x 8192 x 512, 32.9 at 2048 x 2048 x 512, where
// 1024 tiles are 6.9 per SM.  Before, 128 x 64 tiles of four 64 x 32 warps, two CTAs per SM, rows padded to 20 doubles, took
// 4027 us at 4096^3 (3968 now), 2066 at 8192 x 8192 x 512 (1987), 136 at 10770 x 310 x 410 (97): with half the CTAs per SM a
// partial round keeps fewer of them busy.  64 x 64 tiles whose result goes through shared memory, in blocks of eight k: 2048 x 2048 x 512
// 144 us (131 now), 5001 x 5001 x 4 78 (59).  Tried: two warps of 64 x 32 per CTA 155, m16n8k8 and m16n8k16 as m16n8k4 and 4 %
// slower, 128 x 64 tiles with this layout and four stages 3962 at 4096^3, a last row loaded again in place of the zeros beyond an
// operand (65 x 10179 x 180 25 -> 33 us), fragments loaded a step ahead (within 1 %).
//
// Shapes of which those tiles make too few CTAs take 64 x 64 (fp32, fp64) or 32 x 32 (fp64) tiles with K split over the
// CTAs of a cluster and over groups of warps inside a CTA (sgemm64_kernel, dgemm_split_kernel; plan_simt has the rule).
// Device time before -> after: fp32 64 x 64 x 16384 1545 -> 57 us, 459 x 349 x 4636 474 -> 69; fp64
// 64 x 64 x 16384 1388 -> 26, 863 x 251 x 2456 228 -> 42.
//
// All take any M, N > 0 and any K that keeps operand rows 16-byte aligned (a multiple of 4
// floats, 2 doubles): a second instantiation of the large kernels, and the others always, zero-fill the chunks a tile
// reaches beyond A or B (cp.async with a source size of 0) and skip the stores beyond C;
// whole tiles and k blocks take the instantiation without the checks.
//
// CTAs walk C in groups of 16 tile rows so that the operand panels a wave of CTAs needs
// stay in L2.  Work 2*M*N*K flop; minimum HBM bytes (M*K + N*K + M*N) * element.
#include <algorithm>

#include "../clpk_internal.h"
#include "../clpk_ptx.cuh"

namespace clpk {

constexpr int kSimtTile = 128;
constexpr int kSimtBK = 16;
constexpr int kRasterGroup = 16;
constexpr int kSimtSmemMax = 227 * 1024;                // the most dynamic shared memory that a CTA may ask for

// tile -> (tile row, tile column), column-major inside groups of kRasterGroup tile rows
__device__ __forceinline__ void raster(uint32_t tile, uint32_t tiles_m, uint32_t tiles_n, uint32_t *tm, uint32_t *tn)
{
    const uint32_t per_group = kRasterGroup * tiles_n;
    const uint32_t g = tile / per_group, r = tile % per_group;
    const uint32_t rows = min((uint32_t)kRasterGroup, tiles_m - g * kRasterGroup);
    *tm = g * kRasterGroup + r % rows;
    *tn = r / rows;
}

// The launches carry the programmatic-serialisation attribute: a CTA may start under the tail of the kernel before it
// in the stream and waits here until that has completed.  The status word is cleared by the kernel, so that nothing
// sits between two launches.  No operand is `const __restrict__`: the kernel before may still be writing it when this
// one starts, and the read-only path that the qualifier allows wants data that does not change while the kernel runs.
__device__ __forceinline__ void join_stream(uint32_t *status)
{
    griddep_wait();
    griddep_launch_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *status = 0u;
}

// ---- K split over the CTAs of a cluster -----------------------------------------------------------------------------
//
// Each of the S CTAs leaves its partial tiles in its own shared memory ([parts][rows][cols], parts = K groups inside the
// CTA) and sums a share of the rows over all of them, in rank order: the same bits whatever the timing.

template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };
__device__ __forceinline__ void add_to(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void add_to(double2 &a, const double2 &b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, float4)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double2 ld_cluster(uint32_t addr, double2)
{
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}

// `part`: this CTA's partial tiles, just written; called by all threads.
template <typename T, int ROWS, int COLS, int PARTS, int THREADS>
__device__ __forceinline__ void sum_partial_tiles(const T *part, uint32_t S, uint32_t rank, T *C, uint32_t row0, uint32_t col0, uint32_t M,
                                                  uint32_t N, T alpha)
{
    using V = typename Vec16<T>::type;
    constexpr uint32_t per = 16 / sizeof(T), row_vecs = COLS / per, vecs = ROWS * row_vecs;
    cluster_sync();
    const uint32_t local = smem_u32(part);
    for (uint32_t i = rank * vecs / S + threadIdx.x; i < (rank + 1) * vecs / S; i += THREADS) {
        V sum;
        for (uint32_t src = 0; src < S; src++) {
            uint32_t addr;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local + i * 16), "r"(src));
#pragma unroll
            for (int q = 0; q < PARTS; q++) {
                const V v = ld_cluster(addr + q * (ROWS * COLS * (uint32_t)sizeof(T)), V{});
                if (src == 0 && q == 0)
                    sum = v;
                else
                    add_to(sum, v);
            }
        }
        const uint32_t row = row0 + i / row_vecs, col = col0 + i % row_vecs * per;
        if (row < M) {
            const T *e = reinterpret_cast<const T *>(&sum);
            T *dst = C + (size_t)row * N + col;
#pragma unroll
            for (uint32_t t = 0; t < per; t++)
                if (col + t < N)
                    dst[t] = alpha * e[t];
        }
    }
    cluster_sync();                     // nobody leaves while its shared memory is being read
}

// ---------------------------------------------------------------------------------------------
// fp32
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ unsigned long long pack2(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ float2 unpack2(unsigned long long v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// d = a * b + d on two packed fp32 lanes, each rounded to nearest even like fmaf
__device__ __forceinline__ void ffma2(unsigned long long &d, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

constexpr int kSgemmLd = kSimtTile + 4;               // floats per k row of a shared tile
constexpr int kSgemmThreads = 128;
constexpr int kSgemmChunks = 2 * kSimtTile * kSimtBK / 4 / kSgemmThreads;      // 16-byte chunks per thread and k block
constexpr size_t kSgemmTileFloats = (size_t)kSimtBK * kSgemmLd;                // one operand, one buffer: [k][row]
constexpr size_t kSgemmStagingFloats = kSgemmChunks * 4 * (size_t)kSgemmThreads;
constexpr size_t kSgemmSmemBytes = (4 * kSgemmTileFloats + 2 * kSgemmStagingFloats) * sizeof(float);

__device__ __forceinline__ void cp_async_16(void *dst_shared, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_shared)), "l"(src) : "memory");
}

// the same copy, or 16 bytes of zeros when the chunk lies outside the operand (nothing is read then)
__device__ __forceinline__ void cp_async_16_or_zeros(void *dst_shared, const void *src, bool inside)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_shared)), "l"(src),
                 "r"(inside ? 16u : 0u)
                 : "memory");
}

// RAGGED: M, N need not be multiples of the tile nor K of the k block (K a multiple of 4, so that rows stay 16-byte
// aligned): chunks outside the operands arrive as zeros, stores outside C are skipped.
template <bool RAGGED>
__global__ void __launch_bounds__(kSgemmThreads, 2)
sgemm_kernel(const float *A, const float *B, float *C, uint32_t M, uint32_t N,
             uint32_t K, float alpha, uint32_t *status)
{
    extern __shared__ __align__(16) float ssm[];
    float *const tiles = ssm;                                   // [buffer][A, B][k][kSgemmLd]
    float *const staging = ssm + 4 * kSgemmTileFloats;          // [buffer][chunk][thread] of float4
    uint32_t tm, tn;
    raster(blockIdx.x, (M + kSimtTile - 1) / kSimtTile, (N + kSimtTile - 1) / kSimtTile, &tm, &tn);
    join_stream(status);
    // Four warps in a 2 x 2 grid, 64 x 64 outputs per warp, a warp 8 (rows) x 4 (columns) threads, 8 rows x 16
    // columns per thread as 4 x 4 blocks.  A 128-bit shared-memory load takes two passes of the data pipe per warp
    // when every group of four consecutive lanes asks for at most two different 16-byte words, and four passes
    // otherwise (measured with a one-warp probe: lane / 2, lane / 4 and lane % 2 cost two passes, lane % 4 and
    // lane % 8 four).  So lane bits 0 and 2 pick the column block and bits 1, 3, 4 the row block: inside a group of
    // four lanes both fragments have two distinct addresses.
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lx = (lane & 1) | ((lane >> 1) & 2), ly = ((lane >> 1) & 1) | ((lane >> 2) & 6);
    const int fa = (warp >> 1) * 64 + ly * 4, fb = (warp & 1) * 64 + lx * 4;

    // Operands travel global -> staging (asynchronous 16-byte copies, two k blocks ahead) -> registers -> tile
    // (transposed: [row][k] in memory, [k][row] in the tile).  Every thread moves the same chunks through both
    // hops -- rows lrow + 32 c of A and of B, floats lk .. lk + 3 of the k block -- so only its own copies have to
    // have landed before it transposes, and nothing read from global memory is held in registers across the
    // multiply (with the loads going straight to registers the warps stood at the tile stores waiting for them:
    // 53 against 64 TFLOPS for the same loop without the operand traffic).
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    const float *srcA = A + ((size_t)tm * kSimtTile + lrow) * K + lk, *srcB = B + ((size_t)tn * kSimtTile + lrow) * K + lk;
    auto fetch = [&](uint32_t kb) {                              // k block kb into staging buffer kb % 2
        float *st = staging + (kb & 1) * kSgemmStagingFloats + tid * 4;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (RAGGED) {
                const bool in_k = kb * kSimtBK + lk < K;
                const bool in_a = in_k && tm * kSimtTile + lrow + 32 * c < M, in_b = in_k && tn * kSimtTile + lrow + 32 * c < N;
                cp_async_16_or_zeros(st + c * 4 * kSgemmThreads, in_a ? srcA + (size_t)c * 32 * K + (size_t)kb * kSimtBK : A, in_a);
                cp_async_16_or_zeros(st + (4 + c) * 4 * kSgemmThreads, in_b ? srcB + (size_t)c * 32 * K + (size_t)kb * kSimtBK : B, in_b);
            } else {
                cp_async_16(st + c * 4 * kSgemmThreads, srcA + (size_t)c * 32 * K + (size_t)kb * kSimtBK);
                cp_async_16(st + (4 + c) * 4 * kSgemmThreads, srcB + (size_t)c * 32 * K + (size_t)kb * kSimtBK);
            }
        }
    };
    auto transpose = [&](uint32_t kb) {                          // staging buffer kb % 2 into tile buffer kb % 2
        const float *st = staging + (kb & 1) * kSgemmStagingFloats + tid * 4;
        float *sA = tiles + (kb & 1) * 2 * kSgemmTileFloats, *sB = sA + kSgemmTileFloats;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float4 v = *reinterpret_cast<const float4 *>(st + c * 4 * kSgemmThreads);
            // k rows 8..15 keep their columns with bit 3 flipped: a warp stores 8 consecutive rows for four k
            // (lk = 0, 4, 8, 12), and 8 k rows of 132 floats are a multiple of 32 banks apart
            float *dst = (c < 4 ? sA : sB) + lk * kSgemmLd + ((lrow + 32 * (c & 3)) ^ (lk & 8));
            dst[0] = v.x; dst[kSgemmLd] = v.y; dst[2 * kSgemmLd] = v.z; dst[3 * kSgemmLd] = v.w;
        }
    };

    // Accumulators as pairs of neighbouring columns: sm_100's packed fma.rn.f32x2 does two FMAs per issued
    // instruction with the rounding of two scalar FMAs.  8 rows x 8 pairs with the row value duplicated into a
    // fresh register pair just before its eight FMAs runs at 71 of 74 TFLOPS from registers alone with 8 warps per
    // SM; 16 rows x 4 pairs at 51 (register-bank conflicts between the operand pairs).
    unsigned long long acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++)
            acc[i][j] = 0ull;

    const uint32_t nk = (K + kSimtBK - 1) / kSimtBK;
    fetch(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (nk > 1)
        fetch(1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    transpose(0);
    __syncthreads();
    for (uint32_t kb = 0; kb < nk; kb++) {
        // staging buffer kb % 2 was emptied into the tile before the last barrier: refill it two k blocks ahead
        if (kb + 2 < nk)
            fetch(kb + 2);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *sA = tiles + (kb & 1) * 2 * kSgemmTileFloats, *sB = sA + kSgemmTileFloats;
#pragma unroll
        for (int k = 0; k < kSimtBK; k++) {
            const int ca = fa ^ (k & 8), cb = fb ^ (k & 8);
            float a[8];
            unsigned long long b[8];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float4 v = *reinterpret_cast<const float4 *>(sA + k * kSgemmLd + ca + 32 * q);
                a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
            }
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float4 v = *reinterpret_cast<const float4 *>(sB + k * kSgemmLd + cb + 16 * h);
                b[2 * h] = pack2(v.x, v.y);
                b[2 * h + 1] = pack2(v.z, v.w);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const unsigned long long aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    ffma2(acc[i][j], aa, b[j]);
            }
        }
        if (kb + 1 < nk) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");      // k block kb + 1 is in staging (kb + 2 may still fly)
            transpose(kb + 1);
            __syncthreads();
        }
    }

    float *gC = C + (size_t)tm * kSimtTile * N + (size_t)tn * kSimtTile;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = fa + 32 * (i >> 2) + (i & 3);
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const float2 lo = unpack2(acc[i][2 * h]), hi = unpack2(acc[i][2 * h + 1]);
            const float4 v = make_float4(alpha * lo.x, alpha * lo.y, alpha * hi.x, alpha * hi.y);
            if (!RAGGED) {
                *reinterpret_cast<float4 *>(gC + (size_t)r * N + fb + 16 * h) = v;
            } else if (tm * kSimtTile + r < M) {
                const uint32_t col = tn * kSimtTile + fb + 16 * h;
                float *dst = gC + (size_t)r * N + fb + 16 * h;
                if ((N & 3) == 0 && col < N) {
                    *reinterpret_cast<float4 *>(dst) = v;
                } else {
                    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (col + t < N)
                            dst[t] = e[t];
                }
            }
        }
    }
}

// The same product in 64 x 64 tiles for shapes of which 128 x 128 tiles make too few, K split over the CTAs of a cluster
// and over G groups of two warps inside a CTA.  A group takes every G-th k block of its CTA's range through staging
// and tile buffers of its own and meets only its own 64 threads.  64 x 32 outputs per warp, 8 x 8 per thread: four
// 128-bit fragment loads per 32 packed FMAs.  Two groups and three CTAs per SM, or four groups for a CTA that has its
// SM to itself and a long range: with one warp per scheduler the FMA pipe waits on every load (64 x 64 x 16384 in eight
// ranges 68 -> 56 us, 719 x 368 x 6380 116 -> 87).
constexpr int kSgemm64 = 64;
constexpr int kSgemm64Ld = kSgemm64 + 4;
constexpr int kSgemm64GroupThreads = 64;
constexpr size_t kSgemm64TileFloats = (size_t)kSimtBK * kSgemm64Ld;
constexpr size_t kSgemm64StagingFloats = 8 * 4 * (size_t)kSgemm64GroupThreads; // eight chunks per thread
constexpr size_t kSgemm64GroupFloats = 4 * kSgemm64TileFloats + 2 * kSgemm64StagingFloats;
template <int G> constexpr size_t kSgemm64SmemBytes = G * kSgemm64GroupFloats * sizeof(float);
static_assert(kSgemm64 * kSgemm64 <= kSgemm64GroupFloats, "the partial tiles take the buffers' place");

template <int G>
__global__ void __launch_bounds__(G *kSgemm64GroupThreads, G == 2 ? 3 : 1)
sgemm64_kernel(const float *A, const float *B, float *C, uint32_t M, uint32_t N,
               uint32_t K, float alpha, uint32_t S, uint32_t *status)
{
    extern __shared__ __align__(16) float ssm[];
    const int group = threadIdx.x / kSgemm64GroupThreads, tid = threadIdx.x % kSgemm64GroupThreads;
    float *const tiles = ssm + group * kSgemm64GroupFloats;     // [buffer][A, B][k][kSgemm64Ld]
    float *const staging = tiles + 4 * kSgemm64TileFloats;      // [buffer][chunk][thread] of float4
    uint32_t tm, tn;
    const uint32_t rank = blockIdx.x % S;
    raster(blockIdx.x / S, (M + kSgemm64 - 1) / kSgemm64, (N + kSgemm64 - 1) / kSgemm64, &tm, &tn);
    join_stream(status);
    const uint32_t nk_all = (K + kSimtBK - 1) / kSimtBK, kb0 = rank * nk_all / S, kb1 = (rank + 1) * nk_all / S;
    const uint32_t nk = kb1 - kb0 > (uint32_t)group ? (kb1 - kb0 - group - 1) / G + 1 : 0;   // this group's k blocks
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kSgemm64GroupThreads) : "memory"); };

    // the lane map of sgemm_kernel: 8 (rows) x 4 (columns) threads per warp
    const int lane = tid & 31, lx = (lane & 1) | ((lane >> 1) & 2), ly = ((lane >> 1) & 1) | ((lane >> 2) & 6);
    const int fa = ly * 4, fb = (tid >> 5) * 32 + lx * 4;
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    const uint32_t row_a = tm * kSgemm64 + lrow, row_b = tn * kSgemm64 + lrow;
    const float *srcA = A + (size_t)row_a * K + lk, *srcB = B + (size_t)row_b * K + lk;
    auto fetch = [&](uint32_t i) {                              // the group's i-th k block into staging buffer i % 2
        float *st = staging + (i & 1) * kSgemm64StagingFloats + tid * 4;
        const uint32_t k0 = (kb0 + i * G + group) * kSimtBK;
        const bool in_k = k0 + lk < K;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const bool in_a = in_k && row_a + 16 * c < M, in_b = in_k && row_b + 16 * c < N;
            cp_async_16_or_zeros(st + c * 4 * kSgemm64GroupThreads, in_a ? srcA + (size_t)c * 16 * K + k0 : A, in_a);
            cp_async_16_or_zeros(st + (4 + c) * 4 * kSgemm64GroupThreads, in_b ? srcB + (size_t)c * 16 * K + k0 : B, in_b);
        }
    };
    auto transpose = [&](uint32_t i) {
        const float *st = staging + (i & 1) * kSgemm64StagingFloats + tid * 4;
        float *sA = tiles + (i & 1) * 2 * kSgemm64TileFloats, *sB = sA + kSgemm64TileFloats;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float4 v = *reinterpret_cast<const float4 *>(st + c * 4 * kSgemm64GroupThreads);
            float *dst = (c < 4 ? sA : sB) + lk * kSgemm64Ld + ((lrow + 16 * (c & 3)) ^ (lk & 8));     // see sgemm_kernel
            dst[0] = v.x; dst[kSgemm64Ld] = v.y; dst[2 * kSgemm64Ld] = v.z; dst[3 * kSgemm64Ld] = v.w;
        }
    };
    unsigned long long acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j] = 0ull;

#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
        if (i < nk)
            fetch(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (nk > 0)
        transpose(0);
    group_sync();
    for (uint32_t kb = 0; kb < nk; kb++) {
        // this thread emptied its part of staging buffer kb % 2 into the tile
        if (kb + 2 < nk)
            fetch(kb + 2);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *sA = tiles + (kb & 1) * 2 * kSgemm64TileFloats, *sB = sA + kSgemm64TileFloats;
#pragma unroll
        for (int k = 0; k < kSimtBK; k++) {
            const int ca = fa ^ (k & 8), cb = fb ^ (k & 8);
            float a[8];
            unsigned long long b[4];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float4 v = *reinterpret_cast<const float4 *>(sA + k * kSgemm64Ld + ca + 32 * q);
                a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 v = *reinterpret_cast<const float4 *>(sB + k * kSgemm64Ld + cb + 16 * h);
                b[2 * h] = pack2(v.x, v.y);
                b[2 * h + 1] = pack2(v.z, v.w);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const unsigned long long aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    ffma2(acc[i][j], aa, b[j]);
            }
        }
        if (kb + 1 < nk) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            transpose(kb + 1);
            group_sync();
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    __syncthreads();
    float *part = ssm + group * (kSgemm64 * kSgemm64);          // [group][64][64]
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 lo = unpack2(acc[i][2 * h]), hi = unpack2(acc[i][2 * h + 1]);
            *reinterpret_cast<float4 *>(part + (fa + 32 * (i >> 2) + (i & 3)) * kSgemm64 + fb + 16 * h) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    sum_partial_tiles<float, kSgemm64, kSgemm64, G, G * kSgemm64GroupThreads>(ssm, S, rank, C, tm * kSgemm64, tn * kSgemm64, M, N, alpha);
}

// ---------------------------------------------------------------------------------------------
// fp64
// ---------------------------------------------------------------------------------------------

constexpr int kDgemmTile = 64, kDgemmThreads = 128, kDgemmStages = 3;
constexpr int kDgemmPartLd = kDgemmTile + 8;             // doubles per row of a tile of C in shared memory: 16-byte pieces of two rows on all banks
constexpr size_t kDgemmStageDoubles = 2 * (size_t)kDgemmTile * kSimtBK;
constexpr size_t kDgemmSmemBytes = kDgemmStages * kDgemmStageDoubles * sizeof(double);
static_assert(kDgemmTile * kDgemmPartLd * sizeof(double) <= kDgemmSmemBytes, "the tile of C takes the ring's place");

__device__ __forceinline__ void dmma_m8n8k4(double &d0, double &d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// rows g and g + 8 of 16 (g = lane / 4): the same operations as two m8n8k4, in half the instructions
__device__ __forceinline__ void dmma_m16n8k4(double (&upper)[2], double (&lower)[2], double a_upper, double a_lower, double b)
{
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
        : "+d"(upper[0]), "+d"(upper[1]), "+d"(lower[0]), "+d"(lower[1])
        : "d"(a_upper), "d"(a_lower), "d"(b));
}

// 64 x 64 tile, four warps of 32 x 32, four CTAs per SM.  RAGGED as for sgemm_kernel.  STAGED: N is odd, so that pairs of columns are
// not aligned; a tile of C goes through shared memory and leaves in whole rows of single doubles.
template <bool RAGGED, bool STAGED>
__global__ void __launch_bounds__(kDgemmThreads, 4)
dgemm_kernel(const double *A, const double *B, double *C, uint32_t M, uint32_t N,
             uint32_t K, double alpha, uint32_t *status)
{
    static_assert(RAGGED || !STAGED, "whole tiles have an even N");
    extern __shared__ __align__(16) double dsm[];
    uint32_t tm, tn;
    raster(blockIdx.x, (M + kDgemmTile - 1) / kDgemmTile, (N + kDgemmTile - 1) / kDgemmTile, &tm, &tn);
    join_stream(status);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;              // this warp's 32 x 32 corner inside the tile
    const double *gA = A + (size_t)tm * kDgemmTile * K, *gB = B + (size_t)tn * kDgemmTile * K;

    // One stage = A tile [64][16] then B tile [64][16] in 16-byte chunks, eight per row; chunk c of row r lies at c ^ 2 (r % 4), so
    // that the fragment reads of a half warp (four rows, four k) fall in 16 distinct 8-byte banks.  Piece i of it is 16 rows, the
    // first four pieces A's.  Ragged: zeros arrive in place of what lies beyond an operand, and of a whole piece without `more`.
    constexpr int kPieces = 2 * kDgemmTile * 8 / kDgemmThreads;
    auto load_piece = [&](int stage, uint32_t k0, int i, bool more) {
        const int c = tid + kDgemmThreads * (i % (kPieces / 2)), r = c >> 3, kc = (c & 7) * 2;
        const bool is_a = i < kPieces / 2;
        double *dst = dsm + (size_t)stage * kDgemmStageDoubles + (r + (is_a ? 0 : kDgemmTile)) * kSimtBK + (kc ^ ((r & 3) << 2));
        const double *src = (is_a ? gA : gB) + (size_t)r * K + k0 + kc;
        if (RAGGED) {
            const bool inside = more && (is_a ? tm * kDgemmTile + r < M : tn * kDgemmTile + r < N) && k0 + kc < K;
            cp_async_16_or_zeros(dst, inside ? src : A, inside);
        } else {
            cp_async_16(dst, src);
        }
    };
    auto load_stage = [&](int stage, uint32_t k0) {
#pragma unroll
        for (int i = 0; i < kPieces; i++)
            load_piece(stage, k0, i, true);
    };

    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j][0] = acc[i][j][1] = 0.0;

    const uint32_t nk = (K + kSimtBK - 1) / kSimtBK;
#pragma unroll
    for (int s = 0; s < kDgemmStages - 1; s++) {
        if ((uint32_t)s < nk)
            load_stage(s, s * kSimtBK);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int fr = lane >> 2, fk = lane & 3;                        // fragment row (or column of B) and k of this lane
    for (uint32_t kb = 0; kb < nk; kb++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDgemmStages - 2) : "memory");
        __syncthreads();                                            // stage kb has landed; stage kb-1 is free for reuse
        // Whole tiles ask for the next block here.  Ragged ones do so a piece at a time under the multiplications: the tests on
        // each piece would hold up a warp that has its scheduler to itself (109 x 8532 x 4434 345 -> 327 us, 2290 x 1258 x 5472
        // 1140 -> 999; for whole tiles 1 % slower).
        const uint32_t next = kb + kDgemmStages - 1;
        if (!RAGGED && next < nk)
            load_stage(next % kDgemmStages, next * kSimtBK);
        const double *sa = dsm + (size_t)(kb % kDgemmStages) * kDgemmStageDoubles + (wm + fr) * kSimtBK;
        const double *sb = dsm + (size_t)(kb % kDgemmStages) * kDgemmStageDoubles + (kDgemmTile + wn + fr) * kSimtBK;
#pragma unroll
        for (int k4 = 0; k4 < kSimtBK; k4 += 4) {
            const int at = (k4 ^ ((fr & 3) << 2)) + fk;
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                a[i] = sa[8 * i * kSimtBK + at];
#pragma unroll
            for (int j = 0; j < 4; j++)
                b[j] = sb[8 * j * kSimtBK + at];
            if (RAGGED) {
#pragma unroll
                for (int i = 0; i < kPieces / 4; i++)
                    load_piece(next % kDgemmStages, next * kSimtBK, k4 / 4 * (kPieces / 4) + i, next < nk);
            }
#pragma unroll
            for (int i = 0; i < 4; i += 2)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    dmma_m16n8k4(acc[i][j], acc[i + 1][j], a[i], a[i + 1], b[j]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // accumulator tile (i, j): this lane holds row lane/4, columns 2*(lane%4) and the next one
    if constexpr (STAGED) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                *reinterpret_cast<double2 *>(dsm + (wm + 8 * i + fr) * kDgemmPartLd + wn + 8 * j + 2 * fk) = make_double2(alpha * acc[i][j][0], alpha * acc[i][j][1]);
        __syncthreads();
        const uint32_t col = tn * kDgemmTile + lane;
#pragma unroll
        for (int i = 0; i < kDgemmTile / 4; i++) {
            const int r = warp + 4 * i;
            const uint32_t row = tm * kDgemmTile + r;
            double *dst = C + (size_t)row * N + col;
            if (row < M && col < N)
                dst[0] = dsm[r * kDgemmPartLd + lane];
            if (row < M && col + 32 < N)
                dst[32] = dsm[r * kDgemmPartLd + lane + 32];
        }
        return;
    }
    double *gC = C + ((size_t)tm * kDgemmTile + wm) * N + (size_t)tn * kDgemmTile + wn;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (!RAGGED || (tm * kDgemmTile + wm + 8 * i + fr < M && tn * kDgemmTile + wn + 8 * j + 2 * fk < N))
                *reinterpret_cast<double2 *>(gC + (size_t)(8 * i + fr) * N + 8 * j + 2 * fk) = make_double2(alpha * acc[i][j][0], alpha * acc[i][j][1]);
}

// Smaller tiles, K split over the CTAs of a cluster and over WK groups of WM x WN warps inside a CTA; 32 x 32 outputs
// per warp (4 x 4 accumulator tiles, eight fragment loads per 16 DMMAs of 16 cycles each).  A group takes every WK-th
// block of eight k of its CTA's range through a ring of its own; a group of one warp meets nobody.  Three stages, so that
// three CTAs of four one-warp groups fit an SM: with four stages and two CTAs 10215 x 138 x 872 took 122 us against 103,
// 863 x 251 x 2456 50 against 42.
// Rows of 12 doubles put the fragment reads of a half warp into 16 different 8-byte banks.
constexpr int kDsplitBK = 8, kDsplitLd = kDsplitBK + 4, kDsplitStages = 3;
template <int WM, int WN, int WK> struct DgemmSplit {
    static constexpr int rows = 32 * WM, cols = 32 * WN, group_threads = 32 * WM * WN, threads = group_threads * WK;
    static constexpr size_t stage_doubles = (size_t)(rows + cols) * kDsplitLd, group_doubles = kDsplitStages * stage_doubles;
    static constexpr size_t smem_bytes = WK * group_doubles * sizeof(double);
    static constexpr int ctas_per_sm = 220 * 1024 / smem_bytes < 4 ? (int)(220 * 1024 / smem_bytes) : 4;
    static_assert((size_t)rows * cols <= group_doubles, "the partial tiles take the rings' place");
    static_assert(WK == 1 || WM * WN == 1, "groups of several warps would need named barriers");
};

template <int WM, int WN, int WK>
__global__ void __launch_bounds__(DgemmSplit<WM, WN, WK>::threads, DgemmSplit<WM, WN, WK>::ctas_per_sm)
dgemm_split_kernel(const double *A, const double *B, double *C, uint32_t M, uint32_t N,
                   uint32_t K, double alpha, uint32_t S, uint32_t *status)
{
    extern __shared__ __align__(16) double dsm[];
    using D = DgemmSplit<WM, WN, WK>;
    uint32_t tm, tn;
    const uint32_t rank = blockIdx.x % S;
    raster(blockIdx.x / S, (M + D::rows - 1) / D::rows, (N + D::cols - 1) / D::cols, &tm, &tn);
    join_stream(status);
    const int group = threadIdx.x / D::group_threads, tid = threadIdx.x % D::group_threads, lane = tid & 31, warp = tid >> 5;
    const uint32_t nk_all = (K + kDsplitBK - 1) / kDsplitBK, kb0 = rank * nk_all / S, kb1 = (rank + 1) * nk_all / S;
    const uint32_t nk = kb1 - kb0 > (uint32_t)group ? (kb1 - kb0 - group - 1) / WK + 1 : 0;       // this group's blocks
    const int wm = warp / WN * 32, wn = warp % WN * 32;
    double *ring = dsm + group * D::group_doubles;
    auto group_sync = [&]() {
        if constexpr (D::group_threads == 32)
            __syncwarp();
        else
            __syncthreads();
    };

    auto load_stage = [&](uint32_t i) {                          // the group's i-th block
        double *st = ring + (size_t)(i % kDsplitStages) * D::stage_doubles;
        const uint32_t k0 = (kb0 + i * WK + group) * kDsplitBK;
#pragma unroll
        for (int u = 0; u < (D::rows + D::cols) * 4 / D::group_threads; u++) {
            const int c = tid + D::group_threads * u, r = c >> 2, kc = (c & 3) * 2;
            const bool is_a = r < D::rows;
            const uint32_t row = is_a ? tm * D::rows + r : tn * D::cols + (r - D::rows);
            const bool inside = row < (is_a ? M : N) && k0 + kc < K;
            const double *base = is_a ? A : B;
            cp_async_16_or_zeros(st + r * kDsplitLd + kc, inside ? base + (size_t)row * K + k0 + kc : base, inside);
        }
    };
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int d = 0; d < kDsplitStages - 1; d++) {
        if ((uint32_t)d < nk)
            load_stage(d);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int fr = lane >> 2, fk = lane & 3;
    for (uint32_t kb = 0; kb < nk; kb++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDsplitStages - 2) : "memory");
        group_sync();                                            // block kb has landed; the stage of kb - 1 is free
        if (kb + kDsplitStages - 1 < nk)
            load_stage(kb + kDsplitStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double *sa = ring + (size_t)(kb % kDsplitStages) * D::stage_doubles, *sb = sa + D::rows * kDsplitLd;
#pragma unroll
        for (int k4 = 0; k4 < kDsplitBK; k4 += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                a[i] = sa[(wm + 8 * i + fr) * kDsplitLd + k4 + fk];
#pragma unroll
            for (int j = 0; j < 4; j++)
                b[j] = sb[(wn + 8 * j + fr) * kDsplitLd + k4 + fk];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    dmma_m8n8k4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    double *part = dsm + (size_t)group * D::rows * D::cols;      // [group][rows][cols]
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            *reinterpret_cast<double2 *>(part + (wm + 8 * i + fr) * D::cols + wn + 8 * j + 2 * fk) = make_double2(acc[i][j][0], acc[i][j][1]);
    sum_partial_tiles<double, D::rows, D::cols, WK, D::threads>(dsm, S, rank, C, tm * D::rows, tn * D::cols, M, N, alpha);
}

// CTAs that clusters of this size can have running at one per SM: GPCs of 16 to 20 SMs leave some over
static uint64_t simt_capacity(uint32_t cluster)
{
    const uint64_t sms = num_sms() > 0 ? (uint64_t)num_sms() : 148;
    return cluster <= 2 ? sms : cluster == 4 ? sms * 132 / 148 : sms * 120 / 148;
}

template <typename... Params, typename... Args>
static int launch_simt(void (*kernel)(Params...), const char *what, uint64_t ctas, int threads, size_t smem, uint32_t cluster, bool even_share,
                       cudaStream_t s, Args... args)
{
    // An even share per SM: a CTA that may start under the tail of the previous kernel goes where that has ended, and
    // some SMs would take three while others get none.  No more CTAs fit an SM than its share when they ask for enough
    // shared memory (fp32 4195 x 225 x 1980, 264 CTAs of 64 x 64: 151 -> 113 us, fp64 902 x 868 x 2356 182 -> 146).
    if (even_share) {
        const uint64_t share = (ctas - 1) / simt_capacity(cluster) + 1;
        const size_t fill = kSimtSmemMax / (share + 1) + 1024;
        if (share < 8 && fill > smem)
            smem = fill;
    }
    // The attribute is the kernel's, not the call's: a limit of this call's size would refuse the larger request of
    // another host thread between its own setting and its launch.
    CLPK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSimtSmemMax));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = tuning(CLPK_TUNE_GEMM_NO_PDL) == 1 ? 0 : 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
    if (e != cudaSuccess)
        return cuda_fail(e, what);
    return CLPK_OK;
}

// Kernel, tile edge and K ranges for a problem: the cheapest by an estimate in microseconds, fitted to 400 timed launches of all
// kernels on 90 shapes (M and N from 64 to 15000, K to 16000; residuals 5 to 9 %, 13 % for the 32-wide fp64 tile; the chosen plans
// are 2 to 3 % slower than the fastest in the geometric mean), and dgemm_kernel's to 400 more (4 %).  With L CTAs on the busiest
// SM, a block of 16 k costs its CTA  max(alone, L * shared):
//   fp32  128 x 128  max(1.62, 1.43 L)    64 x 64  max(0.51, 0.40 L)    (the pipe's own time: 1.07 and 0.27 L)
//   fp64  whole 64 x 64  max(0.75, 0.607 L)    split 64 x 64  max(0.91, 0.62 L)    32 x 32  max(0.22, 0.16 to 0.174 L, the less the
//   longer)    (0.54, 0.54, 0.13 L)
// A CTA alone on its SM with a range of 32 blocks (fp32) or 24 (fp64) takes twice the K groups: 0.41 and 0.18 a block,
// and 1.5 and 0.6 us more for the longer sum at the end (shorter ranges lose up to 20 % by it, long ones gain up to 33 %).
// The 128 x 128 tiles are kept unless the estimate is 8 % better; a K range has at least four blocks.  Short fp64 sums have an
// estimate of their own (plan_short_f64).
struct SimtPlan {
    uint32_t tile, splits;
    bool wide;                  // twice the K groups
    float us = 0.0f;            // the estimate it was chosen by (fp32 and long fp64 sums)
    bool whole = false;         // sgemm_kernel or dgemm_kernel
};

// dgemm_kernel is not considered for fewer tiles than two SMs of three have one.  32-wide tiles serve most of those better, up to
// three times; not all of them (1481 x 215 x 40: 5.9 us, 4.5 in 64-wide ones).
static uint64_t whole_f64_tiles(uint32_t m, uint32_t n)
{
    const uint64_t tiles = (uint64_t)((m - 1) / kDgemmTile + 1) * ((n - 1) / kDgemmTile + 1);
    return 3 * tiles < 2 * simt_capacity(1) ? 0 : tiles;
}

// fp64 with fewer than 24 blocks: what a CTA costs besides them -- start, pipeline fill, sum, stores -- is then a good part
// of its time, paid once per round of the CTAs that an SM holds (4 of 64 x 64, 3 of 32 x 32).  Fitted to 490 shapes with K from
// 2 to 368 (residuals 6 and 7 %; the chosen plans are 1 % slower than the fastest in the geometric mean, where the estimate
// above was 10 % slower and 2.7 times at worst) and, for dgemm_kernel, to 180 (4 %).
static SimtPlan plan_short_f64(uint32_t m, uint32_t n, uint32_t blocks)
{
    auto per_sm = [&](uint32_t rows, uint32_t cols, uint32_t splits) {
        return (uint32_t)(((uint64_t)((m - 1) / rows + 1) * ((n - 1) / cols + 1) * splits - 1) / simt_capacity(splits) + 1);
    };
    // `held` CTAs at a time, `alone` us for one by itself and `shared` for each of several
    auto rounds = [](uint32_t ctas, uint32_t held, float alone, float shared) {
        auto round = [&](uint32_t c) { return c == 0 ? 0.0f : alone > c * shared ? alone : c * shared; };
        return (float)(ctas / held) * round(held) + round(ctas % held);
    };
    SimtPlan plan = {32, 1, false};
    float best = 1e30f;
    if (whole_f64_tiles(m, n)) {
        best = 0.97f * (2.75f + rounds(per_sm(64, 64, 1), 4, 0.785f * (float)blocks - 0.71f, 0.587f * (float)blocks + 0.36f));
        plan = {kDgemmTile, 1, false, best, true};
    }
    for (uint32_t splits = 1; splits <= 4 && (splits == 1 || blocks >= 4 * splits); splits *= 2)
        for (uint32_t tile = 32; tile <= (splits == 1 ? 32u : 64u); tile *= 2) {
            const uint32_t ctas = per_sm(tile, tile, splits);
            const float range = (float)((blocks - 1) / splits + 1);
            const float t = tile == 64 ? 3.4f + rounds(ctas, 4, 0.92f * range + 1.54f, 0.60f * range + 1.05f)
                                       : 2.0f + rounds(ctas, 3, 0.254f * range + 1.67f, 0.18f * range + 1.12f) + (splits > 1 ? 0.29f * splits : 0.0f);
            if (t < best) {
                best = t;
                plan = {tile, splits, false};
            }
        }
    return plan;
}

static SimtPlan plan_simt(bool f64, uint32_t m, uint32_t n, uint32_t k)
{
    const uint32_t blocks = (k - 1) / kSimtBK + 1;
    if (f64 && blocks < 24)
        return plan_short_f64(m, n, blocks);
    auto ctas = [&](uint32_t rows, uint32_t cols, uint32_t splits) { return (uint64_t)((m - 1) / rows + 1) * ((n - 1) / cols + 1) * splits; };
    auto estimate = [&](uint32_t rows, uint32_t cols, uint32_t splits, float alone, float shared) {
        const float busiest = shared * (float)((ctas(rows, cols, splits) - 1) / simt_capacity(splits) + 1);
        return (float)((blocks - 1) / splits + 1) * (alone > busiest ? alone : busiest);
    };
    float best = 1e30f;
    SimtPlan plan = {32, 1, false};
    if (!f64) {
        const float large = 2.0f + estimate(128, 128, 1, 1.62f, 1.43f);
        best = 0.92f * large;
        plan = {kSimtTile, 1, false, large, true};
    } else if (whole_f64_tiles(m, n)) {
        best = 3.2f + estimate(64, 64, 1, 0.75f, 0.607f);
        plan = {kDgemmTile, 1, false, best, true};
    }
    for (uint32_t splits = 1; splits <= 8 && (splits == 1 || blocks >= 4 * splits); splits *= 2)
        // (fp64 in one range: dgemm_kernel's estimate is below the other 64-wide tiles' wherever it is considered, and where it is
        // not, an SM has three 32-wide tiles at most, which are cheaper too)
        for (uint32_t tile = f64 ? 32 : 64; tile <= (f64 && splits == 1 ? 32u : 64u); tile *= 2) {
            const bool wide = !(f64 && tile == 64) && ctas(tile, tile, splits) <= simt_capacity(splits) && blocks >= (f64 ? 24 : 32) * splits;
            float t;
            if (!f64)
                t = (wide ? 5.6f + estimate(64, 64, splits, 0.405f, 0.0f) : 4.1f + estimate(64, 64, splits, 0.507f, 0.404f)) +
                    (splits > 1 ? 1.1f + 0.08f * splits : 0.0f);
            else if (tile == 64)
                t = 4.56f + estimate(64, 64, splits, 0.907f, 0.616f);
            else
                t = (wide ? 4.5f + estimate(32, 32, splits, 0.178f, 0.0f)
                          : 3.9f + estimate(32, 32, splits, 0.223f, std::min(0.174f, 0.16f + 0.6f * (float)splits / (float)blocks))) +
                    (splits > 1 ? 0.5f * splits : 0.0f);
            if (t < best) {
                best = t;
                plan = {tile, splits, wide, t};
            }
        }
    return plan;
}

float simt_f32_estimate(uint32_t m, uint32_t n, uint32_t k) { return plan_simt(false, m, n, k).us; }

void simt_gemm_plan(bool f64, uint32_t m, uint32_t n, uint32_t k, uint32_t *tile_n, uint32_t *splits, uint32_t *wide)
{
    const SimtPlan plan = plan_simt(f64, m, n, k);
    *tile_n = plan.whole ? 0 : plan.tile;
    *splits = plan.splits;
    *wide = plan.wide ? 1 : 0;
}

// tiles of sgemm_kernel or dgemm_kernel
static uint64_t whole_tiles(int dtype, uint32_t m, uint32_t n)
{
    const uint32_t tile = dtype == CLPK_DT_F32 ? kSimtTile : kDgemmTile;
    return (uint64_t)((m - 1) / tile + 1) * ((n - 1) / tile + 1);
}

int check_simt_gemm(int dtype, const void *a, const void *b, const void *c, uint32_t m, uint32_t n, uint32_t k)
{
    CLPK_REQUIRE(m > 0 && n > 0 && k > 0, "M, N and K must be positive");
    const uint32_t k_unit = dtype == CLPK_DT_F32 ? 4 : 2;            // elements per 16 bytes: operand rows stay aligned
    CLPK_REQUIRE(k % k_unit == 0, "K = %u: a row of A and B must be a multiple of 16 bytes", k);
    CLPK_REQUIRE(((uintptr_t)a % 16) == 0 && ((uintptr_t)b % 16) == 0 && ((uintptr_t)c % 16) == 0, "operands must be 16-byte aligned");
    CLPK_REQUIRE((uint64_t)((m - 1) / 128 + 1) * ((n - 1) / (dtype == CLPK_DT_F32 ? 128 : 64) + 1) <= 0x3FFFFFFFull, "too many tiles");
    return CLPK_OK;
}

int launch_simt_gemm(int dtype, const void *a, const void *b, void *c, uint32_t m, uint32_t n, uint32_t k, float alpha,
                     uint32_t *status, cudaStream_t s)
{
    const uint32_t tile = dtype == CLPK_DT_F32 ? kSimtTile : kDgemmTile;
    const uint64_t tiles = whole_tiles(dtype, m, n);
    // whole tiles and whole k blocks take the kernel without the bounds checks
    const bool ragged = m % tile != 0 || n % tile != 0 || k % kSimtBK != 0;
    const SimtPlan plan = plan_simt(dtype == CLPK_DT_F64, m, n, k);
    const uint64_t ctas = (uint64_t)((m - 1) / plan.tile + 1) * ((n - 1) / plan.tile + 1) * plan.splits;
    if (dtype == CLPK_DT_F32) {
        const float *fa = static_cast<const float *>(a), *fb = static_cast<const float *>(b);
        float *fc = static_cast<float *>(c);
        if (!plan.whole)
            return plan.wide ? launch_simt(sgemm64_kernel<4>, "launch sgemm64", ctas, 4 * kSgemm64GroupThreads, kSgemm64SmemBytes<4>, plan.splits, false, s, fa, fb,
                                       fc, m, n, k, alpha, plan.splits, status)
                         : launch_simt(sgemm64_kernel<2>, "launch sgemm64", ctas, 2 * kSgemm64GroupThreads, kSgemm64SmemBytes<2>, plan.splits, true, s, fa, fb,
                                       fc, m, n, k, alpha, plan.splits, status);
        return launch_simt(ragged ? sgemm_kernel<true> : sgemm_kernel<false>, "launch sgemm", tiles, kSgemmThreads, kSgemmSmemBytes, 1, false, s, fa, fb,
                           fc, m, n, k, alpha, status);
    }
    const double *da = static_cast<const double *>(a), *db = static_cast<const double *>(b);
    double *dc = static_cast<double *>(c);
    if (plan.whole) {
        const bool odd = n % 2 != 0;
        return launch_simt(odd ? dgemm_kernel<true, true> : ragged ? dgemm_kernel<true, false> : dgemm_kernel<false, false>, "launch dgemm", tiles, kDgemmThreads,
                           kDgemmSmemBytes, 1, true, s, da, db, dc, m, n, k, alpha, status);
    }
    if (plan.tile == 64)
        return launch_simt(dgemm_split_kernel<2, 2, 1>, "launch dgemm 64", ctas, DgemmSplit<2, 2, 1>::threads, DgemmSplit<2, 2, 1>::smem_bytes, plan.splits,
                           true, s, da, db, dc, m, n, k, alpha, plan.splits, status);
    if (plan.tile == 32 && plan.wide)
        return launch_simt(dgemm_split_kernel<1, 1, 8>, "launch dgemm 32", ctas, DgemmSplit<1, 1, 8>::threads, DgemmSplit<1, 1, 8>::smem_bytes, plan.splits,
                           false, s, da, db, dc, m, n, k, alpha, plan.splits, status);
    return launch_simt(dgemm_split_kernel<1, 1, 4>, "launch dgemm 32", ctas, DgemmSplit<1, 1, 4>::threads, DgemmSplit<1, 1, 4>::smem_bytes, plan.splits, true, s,
                       da, db, dc, m, n, k, alpha, plan.splits, status);
}

} // namespace clpk
