// C[M][N] = A[M][K] * B[N][K]^T on tcgen05.mma, the in-house replacement for the
// cuBLASLt call the reference makes for its "GEMM peak" rows.
//
// Shape of the dense kernel (gemm_kernel; the block-scaled FP4 kernel further down
// keeps a 256 x 256 cluster tile because its scale factors need tensor-memory columns)
//  * Persistent: one 2-CTA cluster per SM pair, tiles handed out round-robin.
//  * A cluster computes a 512 x 256 tile with 2-SM MMAs (cta_group::2, M = 256,
//    N = 256), two row blocks sharing one B tile; each CTA holds 256 x 256 of the
//    accumulator, i.e. all of its tensor memory.  The MMA reads both CTAs' shared
//    memory.  No TMA multicast anywhere: each CTA fetches what it needs itself.
//  * Warp roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer (leader
//    CTA only) and TMEM owner, warps 2-9 epilogue (TMEM -> registers -> output
//    type -> swizzled staging box in shared memory -> TMA store).  The roles
//    that issue TMA or tcgen05 instructions run their loops as whole warps and
//    let one elected lane issue.
//  * K is consumed in blocks of 128 bytes per row (64 x 16-bit, 128 x 8-bit),
//    the width of one 128-byte-swizzled TMA box; a stage is two 16 KiB A
//    sub-tiles (one per row block) and this CTA's 16 KiB half of B, four
//    stages.  Both CTAs' loads signal the leader's "full" barrier;
//    tcgen05.commit releases a stage in both CTAs at once.
//  * Every mbarrier wait is bounded; on expiry the status word is set and all
//    roles fall through to the common exit, which frees tensor memory.
//
// Algorithmic work: 2*M*N*K flop per call; HBM traffic at least
// (M*K + N*K)*elem + M*N*2 bytes (each operand read once, C written once).
#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "../clpk_internal.h"
#include "../clpk_ptx.cuh"

namespace clpk {

constexpr uint32_t kRowBytesK = 128;                        // K bytes per row per stage
constexpr uint32_t kHalfTileBytes = 128 * kRowBytesK;       // 16 KiB: 128 rows x 128 B
constexpr uint32_t kTileMN = 256;
constexpr int kGemmThreads = 320;                          // dense kernel: producer, MMA, 8 epilogue warps

struct GemmParams {
    uint32_t m, n, k;
    uint32_t k_blocks;          // K / (elements per 128 B)
    uint32_t k_block_elems;
    void *c;                    // bf16, or fp32 (TF32) / int32 (I8): see out_elem_bytes()
    float alpha;
    uint32_t *status;
    uint32_t group;             // tile columns per raster group (both kernels)
    unsigned int *wave_sync;    // {arrivals, CTAs that are done} of this launch, or NULL: see wave_align()
    uint32_t align_at;          // K block of a tile before which the producers meet
    uint32_t align_period;      // ... in every align_period-th wave
    unsigned long long *clock;  // two words: CTA 0 stores the SM cycles and nanoseconds it ran for (clpk_gemm_last_clock)
};

// Launches of a small GEMM repeat every 40-100 us, and 6-7 us of each are the CTA's set-up (barriers, tensor
// memory, descriptor prefetch) and the launch gap.  The launches therefore carry the
// programmatic-serialisation attribute: a CTA of launch i + 1 takes an SM as soon as launch i's CTA there has
// exited, does its set-up, and then waits here until launch i has completed as a whole and its writes are visible.
// Nothing of global memory is read or written before that point.
__device__ __forceinline__ void join_previous_launch(const GemmParams &p)
{
    griddep_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *p.status = 0u;             // by the kernel: no stream operation sits between two launches
    griddep_launch_dependents();
}

// Output element of a GEMM dtype: fp32 for TF32, int32 for I8, bf16 for everything else.
template <int DT> struct OutBytes { static constexpr uint32_t value = (DT == CLPK_DT_TF32 || DT == CLPK_DT_I8) ? 4u : 2u; };

// 2-D tile load whose completion bytes go to the pair's leader CTA: leader_bar is its barrier's address (leader_addr).
__device__ __forceinline__ void tma_load_pair_at(void *smem_dst, const CUtensorMap *tmap, int32_t x, int32_t y,
                                                 uint32_t leader_bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(leader_bar), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ uint32_t leader_addr(const void *p)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}

// Roles that issue TMA or tcgen05 instructions run their loops with the whole warp and let
// one elected lane issue.  Addresses and descriptors are then warp-uniform values, which is
// what those instructions take.  With the loop inside `if (lane == 0)` each instruction cost
// its thread 110-130 cycles (measured with clock64 around it: four MMAs 460 cycles, against
// 115 this way), and a thread that must issue four MMAs and a commit per 512 tensor-core
// cycles, or eight and a commit per 1024, was the slowest stage of the pipeline.
// warp_wait: every lane waits; the verdict is made uniform so that the warp stays together.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, mbar_wait(bar, parity) ? 1 : 0) != 0;
}

// DT: BF16 / F16 -> kind::f16 (K = 16 per instruction); E4M3 / E5M2 -> kind::f8f6f4 (K = 32);
// TF32 -> kind::tf32 (K = 8, fp32 out); I8 -> kind::i8 (K = 32, int32 out).  Always 128 bytes of K per stage.
//
// Tile shape.  A cluster computes 512 x 256 of C: two M = 256 row blocks ("halves") that
// share one B tile.  Row block h covers cluster rows [256h, 256h + 256); CTA r of the pair
// owns the r-th 128 of them and keeps that part of the accumulator in tensor-memory
// columns [256h, 256h + 256) -- all 512 columns of each CTA are accumulator.  Per stage a
// CTA loads two 16 KiB A sub-tiles and its 16 KiB half of B (48 KiB; four stages), and the
// leader issues eight 2-CTA instructions (2 halves x 4 K steps).  Against a 256 x 256
// cluster tile this reads a third fewer operand bytes per flop from L2 and DRAM and reads
// B from shared memory once for two row blocks; the price is that the accumulator cannot
// be double-buffered, so the epilogue of a tile (a few microseconds per ~200) is exposed.
// Rows of C beyond M (M a multiple of 256 but not of 512) come out of zero-filled TMA boxes
// and are not stored.
constexpr int kDenseStages = 4;
constexpr uint32_t kDenseStageBytes = 3 * kHalfTileBytes;          // A half 0, A half 1, B half
constexpr uint32_t kDenseTileM = 512;

constexpr int kEpilogueWarps = 8;
constexpr uint32_t kStagingBytes = 32 * 128;                       // 32 rows x 128 bytes of C

struct DenseSmem {
    uint64_t full[kDenseStages];
    uint64_t empty[kDenseStages];
    uint64_t tmem_full;
    uint64_t tmem_empty;
    uint32_t tmem_base;
};

// Tiles are walked in groups of `group` tile columns, M fastest inside a group.
__device__ __forceinline__ void dense_tile_coords(uint32_t tile, uint32_t tiles_m, uint32_t tiles_n, uint32_t group,
                                                  uint32_t &mb, uint32_t &nb)
{
    const uint32_t per_group = group * tiles_m;
    const uint32_t g = tile / per_group;
    const uint32_t within = tile - g * per_group;
    const uint32_t first_n = g * group;
    const uint32_t width = (tiles_n - first_n) < group ? (tiles_n - first_n) : group;
    mb = within / width;
    nb = first_n + within % width;
}

// Epilogue of one warp for one tile of the dense kernel: the warp's 32 rows (TMEM lanes) x 128 columns of each
// of the two row blocks, moved in boxes of 128 bytes per row (64 bf16 or 32 fp32/int32 columns): tcgen05.ld ->
// convert -> the warp's own 4 KiB staging box in shared memory, written in the 128-byte swizzle so that the 32
// lanes (one row each) spread over the banks -> one TMA store per box, which writes whole lines of C and clips
// rows and columns beyond M and N.  (A thread-per-row store straight to global memory costs 32 partial-sector
// transactions per instruction and held the drain of a 256 x 256 CTA tile at 8 us.)  `empty_bar` (in the leader
// CTA) is arrived on as soon as the tile's last tcgen05.ld has landed: the next tile may then overwrite tensor
// memory while the tail of the stores is still in flight.
//   taddr0   : tensor-memory address of this warp's lanes, column 0 of its 128 columns, row block 0
//   row0/col0: C coordinates of the same element
// What a tile's hand-over costs was traced with clock64 stamps on 4 clusters at a fixed 1.84 GHz (K from 1024 to
// 16384: a stage costs its 1024 cycles, a tile a constant on top).  The main loop cannot start the next tile
// before tensor memory is free (both row blocks fill all 512 columns), so everything between the tile's last
// instruction retiring and the arrive on `empty_bar` is exposed once per tile.  In the first version of this
// epilogue that was 5 200 cycles, of which the tcgen05.ld themselves were 700 (a probe reads tensor memory at
// 245 bytes per cycle with eight warps): the rest was two staging boxes stored before row block 1 was read (the
// second box waits until TMA has read the first out of shared memory, 800-1400 cycles behind the operand loads),
// and an mbarrier.arrive.release.cluster that took 1 650 cycles to retire because a release waits for the warp's
// earlier shared-memory and bulk stores.  Now every column is read and converted before anything is stored and
// the arrive is relaxed (the hand-over carries no memory): 2 200 cycles, 8192^3 fp8 3.9 % and NVFP4 5.5 % fewer.

// one staging box out: wait until the previous store has read the box, fill it, hand it to TMA
__device__ __forceinline__ void store_staged_box(const uint32_t (&w)[32], uint8_t *box, const CUtensorMap *tmap_c, uint32_t col,
                                                 uint32_t row, int lane)
{
    uint8_t *my_row = box + lane * 128;
    const uint32_t sw = (uint32_t)(lane & 7);
    if (lane == 0)
        bulk_wait_read<0>();
    __syncwarp();
#pragma unroll
    for (uint32_t j = 0; j < 8; j++)
        *reinterpret_cast<uint4 *>(my_row + ((j ^ sw) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
        tma_store_2d(tmap_c, box, (int32_t)col, (int32_t)row);
        bulk_commit();
    }
}

__device__ __forceinline__ void pack_bf16x64(uint32_t (&w)[32], const uint32_t (&r0)[32], const uint32_t (&r1)[32], float alpha)
{
    // The conversion sits between the reads and the release of tensor memory; alpha = 1 (every dense row of the
    // benchmark) skips the 64 multiplies, which are two thirds of its instructions.  x * 1.0f is x, bit for bit.
    if (alpha == 1.0f) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            __nv_bfloat162 v0 = __floats2bfloat162_rn(__uint_as_float(r0[2 * i]), __uint_as_float(r0[2 * i + 1]));
            __nv_bfloat162 v1 = __floats2bfloat162_rn(__uint_as_float(r1[2 * i]), __uint_as_float(r1[2 * i + 1]));
            w[i] = *reinterpret_cast<uint32_t *>(&v0);
            w[16 + i] = *reinterpret_cast<uint32_t *>(&v1);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) {
        __nv_bfloat162 v0 = __floats2bfloat162_rn(__uint_as_float(r0[2 * i]) * alpha, __uint_as_float(r0[2 * i + 1]) * alpha);
        __nv_bfloat162 v1 = __floats2bfloat162_rn(__uint_as_float(r1[2 * i]) * alpha, __uint_as_float(r1[2 * i + 1]) * alpha);
        w[i] = *reinterpret_cast<uint32_t *>(&v0);
        w[16 + i] = *reinterpret_cast<uint32_t *>(&v1);
    }
}

template <int DT>
__device__ __forceinline__ void drain_warp_tile_wide(uint32_t taddr0, uint32_t row0, uint32_t col0, uint8_t *box,
                                                     const CUtensorMap *tmap_c, float alpha, uint64_t *empty_bar, int lane)
{
    // The hand-over carries no memory (the reads have completed: tcgen05.wait::ld), so the arrive needs no release:
    // with it the instruction took 1 650 cycles to retire here -- it waits for the warp's earlier shared-memory and
    // bulk stores -- against 400 without.
    auto release = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
            mbar_arrive_cluster_relaxed(empty_bar, 0);
    };
    if constexpr (OutBytes<DT>::value == 2) {
        // 16-bit outputs: every column of the warp's lanes is read and packed (128 registers) before anything is
        // written out, so that tensor memory is held for the reads alone: row block 0 with four tcgen05.ld in
        // flight, row block 1 in two rounds of two (the register file holds no more).
        uint32_t w0[32], w1[32], w2[32], w3[32];
        {
            uint32_t r0[32], r1[32], r2[32], r3[32];
            tmem_ld_32x32b_x32(taddr0, r0);
            tmem_ld_32x32b_x32(taddr0 + 32, r1);
            tmem_ld_32x32b_x32(taddr0 + 64, r2);
            tmem_ld_32x32b_x32(taddr0 + 96, r3);
            tmem_ld_wait();
            pack_bf16x64(w0, r0, r1, alpha);
            pack_bf16x64(w1, r2, r3, alpha);
        }
        {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32b_x32(taddr0 + 256, r0);
            tmem_ld_32x32b_x32(taddr0 + 256 + 32, r1);
            tmem_ld_wait();
            pack_bf16x64(w2, r0, r1, alpha);
        }
        {
            uint32_t r0[32], r1[32];
            tmem_ld_32x32b_x32(taddr0 + 256 + 64, r0);
            tmem_ld_32x32b_x32(taddr0 + 256 + 96, r1);
            tmem_ld_wait();
            release();
            pack_bf16x64(w3, r0, r1, alpha);
        }
        store_staged_box(w0, box, tmap_c, col0, row0, lane);
        store_staged_box(w1, box, tmap_c, col0 + 64, row0, lane);
        store_staged_box(w2, box, tmap_c, col0, row0 + 256, lane);
        store_staged_box(w3, box, tmap_c, col0 + 64, row0 + 256, lane);
    } else {
        // 32-bit outputs: a row block's 128 columns per round, four boxes of 32 columns
#pragma unroll 1
        for (uint32_t h = 0; h < 2; h++) {
            uint32_t r0[32], r1[32], r2[32], r3[32];
            tmem_ld_32x32b_x32(taddr0 + h * 256, r0);
            tmem_ld_32x32b_x32(taddr0 + h * 256 + 32, r1);
            tmem_ld_32x32b_x32(taddr0 + h * 256 + 64, r2);
            tmem_ld_32x32b_x32(taddr0 + h * 256 + 96, r3);
            tmem_ld_wait();
            if (h == 1)
                release();
            if constexpr (DT == CLPK_DT_TF32) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    r0[i] = __float_as_uint(__uint_as_float(r0[i]) * alpha);
                    r1[i] = __float_as_uint(__uint_as_float(r1[i]) * alpha);
                    r2[i] = __float_as_uint(__uint_as_float(r2[i]) * alpha);
                    r3[i] = __float_as_uint(__uint_as_float(r3[i]) * alpha);
                }
            }
            store_staged_box(r0, box, tmap_c, col0, row0 + h * 256, lane);
            store_staged_box(r1, box, tmap_c, col0 + 32, row0 + h * 256, lane);
            store_staged_box(r2, box, tmap_c, col0 + 64, row0 + h * 256, lane);
            store_staged_box(r3, box, tmap_c, col0 + 96, row0 + h * 256, lane);
        }
    }
}

// The same for a kernel with a single accumulator (bf16 output, one row block), where the
// next tile's main loop cannot start before tensor memory is free: all 128 columns are read
// and tensor memory is released before anything is written out.  Two rounds of two
// tcgen05.ld (64 fp32 registers in flight, 32 packed ones kept) rather than one of four,
// which would not fit the register file.
// ROUNDS = boxes of 64 columns this warp owns: 2 (a 128-column share) or 1 (a 64-column share).
template <int ROUNDS>
__device__ __forceinline__ void drain_warp_tile_early(uint32_t taddr0, uint32_t row0, uint32_t col0, uint8_t *box,
                                                      const CUtensorMap *tmap_c, float alpha, uint64_t *empty_bar,
                                                      int lane)
{
    uint8_t *my_row = box + lane * 128;
    const uint32_t sw = (uint32_t)(lane & 7);
    uint32_t w[ROUNDS][32];
#pragma unroll
    for (uint32_t b = 0; b < ROUNDS; b++) {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(taddr0 + b * 64, r0);
        tmem_ld_32x32b_x32(taddr0 + b * 64 + 32, r1);
        tmem_ld_wait();
        if (b == ROUNDS - 1) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                mbar_arrive_cluster_relaxed(empty_bar, 0);      // see drain_warp_tile_wide
        }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            __nv_bfloat162 v0 = __floats2bfloat162_rn(__uint_as_float(r0[2 * i]) * alpha, __uint_as_float(r0[2 * i + 1]) * alpha);
            __nv_bfloat162 v1 = __floats2bfloat162_rn(__uint_as_float(r1[2 * i]) * alpha, __uint_as_float(r1[2 * i + 1]) * alpha);
            w[b][i] = *reinterpret_cast<uint32_t *>(&v0);
            w[b][16 + i] = *reinterpret_cast<uint32_t *>(&v1);
        }
    }
#pragma unroll
    for (uint32_t b = 0; b < ROUNDS; b++) {
        // the previous box must have been read out of shared memory by its store
        if (lane == 0)
            bulk_wait_read<0>();
        __syncwarp();
#pragma unroll
        for (uint32_t j = 0; j < 8; j++)
            *reinterpret_cast<uint4 *>(my_row + ((j ^ sw) << 4)) =
                make_uint4(w[b][4 * j], w[b][4 * j + 1], w[b][4 * j + 2], w[b][4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(tmap_c, box, (int32_t)(col0 + b * 64), (int32_t)row0);
            bulk_commit();
        }
    }
}

// Keeping the clusters in step.  The schedule is static, so all clusters start wave w
// (their w-th tile) together only if they run at exactly the same speed.  They do not:
// measured on a B200, the start times of a wave spread by about 4 us more with every
// wave (some SM pairs are persistently ~1.7 % slower), 70 us after 20 waves.  Clusters
// that share an operand panel then ask for it that far apart, the L2 has long replaced
// it, and every panel is fetched from DRAM several times per wave.  So the producers
// meet before each wave: every CTA adds one to a counter and waits until the counter
// shows that all CTAs of the wave have arrived.  There is one CTA per SM, so they are normally all resident; the wait
// is bounded all the same: a CTA that has waited 40 us (another stream's kernel holds an SM) stops taking part, after
// which the others time out once each and the kernel finishes unaligned.  The last CTA to leave clears the counter for
// the launch that gets it next (leave_wave_sync).  A cooperative launch behind two clearing operations, the first form
// of this, cost about 5 us a GEMM: e4m3 8192 x 8192 x 512 40.3 -> 35.8 us, x 1024 67 -> 62, bf16 x 1024 113 -> 105, NVFP4
// 16384 x 16384 x 1024 196 -> 170, back to back.
__device__ unsigned int g_wave_dropouts;       // producers that have stopped taking part since the library was loaded

__device__ __forceinline__ void wave_align(const GemmParams &p, uint32_t wave, uint32_t n_tiles, uint32_t n_clusters,
                                           bool &enabled)
{
    // every align_period-th wave (short tiles drift less per wave and a meeting costs about a microsecond)
    if (!enabled || wave == 0 || wave % p.align_period != 0)
        return;
    // arrivals expected up to and including this meeting: two CTAs per cluster for each earlier
    // meeting (those waves were full) plus two per tile of this wave
    const uint32_t in_wave = n_tiles - wave * n_clusters < n_clusters ? n_tiles - wave * n_clusters : n_clusters;
    const unsigned int target = 2u * (n_clusters * (wave / p.align_period - 1u) + in_wave);
    atomicAdd(p.wave_sync, 1u);
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (;;) {
        unsigned int seen;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.wave_sync) : "memory");
        if (seen >= target)
            return;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 40000ull) {
            enabled = false;
            atomicAdd(&g_wave_dropouts, 1u);
            return;
        }
        __nanosleep(64);
    }
}

// By the thread that arrived for its CTA's producer, at the end of the kernel.
__device__ __forceinline__ void leave_wave_sync(const GemmParams &p)
{
    if (!p.wave_sync)
        return;
    __threadfence();                                        // this CTA's arrivals come before its leaving
    if (atomicInc(p.wave_sync + 1, gridDim.x - 1) == gridDim.x - 1)
        atomicExch(p.wave_sync, 0u);
}

template <int DT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads)
    gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                const __grid_constant__ CUtensorMap tmap_c, GemmParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // The runtime only guarantees 16-byte alignment of dynamic shared memory;
    // the swizzled tiles need 1024.
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *staging = smem + (size_t)kDenseStages * kDenseStageBytes;           // one 4 KiB box per epilogue warp
    DenseSmem *sh = reinterpret_cast<DenseSmem *>(staging + kEpilogueWarps * kStagingBytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t cluster_id = blockIdx.x >> 1;
    const uint32_t n_clusters = gridDim.x >> 1;
    const uint32_t tiles_m = (p.m + kDenseTileM - 1) / kDenseTileM, tiles_n = (p.n + kTileMN - 1) / kTileMN;
    const uint32_t n_tiles = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kDenseStages; s++) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        mbar_init(&sh->tmem_full, 1);
        mbar_init(&sh->tmem_empty, 16);      // 8 epilogue warps x 2 CTAs
        mbar_fence_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_c);
    }
    if (warp == 1)
        tmem_alloc<2>(&sh->tmem_base, 512);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    tc_fence_after_sync();
    const uint32_t tmem = sh->tmem_base;
    join_previous_launch(p);
    const unsigned long long clk0 = clock64(), ns0 = globaltimer_ns();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        {
            const uint32_t full0 = leader_addr(&sh->full[0]);      // barriers are 8 bytes apart
            uint32_t it = 0;
            bool ok = true, aligned = p.wave_sync != nullptr;
            for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
                uint32_t mb, nb;
                dense_tile_coords(tile, tiles_m, tiles_n, p.group, mb, nb);
                const int32_t row_a0 = (int32_t)(mb * kDenseTileM + rank * 128);
                const int32_t row_b = (int32_t)(nb * kTileMN + rank * 128);
                // Meet the other producers after the tile's first two stages are on their way, not
                // before: the MMA thread then has work while the slowest producer arrives.
                const uint32_t align_at = p.k_blocks > p.align_at ? p.align_at : 0u;
                for (uint32_t kb = 0; kb < p.k_blocks; kb++, it++) {
                    if (kb == align_at) {
                        if (lane == 0)
                            wave_align(p, tile / n_clusters, n_tiles, n_clusters, aligned);
                        aligned = __shfl_sync(0xffffffffu, aligned ? 1 : 0, 0) != 0;
                    }
                    const uint32_t s = it % kDenseStages, round = it / kDenseStages;
                    if (round > 0 && !warp_wait(&sh->empty[s], (round - 1) & 1)) {
                        if (lane == 0)
                            atomicCAS(p.status, 0u, 0x201u);
                        ok = false;
                        break;
                    }
                    uint8_t *st = smem + (size_t)s * kDenseStageBytes;
                    const int32_t x = (int32_t)(kb * p.k_block_elems);
                    if (elect_one()) {
                        if (rank == 0)
                            mbar_expect_tx(&sh->full[s], 2 * kDenseStageBytes);
                        tma_load_pair_at(st, &tmap_a, x, row_a0, full0 + 8 * s);
                        tma_load_pair_at(st + kHalfTileBytes, &tmap_a, x, row_a0 + 256, full0 + 8 * s);
                        tma_load_pair_at(st + 2 * kHalfTileBytes, &tmap_b, x, row_b, full0 + 8 * s);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA) ----------------
        if (rank == 0) {
            constexpr uint32_t kAFmt = DT == CLPK_DT_BF16 ? kFmtBF16 : DT == CLPK_DT_F16 ? kFmtF16 : DT == CLPK_DT_TF32 ? kFmtTF32
                                     : DT == CLPK_DT_I8 ? kFmtS8 : DT == CLPK_DT_E5M2 ? kFmtE5M2 : kFmtE4M3;
            // the E5M2 variant multiplies e5m2 A by e4m3 B (the pairing the reference's fp8_e5m2 row uses)
            constexpr uint32_t kBFmt = DT == CLPK_DT_E5M2 ? kFmtE4M3 : kAFmt;
            const uint32_t idesc = make_idesc(256, 256, kAFmt, kBFmt, DT == CLPK_DT_I8 ? kAccS32 : kAccF32);
            uint32_t it = 0, tcount = 0;
            bool ok = true;
            for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters, tcount++) {
                if (tcount > 0 && !warp_wait(&sh->tmem_empty, (tcount - 1) & 1)) {
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x202u);
                    break;
                }
                tc_fence_after_sync();
                for (uint32_t kb = 0; kb < p.k_blocks; kb++, it++) {
                    const uint32_t s = it % kDenseStages, round = it / kDenseStages;
                    if (!warp_wait(&sh->full[s], round & 1)) {
                        if (lane == 0)
                            atomicCAS(p.status, 0u, 0x203u);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t base = smem_u32(smem + (size_t)s * kDenseStageBytes);
                    const uint64_t bd = make_smem_desc(base + 2 * kHalfTileBytes, 16, 1024, kSwizzle128B);
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t h = 0; h < 2; h++) {
                            const uint64_t ad = make_smem_desc(base + h * kHalfTileBytes, 16, 1024, kSwizzle128B);
                            const uint32_t d = tmem + h * 256;
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; kk++) {
                                // +32 bytes of K per instruction: +2 in the (>>4) address field
                                if constexpr (DT == CLPK_DT_E4M3 || DT == CLPK_DT_E5M2)
                                    mma2_f8f6f4_ss(d, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                                else if constexpr (DT == CLPK_DT_TF32)
                                    mma2_tf32_ss(d, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                                else if constexpr (DT == CLPK_DT_I8)
                                    mma2_i8_ss(d, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                                else
                                    mma2_f16_ss(d, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                            }
                        }
                        tc_commit_pair(&sh->empty[s], 3);
                    }
                    __syncwarp();
                }
                if (ok && elect_one())
                    tc_commit_pair(&sh->tmem_full, 3);
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue warps ----------------
        // Eight warps: warp w may read TMEM lanes 32 (w % 4) .. +31; the two warps of a lane
        // quarter split each row block's 256 columns in halves (drain_warp_tile).
        const uint32_t q = (uint32_t)(warp & 3);
        const uint32_t col_half = (uint32_t)(warp - 2) >> 2;
        uint8_t *box = staging + (size_t)(warp - 2) * kStagingBytes;
        uint32_t tcount = 0;
        for (uint32_t tile = cluster_id; tile < n_tiles; tile += n_clusters, tcount++) {
            uint32_t mb, nb;
            dense_tile_coords(tile, tiles_m, tiles_n, p.group, mb, nb);
            // warp-uniform verdict: the tcgen05.ld below is warp-aligned
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->tmem_full, tcount & 1) ? 1 : 0)) {
                if (lane == 0)
                    atomicCAS(p.status, 0u, 0x204u);
                break;
            }
            tc_fence_after_sync();
            drain_warp_tile_wide<DT>(tmem + col_half * 128 + ((q * 32) << 16), mb * kDenseTileM + rank * 128 + q * 32,
                                     nb * kTileMN + col_half * 128, box, &tmap_c, p.alpha, &sh->tmem_empty, lane);
        }
        // The staging box must have been read before this CTA's shared memory goes away; the writes themselves
        // complete like any other store before the grid is reported finished, so they are not waited for here
        // (that wait was about a microsecond at the end of every launch).
        if (lane == 0)
            bulk_wait_read<0>();
    }

    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    if (threadIdx.x == 0)
        leave_wave_sync(p);
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.clock) {
        p.clock[0] = clock64() - clk0;
        p.clock[1] = globaltimer_ns() - ns0;
    }
    if (warp == 1)
        tmem_dealloc<2>(tmem, 512);
}

#include "../clpk_gemm_tiles.cuh"
#include "../clpk_gemm_f32.cuh"


// ---------------------------------------------------------------------------------
// NVFP4 GEMM: e2m1 operands, one ue4m3 scale per 16 elements along K
// ---------------------------------------------------------------------------------
//
// Same skeleton as gemm_kernel (2-CTA clusters, TMA ring, one MMA thread, eight epilogue
// warps) with these differences:
//  * 256 x 256 tile per cluster, one accumulator.  K per stage is 256 elements (128 bytes
//    of packed fp4) = four tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X
//    (K = 64), 512 tensor-core cycles.
//  * Every stage also carries scale factors: 2 KiB for this CTA's 128 rows of A
//    and 4 KiB for all 256 columns of B (each CTA of the pair needs B's scales for
//    the whole tile), pre-arranged in global memory in the order tensor memory
//    wants them: per instruction a 512-byte block of 32 rows x 16 bytes, byte
//    (r % 32) * 16 + (r / 32) * 4 + j for row r's j-th factor.  One
//    tcgen05.cp.cta_group::2.32x128b.warpx4 per block copies it from shared to
//    tensor memory in both CTAs (4 columns, replicated in the four lane quarters).
//  * Twelve such copies are needed per stage (six for MXFP4).  The MMA warp issues them itself, in front of the
//    stage's four instructions: tcgen05.cp and tcgen05.mma of one thread run in the order they were issued, so no
//    barrier sits between a stage's factors reaching tensor memory and its multiplies.  (Four dedicated copy warps
//    handing over through an mbarrier were the first design: a stage's copies could start only when the ring's
//    previous pass over that stage had retired -- its tensor-memory columns -- and then queued behind the four
//    stages of instructions issued meanwhile, so the pipe ran dry once per ring: 585 cycles per 512-cycle stage.
//    With the copies in line MXFP4 runs at 513 and NVFP4 at 552: a copy takes about 3 cycles of the pipe, and
//    issuing a stage's seventeen instructions takes the elected lane 304 cycles, eleven 234.)  Writing the factors
//    through registers (tcgen05.st from both CTAs) was
//    tried and is slower: the per-stage cross-CTA mbarrier arrive costs about a microsecond.
//  * Two producer warps per CTA: one loads the A and B tiles (full / empty), one the scale factors (sf_full); both
//    reuse a stage when its instructions have retired (empty).
//  * Tensor memory (256-wide tile): accumulator in columns [0,256), then one 48-column scale area
//    per pipeline stage (16 columns A, 32 columns B).  No room is left for a second
//    accumulator, so a tile's epilogue is not overlapped with the next main loop; the
//    epilogue therefore reads all of its columns and releases tensor memory before it
//    writes anything out (drain_warp_tile_early).  The 128-wide tile (TN = 128) has two
//    128-column accumulators and overlaps the epilogue completely.
//  * MXFP4 (MX = true: kind::mxf4.block_scale.scale_vec::2X, one ue8m0 scale per 32
//    elements) has two factors per row per instruction, so one 32-bit word serves
//    two instructions: the instruction descriptor's scale-factor id picks bytes 0-1
//    or 2-3.  Half the blocks (2 of A + 4 of B per stage), half the copies.
//  * What it costs, in CTA 0's own cycles (clock64 and %globaltimer around the whole kernel,
//    clpk_gemm_last_clock) on 4 clusters at a fixed 1.84 GHz with K from 1024 to 16384: a stage 552 cycles
//    (NVFP4; MXFP4 513) against the 512 of its four instructions -- each scale copy takes about 3 cycles of the
//    pipe -- and a tile about 1 600 more for the hand-over of tensor memory (see drain_warp_tile_wide).  The
//    128-wide tile hides the hand-over but reads A twice as often and is 35 % slower; two N = 128 instructions per K
//    step on the 256-wide tile cost 7 %.  Without effect: an L2 prefetch cursor ahead of the loads (slower), parked
//    mbarrier waits, one polling lane per epilogue warp, raster group widths from 4 to 32, four stages instead of
//    five (3 %), C stored with the L2 evict-first policy.

// rows of a block-scaled operand rounded up to whole 256-row tiles
static inline uint32_t padded_rows(uint32_t rows) { return (rows + 255u) / 256u * 256u; }

constexpr int kNvMaxStages = 6;
constexpr int kNvGemmThreads = 32 * (3 + kEpilogueWarps);                   // operand producer, MMA, 8 epilogue warps, scale producer
constexpr uint32_t kNvSfCol = 256;                             // first scale column: after the accumulator(s)

// TN = width of the cluster tile in columns of C.
//   TN = 256: 256 x 256 tile, ONE accumulator (256 columns) and five 48-column scale areas.  Every operand
//             byte is used for 256 outputs, the least L2 traffic per flop; the epilogue of a tile is exposed.
//   TN = 128: 256 x 128 tile, TWO accumulators (2 x 128 columns) and six 32-column scale areas, 448 columns
//             in all.  The epilogue of tile t drains one accumulator while the main loop of tile t + 1 fills
//             the other; the price is half again as many operand bytes per flop (A is re-read for every 128
//             columns instead of every 256) and instructions half as long.
template <bool MX, int TN> struct BlockScaled {
    static constexpr uint32_t a_blocks = MX ? 2 : 4;            // 512-byte scale blocks of A per stage (per CTA)
    static constexpr uint32_t b_blocks = (MX ? 4 : 8) * TN / 256; // ... of B (all TN columns)
    static constexpr uint32_t blocks = a_blocks + b_blocks;
    static constexpr uint32_t sf_bytes = blocks * 512;
    static constexpr uint32_t sf_per_kblock = MX ? 8 : 16;      // factors per row per 256 elements of K
    static constexpr uint32_t b_rows = TN / 2;                  // rows of B this CTA stages
    static constexpr uint32_t b_tile_bytes = b_rows * kRowBytesK;
    static constexpr uint32_t tile_bytes = kHalfTileBytes + b_tile_bytes;          // A half + this CTA's part of B
    static constexpr uint32_t stage_bytes = tile_bytes + 2048 + 4096 * TN / 256;   // + room for NVFP4's scale blocks
    static constexpr int stages = TN == 256 ? 5 : 6;
    static constexpr uint32_t n_acc = 256 / TN;                 // accumulators in tensor memory
    static constexpr uint32_t sf_cols = 16 + TN / 8;            // tensor-memory columns per stage: 16 for A, 4 per 128 columns of B per instruction
    static constexpr uint32_t b_cols_per_instr = TN / 32;       // scale columns of B per instruction (NVFP4)
    static constexpr size_t smem_bytes = (size_t)stages * stage_bytes + kEpilogueWarps * kStagingBytes + 512 + 1024;
    static_assert(kNvSfCol + stages * sf_cols <= 512, "tensor memory columns");
    static_assert(stages <= kNvMaxStages, "barrier arrays");
};

struct NvGemmSmem {
    uint64_t full[kNvMaxStages];     // operand tiles of both CTAs landed (leader's barrier)
    uint64_t sf_full[kNvMaxStages];  // scale factors of both CTAs landed (leader's barrier)
    uint64_t empty[kNvMaxStages];    // the stage's MMAs retired (both CTAs)
    uint64_t tmem_full[2];           // per accumulator
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
};
static_assert(sizeof(NvGemmSmem) <= 512, "NvGemmSmem");

// Row-major scale bytes [rows][k / block] of both operands -> 512-byte blocks in tensor-memory order, one 32-bit word
// (four factors) per row per block.  NVFP4: 16 factors per row per stage = 4 words; MXFP4: 8 factors = 2 words.
// A's blocks are ordered [rows/128][k/256][words]; B's [rows/256][k/256][words][2] for the 256-wide tile (b_pairs),
// like A's for the 128-wide one.  Rows at and beyond an operand's `rows` (it is padded up to whole tiles) get zero
// factors: their elements arrive as zeros from the operand's tensor map, and zero times any finite factor is zero.
//
// One warp takes 128 rows x one stage: a lane loads the stage's words of rows r, r + 32, r + 64, r + 96 and holds
// their transpose, one 16-byte piece of every block.  Eight neighbouring stages are one CTA, so that a row's 128-byte
// line is read once.  The kernel is latency: launched with the programmatic attribute like the GEMM behind it, so that
// both set up under the tail of what precedes.  NVFP4 one-call GEMM, device time at 2048^3 / 4096^3: 20.4 / 55.3 us with
// one launch per operand through shared memory, 10.9 / 37.5 now, 8.1 / 31.2 with the scales already packed.
template <int WORDS>
__global__ void __launch_bounds__(256) pack_scales_kernel(PackOperand oa, PackOperand ob, uint32_t kblocks, uint32_t b_pairs)
{
    griddep_wait();
    griddep_launch_dependents();
    const uint32_t lane = threadIdx.x & 31, kgroups = (kblocks + 7) / 8;
    const uint32_t kb = blockIdx.x % kgroups * 8 + (threadIdx.x >> 5);
    uint32_t group = blockIdx.x / kgroups;
    const bool is_b = group >= oa.row_groups;
    const PackOperand &op = is_b ? ob : oa;
    group -= is_b ? oa.row_groups : 0;
    if (kb >= kblocks)
        return;
    uint32_t w[4][WORDS];
#pragma unroll
    for (int i = 0; i < 4; i++)
        load_scale_words<WORDS>(op, group * 128 + i * 32 + lane, kb, kblocks, w[i]);
#pragma unroll
    for (int j = 0; j < WORDS; j++)
        // block byte (r % 32) * 16 + (r / 32) * 4 of row r
        reinterpret_cast<uint4 *>(op.out)[scale_block<WORDS>(group, kb, j, kblocks, is_b && b_pairs) * 32 + lane] = make_uint4(w[0][j], w[1][j], w[2][j], w[3][j]);
}

template <bool MX, int TN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kNvGemmThreads)
    gemm_block_scaled_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                     const __grid_constant__ CUtensorMap tmap_c, GemmParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    using BS = BlockScaled<MX, TN>;
    constexpr int kNvStages = BS::stages;
    constexpr uint32_t kNvStageBytes = BS::stage_bytes, kNvSfColsPerStage = BS::sf_cols;
    uint8_t *staging = smem + (size_t)kNvStages * kNvStageBytes;                 // one 4 KiB box per epilogue warp
    NvGemmSmem *sh = reinterpret_cast<NvGemmSmem *>(staging + kEpilogueWarps * kStagingBytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t cluster_id = blockIdx.x >> 1;
    const uint32_t n_clusters = gridDim.x >> 1;
    const uint32_t tiles_m = (p.m + kTileMN - 1) / kTileMN, tiles_n = (p.n + TN - 1) / TN;
    const uint32_t n_tiles = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kNvStages; s++) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->sf_full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int acc = 0; acc < 2; acc++) {
            mbar_init(&sh->tmem_full[acc], 1);
            mbar_init(&sh->tmem_empty[acc], 2 * kEpilogueWarps);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_sfa);
        tma_prefetch_desc(&tmap_sfb);
        tma_prefetch_desc(&tmap_c);
    }
    if (warp == 1)
        tmem_alloc<2>(&sh->tmem_base, 512);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    tc_fence_after_sync();
    const uint32_t tmem = sh->tmem_base;
    join_previous_launch(p);
    const unsigned long long clk0 = clock64(), ns0 = globaltimer_ns();
    constexpr int kScaleProducerWarp = 2 + kEpilogueWarps;

    if (warp == 0) {
        // ---------------- operand producer (both CTAs): A and B tiles ----------------
        // The scale factors have a producer warp of their own (below): their copies on to tensor
        // memory can then start when 6 KiB have landed instead of 70.
        const uint32_t full0 = leader_addr(&sh->full[0]);          // barriers are 8 bytes apart
        uint32_t it = 0;
        bool ok = true, aligned = p.wave_sync != nullptr;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            uint32_t mb, nb;
            dense_tile_coords(tile, tiles_m, tiles_n, p.group, mb, nb);
            const int32_t row_a = (int32_t)(mb * kTileMN + rank * 128);
            const int32_t row_b = (int32_t)(nb * TN + rank * BS::b_rows);
            const uint32_t align_at = p.k_blocks > p.align_at ? p.align_at : 0u;
            for (uint32_t kb = 0; kb < p.k_blocks; kb++, it++) {
                if (kb == align_at) {
                    if (lane == 0)
                        wave_align(p, tile / n_clusters, n_tiles, n_clusters, aligned);
                    aligned = __shfl_sync(0xffffffffu, aligned ? 1 : 0, 0) != 0;
                }
                const uint32_t s = it % kNvStages, round = it / kNvStages;
                if (round > 0 && !warp_wait(&sh->empty[s], (round - 1) & 1)) {
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x211u);
                    ok = false;
                    break;
                }
                uint8_t *st = smem + (size_t)s * kNvStageBytes;
                const int32_t x = (int32_t)(kb * kRowBytesK);
                if (elect_one()) {
                    if (rank == 0)
                        mbar_expect_tx(&sh->full[s], 2 * BS::tile_bytes);
                    tma_load_pair_at(st, &tmap_a, x, row_a, full0 + 8 * s);
                    tma_load_pair_at(st + kHalfTileBytes, &tmap_b, x, row_b, full0 + 8 * s);
                }
                __syncwarp();
            }
        }
    } else if (warp == kScaleProducerWarp) {
        // ---------------- scale-factor producer (both CTAs) ----------------
        // The stage's scale area in shared memory (and its tensor-memory columns) are free again when the previous
        // round's instructions on the stage have retired: the copies run in front of them in the same queue.
        const uint32_t sf_full0 = leader_addr(&sh->sf_full[0]);
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            uint32_t mb, nb;
            dense_tile_coords(tile, tiles_m, tiles_n, p.group, mb, nb);
            const uint32_t sfa_block0 = (mb * 2 + rank) * p.k_blocks * BS::a_blocks;
            const uint32_t sfb_block0 = nb * p.k_blocks * BS::b_blocks;
            for (uint32_t kb = 0; kb < p.k_blocks; kb++, it++) {
                const uint32_t s = it % kNvStages, round = it / kNvStages;
                if (round > 0 && !warp_wait(&sh->empty[s], (round - 1) & 1)) {
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x216u);
                    ok = false;
                    break;
                }
                uint8_t *sf = smem + (size_t)s * kNvStageBytes + BS::tile_bytes;
                if (elect_one()) {
                    if (rank == 0)
                        mbar_expect_tx(&sh->sf_full[s], 2 * BS::sf_bytes);
                    tma_load_pair_at(sf, &tmap_sfa, 0, (int32_t)(sfa_block0 + kb * BS::a_blocks), sf_full0 + 8 * s);
                    tma_load_pair_at(sf + BS::a_blocks * 512, &tmap_sfb, 0, (int32_t)(sfb_block0 + kb * BS::b_blocks),
                                     sf_full0 + 8 * s);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA) ----------------
        // The whole warp runs the loop and waits; one elected lane issues.  Descriptors and
        // addresses are then warp-uniform values, which is what tcgen05 instructions take:
        // with the loop inside `if (lane == 0)` every operand had to be moved over from a
        // per-thread register, and an instruction cost its thread about 110 cycles.
        if (rank == 0) {
            // MXFP4: instruction kk reads bytes 0-1 (id 0) or 2-3 (id 2) of word kk / 2
            const uint32_t idesc = make_idesc_block_scaled(256, TN, kFmtE2M1, kFmtE2M1, MX ? 1u : 0u, 0, 0);
            const uint32_t idesc_hi = make_idesc_block_scaled(256, TN, kFmtE2M1, kFmtE2M1, 1u, 2, 2);
            uint32_t it = 0, tcount = 0;
            bool ok = true;
            for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters, tcount++) {
                // accumulator `acc` is free again when the epilogue of its previous tile has read it out
                const uint32_t acc = tcount % BS::n_acc, use = tcount / BS::n_acc;
                if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&sh->tmem_empty[acc], (use - 1) & 1) ? 1 : 0)) {
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x212u);
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d_t = tmem + acc * TN;
                for (uint32_t kb = 0; kb < p.k_blocks; kb++, it++) {
                    const uint32_t s = it % kNvStages, round = it / kNvStages;
                    // the scale factors usually arrive first (6 KiB against 64): wait for them, then the tiles
                    const bool landed = mbar_wait(&sh->sf_full[s], round & 1) && mbar_wait(&sh->full[s], round & 1);
                    if (!__all_sync(0xffffffffu, landed ? 1 : 0)) {
                        if (lane == 0)
                            atomicCAS(p.status, 0u, 0x213u);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t base = smem_u32(smem + (size_t)s * kNvStageBytes);
                    const uint32_t sfa_t = tmem + kNvSfCol + s * kNvSfColsPerStage, sfb_t = sfa_t + 16;
                    const uint64_t ad = make_smem_desc(base, 16, 1024, kSwizzle128B);
                    const uint64_t bd = make_smem_desc(base + kHalfTileBytes, 16, 1024, kSwizzle128B);
                    if (elect_one()) {
                        // the stage's scale factors go to tensor memory in front of its instructions, in the same queue:
                        // 512-byte blocks, A's (4 columns each, from column 0), then B's (from column 16)
                        const uint32_t sf_s = base + BS::tile_bytes;
#pragma unroll
                        for (uint32_t blk = 0; blk < BS::blocks; blk++) {
                            const uint32_t col = blk < BS::a_blocks ? 4 * blk : 16 + 4 * (blk - BS::a_blocks);
                            tmem_cp_32x128b_warpx4<2>(sfa_t + col, make_smem_desc(sf_s + blk * 512, 16, 128, kSwizzleNone));
                        }
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; kk++) {
                            if constexpr (MX)
                                mma2_mxf4_bs(d_t, ad + 2 * kk, bd + 2 * kk, (kk & 1) ? idesc_hi : idesc, sfa_t + 4 * (kk / 2),
                                             sfb_t + BS::b_cols_per_instr * (kk / 2), (kb | kk) ? 1u : 0u);
                            else
                                mma2_nvf4_bs(d_t, ad + 2 * kk, bd + 2 * kk, idesc, sfa_t + 4 * kk, sfb_t + BS::b_cols_per_instr * kk,
                                             (kb | kk) ? 1u : 0u);
                        }
                        tc_commit_pair(&sh->empty[s], 3);
                    }
                    __syncwarp();
                }
                if (ok && elect_one())
                    tc_commit_pair(&sh->tmem_full[acc], 3);
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue warps: one row block, tensor memory released before the stores ----------------
        const uint32_t q = (uint32_t)(warp & 3);
        const uint32_t col_half = (uint32_t)(warp - 2) >> 2;
        uint8_t *box = staging + (size_t)(warp - 2) * kStagingBytes;
        uint32_t tcount = 0;
        for (uint32_t tile = cluster_id; tile < n_tiles; tile += n_clusters, tcount++) {
            uint32_t mb, nb;
            dense_tile_coords(tile, tiles_m, tiles_n, p.group, mb, nb);
            const uint32_t acc = tcount % BS::n_acc, use = tcount / BS::n_acc;
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->tmem_full[acc], use & 1) ? 1 : 0)) {
                if (lane == 0)
                    atomicCAS(p.status, 0u, 0x214u);
                break;
            }
            tc_fence_after_sync();
            drain_warp_tile_early<TN / 128>(tmem + acc * TN + col_half * (TN / 2) + ((q * 32) << 16), mb * kTileMN + rank * 128 + q * 32,
                                            nb * TN + col_half * (TN / 2), box, &tmap_c, p.alpha, &sh->tmem_empty[acc], lane);
        }
        // The staging box must have been read before this CTA's shared memory goes away; the writes themselves
        // complete like any other store before the grid is reported finished, so they are not waited for here
        // (that wait was about a microsecond at the end of every launch).
        if (lane == 0)
            bulk_wait_read<0>();
    }

    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    if (threadIdx.x == 0)
        leave_wave_sync(p);
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.clock) {
        p.clock[0] = clock64() - clk0;
        p.clock[1] = globaltimer_ns() - ns0;
    }
    if (warp == 1)
        tmem_dealloc<2>(tmem, 512);
}

// ---- host side -----------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static int get_encode_fn(EncodeTiledFn *out)
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        CLPK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres));
        if (qres != cudaDriverEntryPointSuccess || !sym) {
            set_error("cuTensorMapEncodeTiled is not available from this driver");
            return CLPK_ERR_CUDA;
        }
        fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    *out = fn;
    return CLPK_OK;
}

// Row-major [rows][row_bytes] operand, box = box_rows (128 unless said otherwise) x 128 bytes, 128-byte swizzle.
static int make_operand_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows = 128)
{
    EncodeTiledFn enc;
    int rc = get_encode_fn(&enc);
    if (rc != CLPK_OK)
        return rc;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {kRowBytesK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return CLPK_ERR_CUDA;
    }
    return CLPK_OK;
}


// C [m][n] row-major for the epilogue's stores: box = 32 rows x 128 bytes, 128-byte swizzle; `chunk_box`: 32 rows x
// 32 columns, which are 64 bytes (64-byte swizzle) of a 16-bit output.
static int make_output_map(CUtensorMap *map, void *base, uint64_t m, uint64_t n, int dtype, bool chunk_box = false)
{
    EncodeTiledFn enc;
    int rc = get_encode_fn(&enc);
    if (rc != CLPK_OK)
        return rc;
    const bool wide = dtype == CLPK_DT_TF32 || dtype == CLPK_DT_I8;
    const CUtensorMapDataType type = dtype == CLPK_DT_TF32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : dtype == CLPK_DT_I8 ? CU_TENSOR_MAP_DATA_TYPE_INT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint32_t elem = wide ? 4 : 2;
    const cuuint64_t dims[2] = {n, m};
    const cuuint64_t strides[1] = {n * elem};
    const cuuint32_t box[2] = {chunk_box ? kTilesChunk : 128 / elem, 32};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, type, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     chunk_box && elem == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (output) failed with CUresult %d", (int)r);
        return CLPK_ERR_CUDA;
    }
    return CLPK_OK;
}

// Packed scale factors: rows of 512 bytes (128 x u32); a box is `rows_per_box` consecutive rows.
static int make_scale_map(CUtensorMap *map, const void *base, uint64_t n_rows, uint32_t rows_per_box)
{
    EncodeTiledFn enc;
    int rc = get_encode_fn(&enc);
    if (rc != CLPK_OK)
        return rc;
    const cuuint64_t dims[2] = {128, n_rows};
    const cuuint64_t strides[1] = {512};
    const cuuint32_t box[2] = {128, rows_per_box};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (scales) failed with CUresult %d", (int)r);
        return CLPK_ERR_CUDA;
    }
    return CLPK_OK;
}


// B's packed scale factors for gemm_tiles_kernel: [rows / 256 * K blocks * words][half of the 256 rows][512 bytes]; a box
// is one K block's words of one half, or of both.
static int make_scale_map_b(CUtensorMap *map, const void *base, uint64_t n_rows, uint32_t words, uint32_t halves)
{
    EncodeTiledFn enc;
    int rc = get_encode_fn(&enc);
    if (rc != CLPK_OK)
        return rc;
    const cuuint64_t dims[3] = {128, 2, n_rows / 2};
    const cuuint64_t strides[2] = {512, 1024};
    const cuuint32_t box[3] = {128, halves, words};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (scales) failed with CUresult %d", (int)r);
        return CLPK_ERR_CUDA;
    }
    return CLPK_OK;
}

constexpr size_t kGemmSmemBytes = (size_t)kDenseStages * kDenseStageBytes + kEpilogueWarps * kStagingBytes + sizeof(DenseSmem) + 1024;

// One pair of wave counters per launch, from a ring of 32 per device so that launches on different streams do not share
// one; zero between launches.  The slot is chosen by the host, from one process-wide index: 32 launches later, on whatever
// device, it is handed out again, and a launch captured in a graph keeps its slot for every replay.  So two running
// kernels can share a slot -- eager launches only with more than 32 of them in flight, a replay with any other launch.
// That costs alignment, not correctness: whoever does not see its wave complete within 40 us stops taking part, a wave
// that is counted too soon runs unaligned, and the slot is zero again when all its kernels have ended (every CTA arrives
// before it leaves, and the grids of a device are all the same size, so the last CTA of all clears it).
constexpr int kSyncSlots = 32;
__device__ unsigned int g_wave_sync[kSyncSlots][2];
static std::atomic<unsigned> g_next_sync_slot{0};
static thread_local int g_last_aligned = -1;
// {SM cycles, nanoseconds} CTA 0 of the last GEMM launch on this device ran for (both tensor kernels write it).
__device__ unsigned long long g_gemm_clock[2];

// Launches a persistent cluster kernel whose last parameter is GemmParams, with a wave counter when the alignment is on.
template <typename Kernel, typename... Maps>
static int launch_persistent(Kernel kernel, const char *what, int threads, size_t smem, cudaStream_t s, GemmParams p,
                             uint32_t n_tiles, const Maps &...maps)
{
    CLPK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int grid = (num_sms() / 2) * 2;
    p.wave_sync = nullptr;
    CLPK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&p.clock), g_gemm_clock));
    // nothing to keep in step in the first two waves: small problems skip the counter
    const bool worth_aligning = n_tiles > 2u * (uint32_t)(grid / 2) * p.align_period;
    if (worth_aligning && tuning(CLPK_TUNE_GEMM_NO_ALIGN) != 1) {
        unsigned int *base = nullptr;
        CLPK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&base), g_wave_sync));
        p.wave_sync = base + 2 * (g_next_sync_slot.fetch_add(1) % kSyncSlots);
    }
    g_last_aligned = p.wave_sync ? 1 : 0;
    cudaLaunchConfig_t plain = {};
    plain.gridDim = dim3((unsigned)grid);
    plain.blockDim = dim3((unsigned)threads);
    plain.dynamicSmemBytes = smem;
    plain.stream = s;
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = tuning(CLPK_TUNE_GEMM_NO_PDL) == 1 ? 0 : 1;
    plain.attrs = pdl;
    plain.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&plain, kernel, maps..., p);
    if (e != cudaSuccess)
        return cuda_fail(e, what);
    return CLPK_OK;
}

// How gemm_tiles_kernel splits a problem; tn = 0: leave it to gemm_kernel or gemm_block_scaled_kernel.
struct TilesPlan {
    uint32_t tn, splits;
    uint32_t row_blocks = 1;            // 2: 512 x tn tiles
};

// The plan is the cheapest by a cost estimate in microseconds, fitted to timed launches of both kernels: 2500 for 120
// shapes with M and N from 64 to 14000, K from 256 to 16000 in the six dense types, 300 for 90 block-scaled ones, every
// tile width and split of each (residuals 13 and 6 %; the chosen plans are 1 % slower than the fastest in the geometric
// mean, 19 % at worst).  With W = TN / 256 and T the time to fetch what all SMs load for one K block of 128 bytes:
//   gemm_kernel               3.6 + waves * (0.57 per K block of a 512 x 256 tile + 2.9), and 4 for the producers'
//                             meetings when there are more than two waves
//   gemm_tiles_kernel, dense  3.9 + waves * (K blocks * (0.118 to issue a block + 0.175 W for its instructions + T at
//                             54 TB/s) + 1.1 W of epilogue) and, split, 1 + 4.3 W per exchanged share of the tile
//   gemm_block_scaled_kernel  4.0 + waves * (K blocks * (0.275 + T at 43 TB/s) + 0.7)
//   gemm_tiles_kernel, FP4    3.3 + waves * (K blocks * (0.25 + 0.06 W + T at 62 TB/s) + 1.4 W) and the same exchange
//   gemm_tiles_kernel, 512    4.75 + waves * (K blocks * (0.157 + 0.344 W + T at 106 TB/s) + 1.2 W of epilogue, 3.2 W from
//                             tn = 160 on, where tensor memory holds one accumulator); from 24000 launches, residual 6 %.
//                             Not used beyond four waves, narrow ones not beyond two (e4m3 13065 x 1248 x 464, four waves
//                             of tn = 128: 14.6 us in large tiles, 18.6 in these), and only where gemm_kernel would be taken: 77922
//                             random shapes that take it are 1.15 times as fast in the geometric mean.  Operand rows that are
//                             an odd multiple of 16 bytes, where a row's 128 bytes lie in five 32-byte sectors instead of
//                             four, gain less (1.11 against 1.20 times), and of them tn = 96 was slower from six blocks on
//                             (e4m3 270 x 13928 x 784: 11.6 us in large tiles, 12.9 in these; 22 of 50, and none of 600 others),
//                             so narrow tiles are left to short sums there.  77 wider ones, all but one with such rows, were
//                             timed 2 to 5 % slower once and most of them no slower again.  Against
//                             the 256-row tiles the estimate is not sharp enough (228 of 831 more than 2 % slower)
// Splits of 2 and 4 are clusters of 4 and 8 CTAs, of which the chip holds 33 and 15 at a time.  From the fifth wave of
// 512 x 256 tiles on (16384 x 16384 x 256: 140 against 142 us) and the third of block-scaled ones the large tiles'
// smaller operand traffic wins at every K; an FP4 tile 256 wide that is not split is the large kernel's own.  An FP4 A of a few
// rows, whose lines more than half the pairs ask for at once, costs them 0.04 a block more, up to eight rows 0.15 (mxf4
// 9 x 9336 x 14592: 32 us in 128-wide tiles, 26 in large ones; of 1400 shapes with few rows 87 were more than 3 % slower
// than in large tiles, at worst 1.31 times, and with the term 17, at worst 1.10).  Where the scales are arranged on the way it
// does not show (nvf4 5 x 5632 x 3840: 10.2 us in 128-wide tiles, 11.4 in large ones; 35 shapes with up to 48 rows 0.835 and
// 0.832 of the time before), so `arranged`: FP4 whose scales lie in the workspace already.
// `sectors`: rows of the operands are whole 32-byte sectors.
static TilesPlan plan_tiles(uint32_t m, uint32_t n, uint32_t k_blocks, bool sectors, bool fp4, bool arranged)
{
    const uint32_t pairs = (uint32_t)num_sms() / 2;
    auto ceil_div = [](uint32_t a, uint32_t b) { return (a - 1) / b + 1; };
    // bytes that `clusters` clusters of `splits` pairs load for one K block of a 256 x tn tile each
    auto fetched = [&](uint64_t clusters, uint32_t splits, uint32_t tn) {
        return (float)clusters * splits * ((m < 256 ? m : 256) + (n < tn ? n : tn)) * kRowBytesK;
    };
    const uint64_t big_tiles = (uint64_t)ceil_div(m, fp4 ? kTileMN : kDenseTileM) * ceil_div(n, kTileMN);
    TilesPlan plan = {0, 1};
    if (pairs == 0 || big_tiles > (fp4 ? 2ull : 4ull) * pairs)
        return plan;
    const float big_waves = (float)((big_tiles - 1) / pairs + 1);
    const float big = fp4 ? 4.0f + big_waves * (k_blocks * (0.275f + fetched(big_tiles < pairs ? big_tiles : pairs, 1, 256) / 43.2e6f) + 0.7f)
                          : 3.6f + (big_waves > 2 ? 4.0f : 0.0f) + big_waves * (k_blocks * 0.57f + 2.9f);
    float best = 0.97f * big;
    const float launch = fp4 ? 3.3f : 3.9f, issue = fp4 ? 0.25f : 0.118f, wide_issue = fp4 ? 0.06f : 0.175f;
    const float rate = fp4 ? 62.4e6f : 53.8e6f, drain = fp4 ? 1.36f : 1.14f;
    for (uint32_t splits = 1; splits <= 4; splits *= 2) {
        const uint32_t resident = splits == 1 ? pairs : splits == 2 ? pairs * 33 / 74 : pairs * 15 / 74;
        if (resident == 0 || k_blocks < splits)
            break;
        // scale factors come in blocks of 128 columns, of which a 64-wide tile uses half
        for (uint32_t tn = fp4 ? 64 : 32; tn <= (fp4 && splits == 1 ? 128u : 256u); tn = fp4 ? 2 * tn : tn + 32) {
            const uint64_t tiles = (uint64_t)ceil_div(m, kTilesM) * ceil_div(n, tn);
            const float waves = (float)((tiles - 1) / resident + 1), wide = (float)tn / 256.0f;
            float block = issue + wide_issue * wide + fetched(tiles < resident ? tiles : resident, splits, tn) / rate;
            if (arranged && splits == 1 && m <= 48 && tiles > pairs * 40 / 74)
                block += m <= 8 ? 0.15f : 0.04f;
            float t = launch + waves * (ceil_div(k_blocks, splits) * block + drain * wide);
            if (splits > 1)
                t += waves * (1.0f + 4.3f * wide * (splits - 1) / splits);
            if (t < best) {
                best = t;
                plan = {tn, splits};
            }
        }
    }
    // Where the 512 x 256 tiles are left over, narrower ones of 512 rows may fill the chip better.
    if (!fp4 && plan.tn == 0) {
        for (uint32_t tn = 64; tn < 256; tn += 32) {                      // 32 was cheapest for none of 40 million shapes
            const uint64_t tiles = (uint64_t)ceil_div(m, kDenseTileM) * ceil_div(n, tn);
            if (tiles > (tn >= 192 ? 4ull : 2ull) * pairs || (tn <= 128 && k_blocks > 5 && !sectors))
                continue;
            const float waves = (float)((tiles - 1) / pairs + 1), wide = (float)tn / 256.0f;
            const float loaded = (float)(tiles < pairs ? tiles : pairs) * ((m < kDenseTileM ? m : kDenseTileM) + (n < tn ? n : tn)) * kRowBytesK;
            const float t = 4.75f + waves * (k_blocks * (0.157f + 0.344f * wide + loaded / 105.6e6f) + (tn > 128 ? 3.2f : 1.2f) * wide);
            if (t < best) {
                best = t;
                plan = {tn, 1, 2};
            }
        }
    }
    return plan;
}

// bits of an element of the tcgen05 kinds, 0 for anything else
static uint32_t tensor_elem_bits(int dtype)
{
    switch (dtype) {
    case CLPK_DT_BF16:
    case CLPK_DT_F16:  return 16;
    case CLPK_DT_TF32: return 32;
    case CLPK_DT_E4M3:
    case CLPK_DT_E5M2:
    case CLPK_DT_I8:   return 8;
    case CLPK_DT_MXF4:
    case CLPK_DT_NVF4: return 4;
    default:           return 0;
    }
}

static uint32_t k_blocks_of(uint32_t k, uint32_t elem_bits) { return (uint32_t)(((uint64_t)k * elem_bits / 8 + kRowBytesK - 1) / kRowBytesK); }

// What clpk_gemm does with a problem of a tcgen05 kind; the GEMM_FP4_TILE knob's forced tiles are the large kernel's.
static TilesPlan gemm_plan(uint32_t m, uint32_t n, uint32_t k, uint32_t elem_bits, bool arranged)
{
    const bool fp4 = elem_bits == 4;
    if (fp4 && tuning(CLPK_TUNE_GEMM_FP4_TILE) > 0)
        return {0, 1};
    return plan_tiles(m, n, k_blocks_of(k, elem_bits), (uint64_t)k * elem_bits % 256 == 0, fp4, arranged);
}

static PackOperand pack_operand(const void *in, uint8_t *out, uint32_t rows, uint32_t words)
{
    return {static_cast<const uint32_t *>(in), reinterpret_cast<uint32_t *>(out), rows, padded_rows(rows) / 128,
            (uintptr_t)in % (words * 4) == 0 ? 1u : 0u};
}

// FP4 with row-major scales: the tiles in which gemm_tiles_kernel arranges them on the way (kRaw), tn = 0: in a launch of their own.
// That launch costs about 4 us in front of the product; on the way NVFP4's cost 0.1 us a K block, which their 16 bytes a row
// have the L1 look up, and MXFP4's nothing that shows.  So: up to four waves of 256 x 256 tiles, beyond the first one NVFP4 sums only as
// long as those 4 us allow, and where its words are loaded singly in the first one too.  Device time against the launch in front:
// NVFP4 2048^3 13.4 -> 9.3 us, 1024 x 1024 x 2048 8.5 -> 7.4, 16384 x 256 x 2048 14.5 -> 9.4, 2048 x 2048 x 8192 22.4 -> 20.4, MXFP4 17.2 ->
// 11.7 at 2048 x 2048 x 4096; random shapes 0.82 below one wave (worst 1.02), 0.88 up to two, 0.93 up to four (beyond: 1.03;
// NVFP4 with 16 K blocks and more up to four waves 0.95 to 1.06, from unaligned addresses 1.19).
static TilesPlan raw_scales_plan(const clpk_gemm_args_t *a, const PackOperand &sa, const PackOperand &sb)
{
    const uint64_t tiles = (uint64_t)((a->m - 1) / kTileMN + 1) * ((a->n - 1) / kTileMN + 1), pairs = (uint64_t)num_sms() / 2;
    if (pairs == 0 || tiles > 4 * pairs || tuning(CLPK_TUNE_GEMM_FP4_TILE) > 0)
        return {0, 1};
    const uint64_t waves = (tiles - 1) / pairs + 1;
    if (a->dtype == CLPK_DT_NVF4 && waves * (a->k / 256) > 40 && (waves > 1 || !sa.vector || !sb.vector))
        return {0, 1};
    TilesPlan plan = gemm_plan(a->m, a->n, a->k, 4, false);
    if (plan.tn == 0)
        plan.tn = kTileMN;              // the large tiles, by gemm_tiles_kernel
    return plan;
}

// CTAs in clusters of `cluster`, behind the kernel before them
template <typename Maps, typename Params>
static int launch_clusters(void (*kernel)(Maps, Params), const char *what, uint32_t ctas, int threads, size_t smem, uint32_t cluster, cudaStream_t s,
                           const Maps &maps, const Params &p)
{
    CLPK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTilesSmemMax));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = tuning(CLPK_TUNE_GEMM_NO_PDL) == 1 ? 0 : 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    g_last_aligned = 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, maps, p);
    return e == cudaSuccess ? CLPK_OK : cuda_fail(e, what);
}

// sa, sb: where the arranged scale factors lie (block-scaled kinds), and kRaw: where they come from
template <int DT, uint32_t kRowBlocks = 1, bool kRaw = false>
static int launch_tiles(const clpk_gemm_args_t *a, const CUtensorMap &ta, uint64_t row_bytes, uint32_t k_blocks, TilesPlan plan, cudaStream_t s,
                        const PackOperand &sa = {}, const PackOperand &sb = {})
{
    TilesMapsOf<DT, kRaw> maps;
    maps.a = ta;
    int rc = make_operand_map(&maps.b, a->d_b, a->n, row_bytes, plan.tn / 2);
    if (rc != CLPK_OK)
        return rc;
    rc = make_output_map(&maps.c, a->d_c, a->m, a->n, DT, true);
    if (rc != CLPK_OK)
        return rc;
    if constexpr (kRaw) {
        maps.sa = sa;
        maps.sb = sb;
    } else if constexpr (TilesKind<DT>::fp4) {
        constexpr uint32_t words = TilesKind<DT>::words;
        rc = make_scale_map(&maps.sfa, sa.out, (uint64_t)padded_rows(a->m) / 128 * k_blocks * words, words);
        if (rc != CLPK_OK)
            return rc;
        rc = make_scale_map_b(&maps.sfb, sb.out, (uint64_t)padded_rows(a->n) / 128 * k_blocks * words, words, (plan.tn + 127) / 128);
        if (rc != CLPK_OK)
            return rc;
    }
    TilesParams p;
    p.tiles_m = (a->m - 1) / (kTilesM * kRowBlocks) + 1;
    p.tiles_n = (a->n + plan.tn - 1) / plan.tn;
    p.group = tuning(CLPK_TUNE_GEMM_GROUP) > 0 ? (uint32_t)tuning(CLPK_TUNE_GEMM_GROUP) : 8;
    p.k_blocks = k_blocks;
    p.tn = plan.tn;
    p.splits = plan.splits;
    p.alpha = a->alpha;
    p.status = a->d_status;
    const uint32_t n_tiles = p.tiles_m * p.tiles_n, pairs = (uint32_t)num_sms() / 2;
    const uint32_t clusters = plan.splits > 1 ? n_tiles : (n_tiles < pairs ? n_tiles : pairs);
    constexpr size_t fixed = kEpilogueWarps * kStagingBytes + sizeof(TilesSmem) + 1024;
    static_assert(!kRaw || ((kTilesSmemMax - fixed) / (tiles_block_bytes(256) + tiles_sf_bytes(256)) >= 5 &&
                            (kTilesSmemMax - fixed) / (tiles_block_bytes(128) + tiles_sf_bytes(128)) >= 6), "the stages that tiles_arrange_scales counts on");
    // two K blocks per stage halve the hand-overs (0.195 -> 0.137 us per block at TN = 32), but from TN = 160 on leave
    // too few stages (2048^3 bf16 at TN = 192: 19.3 -> 20.7 us)
    constexpr bool fp4 = TilesKind<DT>::fp4;
    p.kps = plan.tn <= 128 && kRowBlocks == 1 && !fp4 ? 2 : 1;
    const uint32_t stage_bytes = p.kps * tiles_block_bytes(plan.tn, kRowBlocks) + (fp4 ? tiles_sf_bytes(plan.tn) : 0);
    p.stages = (uint32_t)((kTilesSmemMax - fixed) / stage_bytes);
    const uint32_t most = fp4 ? 256 / tiles_sf_cols(plan.tn) : kTilesMaxStages;      // scale factors: 256 tensor-memory columns
    if (p.stages > most)
        p.stages = most;
    p.tmem_cols = fp4 ? 512 : 32;
    while (p.tmem_cols < (n_tiles > clusters && (kRowBlocks == 1 || plan.tn <= 128) ? 2 : 1) * kRowBlocks * plan.tn)
        p.tmem_cols *= 2;
    CLPK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&p.clock), g_gemm_clock));
    const size_t smem = p.stages * stage_bytes + fixed;
    return launch_clusters(gemm_tiles_kernel<DT, kRowBlocks, kRaw>, "gemm_tiles", clusters * 2 * plan.splits, tiles_threads(kRaw), smem, 2 * plan.splits, s, maps, p);
}

template <int DT>
static int launch_dense_tiles(const clpk_gemm_args_t *a, const CUtensorMap &ta, uint64_t row_bytes, uint32_t k_blocks, TilesPlan plan, cudaStream_t s)
{
    return plan.row_blocks == 2 ? launch_tiles<DT, 2>(a, ta, row_bytes, k_blocks, plan, s) : launch_tiles<DT>(a, ta, row_bytes, k_blocks, plan, s);
}

template <int DT>
static int launch_gemm(const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tc, const GemmParams &p, cudaStream_t s)
{
    const uint32_t n_tiles = ((p.m + kDenseTileM - 1) / kDenseTileM) * ((p.n + kTileMN - 1) / kTileMN);
    return launch_persistent(gemm_kernel<DT>, "gemm", kGemmThreads, kGemmSmemBytes, s, p, n_tiles, ta, tb, tc);
}

// TN and K ranges of gemm_f32_kernel; tn = 0: leave it to the kernels of simt_gemm.cu.  Like plan_tiles the cheapest by an
// estimate in microseconds, from timed launches of every width and split: with W = TN / 256
//   5.0 + waves * (chunks of 32 per range * max(0.44, 0.22 + 0.92 W) + 5 W of epilogue) and, split, 1 + 7 W per exchange.
// A chunk is what the converters and the turns of the accumulators take; its instructions alone would be 0.22 to 0.46.  The
// CUDA-core kernels keep what they are estimated to do as fast, sums of few chunks and products of a few tiles, whose
// launch is shorter (688 x 140 x 268: 7.4 us against 9.0; 64 x 64 x 16384 57 against 62).  Beyond 2^28 elements of K, or
// 2^31 rows, coordinates would not fit a tensor map's 32 bits.
static TilesPlan plan_f32(uint32_t m, uint32_t n, uint32_t k)
{
    const uint32_t pairs = (uint32_t)num_sms() / 2, chunks = (k - 1) / kF32Chunk + 1;
    TilesPlan plan = {0, 1};
    if (pairs == 0 || k < 2 * kF32Chunk || k >= 1u << 28 || m >= 1u << 31 || n >= 1u << 31)
        return plan;
    float best = 0.95f * simt_f32_estimate(m, n, k);
    for (uint32_t splits = 1; splits <= 4 && chunks >= 2 * splits; splits *= 2) {
        const uint32_t resident = splits == 1 ? pairs : splits == 2 ? pairs * 33 / 74 : pairs * 15 / 74;
        if (resident == 0)
            break;
        for (uint32_t tn = 32; tn <= 128; tn += 32) {
            const uint64_t tiles = (uint64_t)((m - 1) / kF32M + 1) * ((n - 1) / tn + 1);
            const float waves = (float)((tiles - 1) / resident + 1), wide = (float)tn / 256.0f;
            const float chunk = 0.22f + 0.92f * wide > 0.44f ? 0.22f + 0.92f * wide : 0.44f;
            const float t = 5.0f + waves * ((float)((chunks - 1) / splits + 1) * chunk + 5.0f * wide + (splits > 1 ? 1.0f + 7.0f * wide : 0.0f));
            if (t < best) {
                best = t;
                plan = {tn, splits};
            }
        }
    }
    return plan;
}

template <uint32_t TN>
static int launch_f32(const clpk_gemm_args_t *a, uint32_t splits, cudaStream_t s)
{
    using T = F32Tile<TN>;
    F32Maps maps;
    int rc = make_operand_map(&maps.a, a->d_a, a->m, (uint64_t)a->k * 4);
    if (rc != CLPK_OK)
        return rc;
    rc = make_operand_map(&maps.b, a->d_b, a->n, (uint64_t)a->k * 4, TN / 2);
    if (rc != CLPK_OK)
        return rc;
    F32Params p;
    p.m = a->m;
    p.n = a->n;
    p.k = a->k;
    p.tiles_m = (a->m + kF32M - 1) / kF32M;
    p.tiles_n = (a->n + TN - 1) / TN;
    p.group = tuning(CLPK_TUNE_GEMM_GROUP) > 0 ? (uint32_t)tuning(CLPK_TUNE_GEMM_GROUP) : 8;
    p.chunks = (a->k + kF32Chunk - 1) / kF32Chunk;
    p.splits = splits;
    p.a = static_cast<const float *>(a->d_a);
    p.b = static_cast<const float *>(a->d_b);
    p.c = static_cast<float *>(a->d_c);
    p.alpha = a->alpha;
    p.status = a->d_status;
    const uint32_t n_tiles = p.tiles_m * p.tiles_n, pairs = (uint32_t)num_sms() / 2;
    const uint32_t clusters = splits > 1 ? n_tiles : (n_tiles < pairs ? n_tiles : pairs);
    return launch_clusters(gemm_f32_kernel<TN>, "gemm_f32", clusters * 2 * splits, kF32Threads, T::smem_bytes, 2 * splits, s, maps, p);
}

static int launch_f32_tiles(const clpk_gemm_args_t *a, TilesPlan plan, cudaStream_t s)
{
    switch (plan.tn) {
    case 32:  return launch_f32<32>(a, plan.splits, s);
    case 64:  return launch_f32<64>(a, plan.splits, s);
    case 96:  return launch_f32<96>(a, plan.splits, s);
    default:  return launch_f32<128>(a, plan.splits, s);
    }
}

} // namespace clpk

using namespace clpk;

extern "C" {

int clpk_gemm_plan(int dtype, uint32_t m, uint32_t n, uint32_t k, uint32_t *tile_n, uint32_t *splits, uint32_t *wide)
{
    int rc = require_sm100();
    if (rc != CLPK_OK)
        return rc;
    CLPK_REQUIRE(tile_n && splits, "NULL output");
    CLPK_REQUIRE(m > 0 && n > 0 && k > 0, "M, N and K must be positive");
    uint32_t no_wide = 0;
    if (dtype == CLPK_DT_F32) {
        if (const TilesPlan plan = plan_f32(m, n, k); plan.tn) {
            *tile_n = plan.tn;
            *splits = plan.splits;
            if (wide)
                *wide = 2;
            return CLPK_OK;
        }
    }
    if (dtype == CLPK_DT_F32 || dtype == CLPK_DT_F32_FFMA || dtype == CLPK_DT_F64) {
        simt_gemm_plan(dtype == CLPK_DT_F64, m, n, k, tile_n, splits, wide ? wide : &no_wide);
        return CLPK_OK;
    }
    const uint32_t elem_bits = tensor_elem_bits(dtype);
    CLPK_REQUIRE(elem_bits > 0, "clpk_gemm_plan: dtype %d has no GEMM", dtype);
    const TilesPlan plan = gemm_plan(m, n, k, elem_bits, elem_bits == 4);
    *tile_n = plan.tn;
    *splits = plan.splits;
    if (wide)
        *wide = plan.row_blocks - 1;
    return CLPK_OK;
}

int clpk_gemm_last_launch_aligned(void) { return g_last_aligned; }

int clpk_gemm_wave_state(uint32_t *h_counters_set, uint32_t *h_dropouts, void *stream)
{
    CLPK_REQUIRE(h_counters_set && h_dropouts, "NULL output");
    unsigned int counters[kSyncSlots][2], dropouts = 0;
    void *sym = nullptr;
    CLPK_CUDA(cudaGetSymbolAddress(&sym, g_wave_sync));
    CLPK_CUDA(cudaMemcpyAsync(counters, sym, sizeof counters, cudaMemcpyDeviceToHost, as_stream(stream)));
    CLPK_CUDA(cudaGetSymbolAddress(&sym, g_wave_dropouts));
    CLPK_CUDA(cudaMemcpyAsync(&dropouts, sym, sizeof dropouts, cudaMemcpyDeviceToHost, as_stream(stream)));
    CLPK_CUDA(cudaStreamSynchronize(as_stream(stream)));
    *h_counters_set = 0;
    for (const auto &slot : counters)
        *h_counters_set += (slot[0] != 0) + (slot[1] != 0);
    *h_dropouts = dropouts;
    return CLPK_OK;
}

int clpk_gemm_last_clock(unsigned long long *h_cycles, unsigned long long *h_ns, void *stream)
{
    CLPK_REQUIRE(h_cycles && h_ns, "NULL output");
    unsigned long long v[2] = {0, 0};
    void *sym = nullptr;
    CLPK_CUDA(cudaGetSymbolAddress(&sym, g_gemm_clock));
    CLPK_CUDA(cudaMemcpyAsync(v, sym, sizeof v, cudaMemcpyDeviceToHost, as_stream(stream)));
    CLPK_CUDA(cudaStreamSynchronize(as_stream(stream)));
    *h_cycles = v[0];
    *h_ns = v[1];
    return CLPK_OK;
}

int clpk_gemm_workspace_bytes(int dtype, uint32_t m, uint32_t n, uint32_t k, size_t *bytes)
{
    CLPK_REQUIRE(bytes, "bytes is NULL");
    *bytes = 0;
    const size_t rows = (size_t)padded_rows(m) + padded_rows(n);      // scale blocks cover whole tiles
    if (dtype == CLPK_DT_NVF4)
        *bytes = rows * (k / 16);
    if (dtype == CLPK_DT_MXF4)              // packed into 4-byte words of which each instruction uses two bytes
        *bytes = rows * (k / 32);
    return CLPK_OK;
}

// Width of the block-scaled kernel's cluster tile for a problem: 256 (one accumulator, least operand
// traffic) or 128 (two accumulators, the epilogue overlaps the next tile).  The GEMM_FP4_TILE knob
// forces one; the choice also fixes the order of B's scale blocks in the workspace, so a workspace
// packed by clpk_gemm_pack_scales belongs to the knob setting it was packed under.
static uint32_t fp4_tile_n(uint32_t m, uint32_t n, uint32_t k)
{
    const int t = tuning(CLPK_TUNE_GEMM_FP4_TILE);
    if (t == 1)
        return 256;
    if (t == 2)
        return 128;
    (void)m; (void)n; (void)k;
    return 256;
}

// 32-bit scale words per row per 256 elements of K, and the bytes that all of an operand's take in the workspace
static uint32_t scale_words(int dtype) { return dtype == CLPK_DT_MXF4 ? 2 : 4; }
static size_t scale_bytes(const clpk_gemm_args_t *a, uint32_t rows) { return (size_t)padded_rows(rows) * (a->k / 256) * scale_words(a->dtype) * 4; }

// what the arrangement of row-major scale bytes asks for
static int check_scales(const clpk_gemm_args_t *a)
{
    CLPK_REQUIRE(a->d_sfa && a->d_sfb, "block-scaled FP4 needs d_sfa and d_sfb");
    CLPK_REQUIRE(a->d_workspace && a->workspace_bytes >= scale_bytes(a, a->m) + scale_bytes(a, a->n) && ((uintptr_t)a->d_workspace % 16) == 0,
                 "block-scaled FP4 needs a 16-byte aligned workspace of clpk_gemm_workspace_bytes() bytes");
    CLPK_REQUIRE(((uintptr_t)a->d_sfa % 4) == 0 && ((uintptr_t)a->d_sfb % 4) == 0, "scale arrays must be 4-byte aligned");
    return CLPK_OK;
}

// Row-major scale bytes of both operands -> tile order in the workspace (A's blocks, then B's).
static int pack_scales(const clpk_gemm_args_t *a, cudaStream_t s)
{
    const int rc = check_scales(a);
    if (rc != CLPK_OK)
        return rc;
    const uint32_t words = scale_words(a->dtype);
    uint8_t *wsa = static_cast<uint8_t *>(a->d_workspace), *wsb = wsa + scale_bytes(a, a->m);
    const uint32_t kblocks = a->k / 256;
    const PackOperand oa = pack_operand(a->d_sfa, wsa, a->m, words), ob = pack_operand(a->d_sfb, wsb, a->n, words);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((oa.row_groups + ob.row_groups) * ((kblocks + 7) / 8));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = tuning(CLPK_TUNE_GEMM_NO_PDL) == 1 ? 0 : 1;
    cfg.attrs = pdl;
    cfg.numAttrs = 1;
    const uint32_t b_pairs = fp4_tile_n(a->m, a->n, a->k) == 256 ? 1 : 0;
    const cudaError_t e = words == 4 ? cudaLaunchKernelEx(&cfg, pack_scales_kernel<4>, oa, ob, kblocks, b_pairs)
                                     : cudaLaunchKernelEx(&cfg, pack_scales_kernel<2>, oa, ob, kblocks, b_pairs);
    if (e != cudaSuccess)
        return cuda_fail(e, "launch pack_scales");
    return CLPK_OK;
}

int clpk_gemm_pack_scales(const clpk_gemm_args_t *a, void *stream)
{
    int rc = require_sm100();
    if (rc != CLPK_OK)
        return rc;
    CLPK_REQUIRE(a, "args is NULL");
    CLPK_REQUIRE(a->dtype == CLPK_DT_NVF4 || a->dtype == CLPK_DT_MXF4, "only the block-scaled FP4 kinds have scales to pack");
    CLPK_REQUIRE(a->m > 0 && a->n > 0 && a->k > 0 && a->k % 256 == 0, "M, N positive and K a positive multiple of 256 (got %u, %u, %u)",
                 a->m, a->n, a->k);
    return pack_scales(a, as_stream(stream));
}

int clpk_gemm(const clpk_gemm_args_t *a, void *stream)
{
    int rc = require_sm100();
    if (rc != CLPK_OK)
        return rc;
    CLPK_REQUIRE(a, "args is NULL");
    CLPK_REQUIRE(a->d_a && a->d_b && a->d_c && a->d_status, "NULL buffer");
    if (a->dtype == CLPK_DT_F32 || a->dtype == CLPK_DT_F32_FFMA || a->dtype == CLPK_DT_F64) {
        const int type = a->dtype == CLPK_DT_F64 ? CLPK_DT_F64 : CLPK_DT_F32;
        rc = check_simt_gemm(type, a->d_a, a->d_b, a->d_c, a->m, a->n, a->k);
        if (rc != CLPK_OK)
            return rc;
        if (a->dtype == CLPK_DT_F32)
            if (const TilesPlan plan = plan_f32(a->m, a->n, a->k); plan.tn)
                return launch_f32_tiles(a, plan, as_stream(stream));
        // the CUDA-core fp32 and DMMA fp64 kernels of simt_gemm.cu
        g_last_aligned = 0;
        return launch_simt_gemm(type, a->d_a, a->d_b, a->d_c, a->m, a->n, a->k, a->alpha, a->d_status, as_stream(stream));
    }
    CLPK_REQUIRE(a->m > 0 && a->n > 0 && a->k > 0, "M, N and K must be positive");
    const bool block_scaled = a->dtype == CLPK_DT_NVF4 || a->dtype == CLPK_DT_MXF4;
    // Ragged shapes: TMA fills what a box reads beyond the operands with zeros and clips what a box would store
    // beyond C, so a partial tile costs a whole one but needs no code.  The block-scaled kinds keep K in whole
    // stages of 256 elements (four instructions' scale factors travel as one block); their scale blocks are
    // packed for whole tiles, with zero factors for the rows beyond M and N.
    CLPK_REQUIRE(!block_scaled || a->k % 256 == 0, "block-scaled FP4 needs K to be a multiple of 256 (got %u)", a->k);
    CLPK_REQUIRE(((uintptr_t)a->d_a % 16) == 0 && ((uintptr_t)a->d_b % 16) == 0 && ((uintptr_t)a->d_c % 16) == 0,
                 "operands must be 16-byte aligned");
    const uint32_t elem_bits = tensor_elem_bits(a->dtype);
    if (elem_bits == 0) {
        set_error("clpk_gemm: dtype %d is not available in this build", a->dtype);
        return CLPK_ERR_UNSUPPORTED;
    }
    cudaStream_t s = as_stream(stream);

    const uint64_t row_bytes = (uint64_t)a->k * elem_bits / 8;
    CLPK_REQUIRE(((uint64_t)a->k * elem_bits) % (8 * 16) == 0,
                 "K = %u: a row of %u-bit elements must be a multiple of 16 bytes (the pitch of a TMA tensor map)", a->k, elem_bits);
    const uint32_t out_bytes = (a->dtype == CLPK_DT_TF32 || a->dtype == CLPK_DT_I8) ? 4u : 2u;
    CLPK_REQUIRE(((uint64_t)a->n * out_bytes) % 16 == 0, "N = %u: a row of C must be a multiple of 16 bytes", a->n);
    CUtensorMap ta, tb;
    rc = make_operand_map(&ta, a->d_a, a->m, row_bytes);
    if (rc != CLPK_OK)
        return rc;
    rc = make_operand_map(&tb, a->d_b, a->n, row_bytes);
    if (rc != CLPK_OK)
        return rc;

    GemmParams p;
    p.m = a->m;
    p.n = a->n;
    p.k = a->k;
    p.k_block_elems = kRowBytesK;          // x coordinate is in bytes: the maps are typed UINT8
    p.k_blocks = k_blocks_of(a->k, elem_bits);
    p.c = a->d_c;
    p.alpha = a->alpha;
    p.status = a->d_status;
    // waves of ~(SM pairs) tiles that are about square in elements: twice as many 256-wide tile columns
    // as 512-tall tile rows (74 pairs: 12 x 6)
    p.group = block_scaled ? 8 : 12;          // block-scaled: 256 x 256 tiles, a wave of 74 is about 8 x 9
    p.wave_sync = nullptr;
    p.align_at = 2;
    p.align_period = block_scaled ? 8 : 1;
    if (const int t = tuning(CLPK_TUNE_GEMM_ALIGN_AT); t >= 0)
        p.align_at = (uint32_t)t;
    if (const int t = tuning(CLPK_TUNE_GEMM_GROUP); t > 0)
        p.group = (uint32_t)t;


    if (block_scaled) {
        const bool mx = a->dtype == CLPK_DT_MXF4;
        const uint32_t words = scale_words(a->dtype);
        const size_t sfa_bytes = scale_bytes(a, a->m), sfb_bytes = scale_bytes(a, a->n);
        CLPK_REQUIRE((a->d_sfa != nullptr) == (a->d_sfb != nullptr), "d_sfa and d_sfb: give both, or neither when the workspace is already packed");
        CLPK_REQUIRE(a->d_workspace && a->workspace_bytes >= sfa_bytes + sfb_bytes && ((uintptr_t)a->d_workspace % 16) == 0,
                     "block-scaled FP4 needs a 16-byte aligned workspace of clpk_gemm_workspace_bytes() bytes");
        uint8_t *wsa = static_cast<uint8_t *>(a->d_workspace), *wsb = wsa + sfa_bytes;
        const PackOperand sa = pack_operand(a->d_sfa, wsa, a->m, words), sb = pack_operand(a->d_sfb, wsb, a->n, words);
        if (a->d_sfa) {
            rc = check_scales(a);
            if (rc != CLPK_OK)
                return rc;
            if (const TilesPlan plan = raw_scales_plan(a, sa, sb); plan.tn)
                return mx ? launch_tiles<CLPK_DT_MXF4, 1, true>(a, ta, row_bytes, p.k_blocks, plan, s, sa, sb)
                          : launch_tiles<CLPK_DT_NVF4, 1, true>(a, ta, row_bytes, p.k_blocks, plan, s, sa, sb);
            rc = pack_scales(a, s);
            if (rc != CLPK_OK)
                return rc;
        }
        const uint32_t tn = fp4_tile_n(a->m, a->n, a->k);
        if (const TilesPlan plan = gemm_plan(a->m, a->n, a->k, elem_bits, a->d_sfa == nullptr); plan.tn)
            return mx ? launch_tiles<CLPK_DT_MXF4>(a, ta, row_bytes, p.k_blocks, plan, s, sa, sb)
                      : launch_tiles<CLPK_DT_NVF4>(a, ta, row_bytes, p.k_blocks, plan, s, sa, sb);
        CUtensorMap tsa, tsb;
        rc = make_scale_map(&tsa, wsa, sfa_bytes / 512, words);
        if (rc != CLPK_OK)
            return rc;
        rc = make_scale_map(&tsb, wsb, sfb_bytes / 512, words * tn / 128);
        if (rc != CLPK_OK)
            return rc;
        CUtensorMap tc;
        rc = make_output_map(&tc, a->d_c, a->m, a->n, a->dtype);
        if (rc != CLPK_OK)
            return rc;
        const uint32_t n_tiles = ((a->m + kTileMN - 1) / kTileMN) * ((a->n + tn - 1) / tn);
        if (tn == 128) {
            rc = make_operand_map(&tb, a->d_b, a->n, row_bytes, 64);       // each CTA stages 64 rows of B per stage
            if (rc != CLPK_OK)
                return rc;
            if (tuning(CLPK_TUNE_GEMM_GROUP) <= 0)
                p.group *= 2;                                              // the same panel width in elements
            p.align_period *= 2;
            return mx ? launch_persistent(gemm_block_scaled_kernel<true, 128>, "gemm_mxf4 (256x128)", kNvGemmThreads,
                                          BlockScaled<true, 128>::smem_bytes, s, p, n_tiles, ta, tb, tsa, tsb, tc)
                      : launch_persistent(gemm_block_scaled_kernel<false, 128>, "gemm_nvf4 (256x128)", kNvGemmThreads,
                                          BlockScaled<false, 128>::smem_bytes, s, p, n_tiles, ta, tb, tsa, tsb, tc);
        }
        return mx ? launch_persistent(gemm_block_scaled_kernel<true, 256>, "gemm_mxf4", kNvGemmThreads,
                                      BlockScaled<true, 256>::smem_bytes, s, p, n_tiles, ta, tb, tsa, tsb, tc)
                  : launch_persistent(gemm_block_scaled_kernel<false, 256>, "gemm_nvf4", kNvGemmThreads,
                                      BlockScaled<false, 256>::smem_bytes, s, p, n_tiles, ta, tb, tsa, tsb, tc);
    }
    if (const TilesPlan plan = gemm_plan(a->m, a->n, a->k, elem_bits, false); plan.tn) {
        switch (a->dtype) {
        case CLPK_DT_BF16: return launch_dense_tiles<CLPK_DT_BF16>(a, ta, row_bytes, p.k_blocks, plan, s);
        case CLPK_DT_F16:  return launch_dense_tiles<CLPK_DT_F16>(a, ta, row_bytes, p.k_blocks, plan, s);
        case CLPK_DT_TF32: return launch_dense_tiles<CLPK_DT_TF32>(a, ta, row_bytes, p.k_blocks, plan, s);
        case CLPK_DT_I8:   return launch_dense_tiles<CLPK_DT_I8>(a, ta, row_bytes, p.k_blocks, plan, s);
        case CLPK_DT_E5M2: return launch_dense_tiles<CLPK_DT_E5M2>(a, ta, row_bytes, p.k_blocks, plan, s);
        default:           return launch_dense_tiles<CLPK_DT_E4M3>(a, ta, row_bytes, p.k_blocks, plan, s);
        }
    }
    CUtensorMap tc;
    rc = make_output_map(&tc, a->d_c, a->m, a->n, a->dtype);
    if (rc != CLPK_OK)
        return rc;
    switch (a->dtype) {
    case CLPK_DT_BF16: return launch_gemm<CLPK_DT_BF16>(ta, tb, tc, p, s);
    case CLPK_DT_F16:  return launch_gemm<CLPK_DT_F16>(ta, tb, tc, p, s);
    case CLPK_DT_TF32: return launch_gemm<CLPK_DT_TF32>(ta, tb, tc, p, s);
    case CLPK_DT_I8:   return launch_gemm<CLPK_DT_I8>(ta, tb, tc, p, s);
    case CLPK_DT_E5M2: return launch_gemm<CLPK_DT_E5M2>(ta, tb, tc, p, s);
    default:           return launch_gemm<CLPK_DT_E4M3>(ta, tb, tc, p, s);
    }
}

} // extern "C"
