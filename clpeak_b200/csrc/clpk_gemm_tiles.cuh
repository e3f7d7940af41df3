// The GEMM for shapes that do not fill the chip with the large kernels' tiles (included by gemm.cu).
//
// Same pieces as gemm_kernel -- CTA pairs, TMA ring, elected-lane issue, bounded waits -- with the split of the work
// left to the launch:
//  * Tile 256 x TN per CTA pair, TN = 32 ... 256 in steps of 32, one M = 256 row block (CTA r holds its 128 rows).
//  * Dense kinds, K not split: also 512 x TN, a second row block that shares the tile's B.  The 512 x 256 tiles of gemm_kernel
//    leave the chip idle where they are few or their last wave is nearly empty, and where N is just above a multiple of
//    256; narrower ones of the same height read as little of A.  Up to TN = 128 there are two accumulators, beyond one,
//    whose reading the next tile waits for.  bf16 10149 x 456 x 2176 28.6 -> 19.6 us, e4m3 2882 x 1544 x 4864 29.6 -> 21.3, i8
//    9909 x 488 x 2304 19.6 -> 16.0, tf32 8248 x 1576 x 640 36.8 -> 31.0.
//  * K over 1, 2 or 4 pairs of one cluster.  Every pair accumulates its own K range in tensor memory; then the pairs
//    exchange partial sums through distributed shared memory (each owns every splits-th 32-column chunk of the tile),
//    add them in pair order -- the same order whoever owns the chunk -- and store what they own.  Nothing goes through
//    global memory and no workspace is needed.
//  * Unsplit tiles are walked persistently with two accumulators, so a tile's epilogue overlaps the next main loop.
//
// What bounds it: a K block (128 bytes of K) costs the issuing warps about 0.12 us whatever the tile -- barrier wait,
// four instructions, commit -- against 0.17 us of tensor pipe at TN = 256, so narrow tiles are issue-bound and their
// width is chosen for parallelism; wide ones come within 10 % of the operand traffic's floor.  Below 2 us per K range
// the launch is the time: 4 to 5 us from one launch's last CTA to the next one's first full stage.  Device time, operands in L2, 512 x 256 tiles -> this
// kernel: bf16 512 x 256 x 512 10.2 -> 4.4 us, e4m3 1024 x 1024 x 2048 15.0 -> 6.4, bf16 2048^3 25.1 -> 15.3, e4m3
// 128 x 8192 x 8192 42.4 -> 18.6, bf16 64 x 64 x 16384 147 -> 13.3.  Tried: four K blocks per stage (slower from
// TN = 64 on), asking the next stage's barrier ahead of the instructions (no effect), clusters of 16 for eight splits
// (10 % for single tiles of K > 8000, slower elsewhere).
//
// Block-scaled kinds: TN = 64, 128 or 256 (split, or with one accumulator where the scales are arranged on the way), one K block
// and its scale factors per stage; a block is 13 (NVFP4,
// TN = 128) issued instructions and costs 0.25 us, so that splitting K pays early: NVFP4 95 x 352 x 8960 14.7 -> 8.0 us,
// MXFP4 2654 x 120 x 16384 22.4 -> 11.8, NVFP4 458 x 1176 x 6400 12.4 -> 10.2.
#pragma once

constexpr int kTilesMaxStages = 16;
constexpr uint32_t kTilesChunk = 32;                               // columns of C per tcgen05.ld and per TMA store box
constexpr uint32_t kTilesM = 256;
constexpr uint32_t kTilesSmemMax = 227 * 1024;

struct TilesSmem {
    uint64_t full[kTilesMaxStages];
    uint64_t empty[kTilesMaxStages];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
};

// The block-scaled kinds carry 2 KiB of A's factors and 2 KiB per 128 columns of B's with every K block (MXFP4 fills
// half of that), in the blocks that pack_scales_kernel makes; they go to tensor memory in front of the K block's
// instructions as in gemm_block_scaled_kernel, in columns of their own per stage behind 256 accumulator columns.
template <int DT> struct TilesKind {
    static constexpr bool fp4 = DT == CLPK_DT_NVF4 || DT == CLPK_DT_MXF4;
    static constexpr uint32_t words = DT == CLPK_DT_MXF4 ? 2 : 4;          // 512-byte blocks per 128 rows and K block
};
__host__ __device__ constexpr uint32_t tiles_sf_bytes(uint32_t tn) { return 2048 + (tn + 127) / 128 * 2048; }
__host__ __device__ constexpr uint32_t tiles_sf_cols(uint32_t tn) { return 16 + (tn + 127) / 128 * 16; }

struct TilesMaps {
    CUtensorMap a, b, c;
};
struct TilesScaleMaps {
    CUtensorMap a, b, c, sfa, sfb;
};
// One operand's scale factors on their way from row-major to the order of tensor memory (see pack_scales_kernel).
struct PackOperand {
    const uint32_t *in;
    uint32_t *out;
    uint32_t rows, row_groups;          // row groups of 128 after padding
    uint32_t vector;                    // 1: `in` is aligned to a stage's words
};

// one row's words of a K block of 256 elements; zeros beyond the operand
template <int WORDS>
__device__ __forceinline__ void load_scale_words(const PackOperand &op, uint32_t row, uint32_t kb, uint32_t kblocks, uint32_t (&w)[WORDS])
{
    const uint32_t *src = op.in + ((uint64_t)row * kblocks + kb) * WORDS;
#pragma unroll
    for (int j = 0; j < WORDS; j++)
        w[j] = 0;
    if (row >= op.rows)
        return;
    if (op.vector) {
        if constexpr (WORDS == 4) {
            const uint4 v = *reinterpret_cast<const uint4 *>(src);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        } else {
            const uint2 v = *reinterpret_cast<const uint2 *>(src);
            w[0] = v.x; w[1] = v.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < WORDS; j++)
            w[j] = src[j];
    }
}

// which 512-byte block of the arranged operand has word j of a group of 128 rows' K block; `pairs`: two groups' blocks lie together
template <int WORDS>
__device__ __forceinline__ uint64_t scale_block(uint32_t group, uint32_t kb, uint32_t j, uint32_t kblocks, bool pairs)
{
    return pairs ? (((uint64_t)(group >> 1) * kblocks + kb) * WORDS + j) * 2 + (group & 1) : ((uint64_t)group * kblocks + kb) * WORDS + j;
}

// Block-scaled operands whose scales are still row-major: `out` is where the workspace has their blocks.
struct TilesRawMaps {
    CUtensorMap a, b, c;
    PackOperand sa, sb;
};
template <int DT, bool kRaw> using TilesMapsOf = std::conditional_t<kRaw, TilesRawMaps, std::conditional_t<TilesKind<DT>::fp4, TilesScaleMaps, TilesMaps>>;

constexpr int kTilesScaleWarps = 6;
constexpr int tiles_threads(bool raw) { return kGemmThreads + (raw ? 32 * kTilesScaleWarps : 0); }

struct TilesParams {
    uint32_t tiles_m, tiles_n, group;
    uint32_t k_blocks;                  // of 128 bytes
    uint32_t tn, splits, stages;
    uint32_t kps;                       // K blocks per stage: 1 or 2
    uint32_t tmem_cols;                 // power of two: one accumulator, or two when a cluster has several tiles
    float alpha;
    uint32_t *status;
    unsigned long long *clock;
};

// bytes of one K block in a CTA: its 128 rows of each row block of A and its half of the tile's rows of B
__host__ __device__ constexpr uint32_t tiles_block_bytes(uint32_t tn, uint32_t row_blocks = 1) { return row_blocks * kHalfTileBytes + tn / 2 * kRowBytesK; }

// 32 columns of one row per lane -> the warp's staging box (32 rows x 64 bytes of bf16 in the 64-byte swizzle, or
// x 128 bytes of fp32 / int32 in the 128-byte swizzle) -> one TMA store that clips what lies beyond C.
template <int DT>
__device__ __forceinline__ void tiles_store_chunk(uint32_t (&r)[32], float alpha, uint8_t *boxes, uint32_t &n_stored,
                                                  const CUtensorMap *tmap_c, uint32_t col, uint32_t row, int lane)
{
    if constexpr (OutBytes<DT>::value == 2) {
        // two 2 KiB boxes in turn: the one filled now was handed to TMA two stores ago
        uint8_t *box = boxes + (n_stored & 1) * 2048;
        if (lane == 0)
            bulk_wait_read<1>();
        __syncwarp();
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(r[2 * i]) * alpha, __uint_as_float(r[2 * i + 1]) * alpha);
            w[i] = *reinterpret_cast<uint32_t *>(&v);
        }
        uint8_t *my_row = box + lane * 64;
        const uint32_t sw = (uint32_t)(lane >> 1) & 3;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++)
            *reinterpret_cast<uint4 *>(my_row + ((j ^ sw) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(tmap_c, box, (int32_t)col, (int32_t)row);
            bulk_commit();
        }
    } else {
        if constexpr (DT == CLPK_DT_TF32) {
#pragma unroll
            for (int i = 0; i < 32; i++)
                r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
        }
        store_staged_box(r, boxes, tmap_c, col, row, lane);
    }
    n_stored++;
}

// Partial sums of a 32-column chunk in the owner's shared memory: [8 groups of 4 columns][128 rows][4 words], so that
// a warp's 32 rows are 512 consecutive bytes per group on both sides.
constexpr uint32_t kTilesChunkBytes = kTilesChunk * 128 * 4;

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t cta)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
    return a;
}

// 3-D tile load whose completion bytes go to the leader's barrier
__device__ __forceinline__ void tma_load_pair_3d_at(void *smem_dst, const CUtensorMap *tmap, int32_t x, int32_t y, int32_t z, uint32_t leader_bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(leader_bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// ---------------- scale factors that are still row-major (six warps of each CTA) ----------------
// A unit is 32 bytes of 128 rows, the words of two K blocks (NVFP4) or four (MXFP4), of A (this CTA's rows) or of B (each CTA
// needs those of all its tile's columns).  Neighbouring lanes load those K blocks' words of a row, so that a warp's load touches 16 or
// eight lines and not 32, each of which costs the L1 a cycle and more; a lane then holds the transposes of rows r, r + 32, r + 64,
// r + 96, and the lanes of a K block write them to its stage as 16-byte pieces of the blocks that pack_scales_kernel makes.  A K
// block has two or three units, and two or three sets of warps take turns: one loads while others write theirs.  The CTA pairs of the first tile row and column leave the blocks in the workspace as well, where the next call may look for
// them (d_sfa = d_sfb = NULL).
template <uint32_t kWords>
__device__ __forceinline__ void tiles_arrange_scales(const TilesRawMaps &maps, const TilesParams &p, TilesSmem *sh, uint8_t *smem, uint32_t stage_bytes,
                                                     uint32_t block_bytes, uint32_t w, uint32_t lane, uint32_t kb0, uint32_t kb1)
{
    constexpr uint32_t kGroup = 8 / kWords;                     // K blocks per unit
    // A wait tells the last two phases of a barrier apart, no more.  So a warp may not come to a stage two rounds early: from one
    // K block that it waits for to the next there are no more than the ring has stages (five with 256 columns, else six or more).
    constexpr uint32_t kMostSets = kGroup == 4 ? 2 : 3;
    static_assert((2 - 1) * kGroup + 1 <= 5 && (kMostSets - 1) * kGroup + 1 <= 6, "sets of warps too far apart");
    const uint32_t rank = cluster_ctarank(), r = rank & 1, leader = rank & ~1u;
    const uint32_t cluster_id = blockIdx.x / (2 * p.splits), n_clusters = gridDim.x / (2 * p.splits), n_tiles = p.tiles_m * p.tiles_n;
    const uint32_t b_halves = (p.tn + 127) / 128, per_block = 1 + b_halves;
    const uint32_t unit = w % per_block, sets = per_block == 3 ? 2 : kMostSets;
    if (w >= sets * per_block)
        return;
    const bool is_b = unit > 0;
    const PackOperand op = is_b ? maps.sb : maps.sa;
    const uint32_t full0 = cluster_addr(&sh->full[0], leader);
    const uint32_t n_kb = kb1 - kb0, groups = (n_kb + kGroup - 1) / kGroup;
    const uint32_t x = lane / kGroup, mine = lane % kGroup;
    uint8_t *const sf0 = smem + block_bytes + (is_b ? 2048 + (unit - 1) * 512 : 0) + x * 16;
    const uint32_t step = is_b ? b_halves * 512 : 512;

    uint32_t at = w / per_block, before = 0;                   // the group of four of this tile; K blocks of the tiles in front
    for (uint32_t tile = cluster_id; tile < n_tiles; tile += n_clusters, before += n_kb, at -= groups) {
        uint32_t mb, nb;
        dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
        const uint32_t rows = is_b ? nb * p.tn / 128 + unit - 1 : mb * 2 + r;          // which 128
        const bool keep = is_b ? mb == 0 && r == 0 && nb * p.tn % 128 == 0 : nb == 0;
        // a last group of B's rows without a tile for the other half of its 256: that half is zeros
        const bool pad = is_b && rows % 2 == 0 && (rows + 1) * 128 >= p.tiles_n * p.tn;
        for (; at < groups; at += sets) {
            const uint32_t kb = kb0 + kGroup * at, here = kb1 - kb < kGroup ? kb1 - kb : kGroup;
            uint32_t words[4 * kGroup][kWords];
#pragma unroll
            for (uint32_t i = 0; i < 4 * kGroup; i++)
                load_scale_words<kWords>(op, mine < here ? rows * 128 + 32 / kGroup * i + x : ~0u, kb + mine, p.k_blocks, words[i]);
            auto piece = [&](uint32_t i, uint32_t j) { return make_uint4(words[i][j], words[i + kGroup][j], words[i + 2 * kGroup][j], words[i + 3 * kGroup][j]); };
            uint32_t s = (before + kGroup * at) % p.stages, round = (before + kGroup * at) / p.stages;
            for (uint32_t t = 0; t < here; t++) {
                if (!warp_wait(&sh->empty[s], (round + 1) & 1)) {          // a fresh barrier's preceding phase counts as complete
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x226u);
                    return;
                }
                if (mine == t) {
#pragma unroll
                    for (uint32_t i = 0; i < kGroup; i++)
#pragma unroll
                        for (uint32_t j = 0; j < kWords; j++)
                            *reinterpret_cast<uint4 *>(sf0 + (size_t)s * stage_bytes + j * step + i * (512 / kGroup)) = piece(i, j);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive_remote(full0 + 8 * s);
                if (++s == p.stages) {
                    s = 0;
                    round++;
                }
            }
            if (keep && mine < here) {
                uint4 *out = reinterpret_cast<uint4 *>(op.out) + x;
#pragma unroll
                for (uint32_t j = 0; j < kWords; j++) {
                    const uint64_t block = scale_block<kWords>(rows, kb + mine, j, p.k_blocks, is_b);
#pragma unroll
                    for (uint32_t i = 0; i < kGroup; i++) {
                        out[block * 32 + 32 / kGroup * i] = piece(i, j);
                        if (pad)
                            out[(block + 1) * 32 + 32 / kGroup * i] = make_uint4(0, 0, 0, 0);
                    }
                }
            }
        }
    }
}

// kRowBlocks: of 256 rows that share a tile's B, 1 or 2.  A template parameter, because as one of the launch the small
// shapes took 1.4 % longer.
// kRaw: block-scaled operands whose scales lie row-major as their user has them; the last six warps arrange them.
template <int DT, uint32_t kRowBlocks, bool kRaw>
__global__ void __launch_bounds__(tiles_threads(kRaw)) gemm_tiles_kernel(const __grid_constant__ TilesMapsOf<DT, kRaw> maps, TilesParams p)
{
    constexpr bool kFp4 = TilesKind<DT>::fp4;
    constexpr uint32_t kWords = TilesKind<DT>::words;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t b_at = kRowBlocks * kHalfTileBytes;
    const uint32_t block_bytes = tiles_block_bytes(p.tn, kRowBlocks), stage_bytes = p.kps * block_bytes + (kFp4 ? tiles_sf_bytes(p.tn) : 0);
    uint8_t *staging = smem + (size_t)p.stages * stage_bytes;
    TilesSmem *sh = reinterpret_cast<TilesSmem *>(staging + kEpilogueWarps * kStagingBytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank(), r = rank & 1, leader = rank & ~1u, split = rank >> 1;
    const uint32_t cluster_id = blockIdx.x / (2 * p.splits), n_clusters = gridDim.x / (2 * p.splits);
    const uint32_t n_tiles = p.tiles_m * p.tiles_n;
    const bool two_accs = p.tn <= 128 || (kRowBlocks == 1 && !kFp4);        // two accumulators where they fit
    const uint32_t b_halves = (p.tn + 127) / 128;                // blocks of 128 rows of B that a tile's scale factors come in
    const uint32_t kb0 = split * p.k_blocks / p.splits, kb1 = (split + 1) * p.k_blocks / p.splits;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.stages; s++) {
            mbar_init(&sh->full[s], kRaw ? 1 + 2 * (1 + b_halves) : 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int acc = 0; acc < 2; acc++) {
            mbar_init(&sh->tmem_full[acc], 1);
            mbar_init(&sh->tmem_empty[acc], 2 * kEpilogueWarps);
        }
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
        tma_prefetch_desc(&maps.c);
        if constexpr (kFp4 && !kRaw) {
            tma_prefetch_desc(&maps.sfa);
            tma_prefetch_desc(&maps.sfb);
        }
    }
    if (warp == 1)
        tmem_alloc<2>(&sh->tmem_base, p.tmem_cols);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    tc_fence_after_sync();
    const uint32_t tmem = sh->tmem_base;
    griddep_wait();                        // see join_previous_launch
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *p.status = 0u;
    griddep_launch_dependents();
    const unsigned long long clk0 = clock64(), ns0 = globaltimer_ns();

    const uint32_t q = (uint32_t)(warp & 3), half = (uint32_t)(warp - 2) >> 2;     // epilogue warps
    const uint32_t n_chunks = p.tn / kTilesChunk;
    uint8_t *boxes = staging + (size_t)(warp - 2) * kStagingBytes;
    uint32_t n_stored = 0;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        const uint32_t full0 = cluster_addr(&sh->full[0], leader);
        const uint32_t b_blocks = b_halves * kWords;                 // scale blocks of B per K block
        uint32_t s = 0, parity = 1;                            // parity of the empty barrier's previous phase
        bool ok = true;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            uint32_t mb, nb;
            dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
            const int32_t row_a = (int32_t)(mb * kRowBlocks * kTilesM + r * 128), row_b = (int32_t)(nb * p.tn + r * (p.tn / 2));
            for (uint32_t kb = kb0; kb < kb1; kb += p.kps) {
                if (!warp_wait(&sh->empty[s], parity)) {       // a fresh barrier's preceding phase counts as complete
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x221u);
                    ok = false;
                    break;
                }
                uint8_t *st = smem + (size_t)s * stage_bytes;
                const int32_t x = (int32_t)(kb * kRowBytesK);
                const uint32_t nk = kb1 - kb < p.kps ? kb1 - kb : p.kps;
                if (elect_one()) {
                    if (r == 0)
                        mbar_expect_tx(&sh->full[s], nk * 2 * block_bytes + (kFp4 && !kRaw ? 2 * (kWords * 512 + b_blocks * 512) : 0));
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++)
                        if (h < nk) {
                            uint8_t *blk = st + h * block_bytes;
                            tma_load_pair_at(blk, &maps.a, x + h * kRowBytesK, row_a, full0 + 8 * s);
                            if constexpr (kRowBlocks == 2)
                                tma_load_pair_at(blk + kHalfTileBytes, &maps.a, x + h * kRowBytesK, row_a + (int32_t)kTilesM, full0 + 8 * s);
                            tma_load_pair_at(blk + b_at, &maps.b, x + h * kRowBytesK, row_b, full0 + 8 * s);
                        }
                    if constexpr (kFp4 && !kRaw) {
                        // A's blocks lie [rows / 128][K block][word], B's [rows / 256][K block][word][half of the 256]
                        uint8_t *sf = st + block_bytes;
                        tma_load_pair_at(sf, &maps.sfa, 0, (int32_t)(((mb * 2 + r) * p.k_blocks + kb) * kWords), full0 + 8 * s);
                        const uint32_t col = nb * p.tn;
                        tma_load_pair_3d_at(sf + 2048, &maps.sfb, 0, (int32_t)(col / 128 & 1), (int32_t)((col / 256 * p.k_blocks + kb) * kWords),
                                            full0 + 8 * s);
                    }
                }
                __syncwarp();
                if (++s == p.stages) {
                    s = 0;
                    parity ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the pair's leader) ----------------
        if (r == 0) {
            constexpr uint32_t kAFmt = DT == CLPK_DT_BF16 ? kFmtBF16 : DT == CLPK_DT_F16 ? kFmtF16 : DT == CLPK_DT_TF32 ? kFmtTF32
                                     : DT == CLPK_DT_I8 ? kFmtS8 : DT == CLPK_DT_E5M2 ? kFmtE5M2 : kFmtE4M3;
            constexpr uint32_t kBFmt = DT == CLPK_DT_E5M2 ? kFmtE4M3 : kAFmt;
            constexpr bool kMx = DT == CLPK_DT_MXF4;
            // MXFP4: instruction kk reads bytes 0-1 (id 0) or 2-3 (id 2) of word kk / 2
            const uint32_t idesc = kFp4 ? make_idesc_block_scaled(256, p.tn, kFmtE2M1, kFmtE2M1, kMx ? 1u : 0u, 0, 0)
                                        : make_idesc(256, p.tn, kAFmt, kBFmt, DT == CLPK_DT_I8 ? kAccS32 : kAccF32);
            const uint32_t idesc_hi = make_idesc_block_scaled(256, p.tn, kFmtE2M1, kFmtE2M1, 1u, 2, 2);
            const uint16_t pair_mask = (uint16_t)(3u << leader);
            uint32_t s = 0, parity = 0, tcount = 0;
            bool ok = true;
            for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters, tcount++) {
                const uint32_t acc = two_accs ? tcount & 1 : 0, use = two_accs ? tcount >> 1 : tcount;
                if (use > 0 && !warp_wait(&sh->tmem_empty[acc], (use - 1) & 1)) {
                    if (lane == 0)
                        atomicCAS(p.status, 0u, 0x222u);
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d = tmem + acc * kRowBlocks * p.tn;
                [[maybe_unused]] uint32_t mb, nb = 0;
                if constexpr (kFp4)
                    dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
                for (uint32_t kb = kb0; kb < kb1; kb += p.kps) {
                    if (!warp_wait(&sh->full[s], parity)) {
                        if (lane == 0)
                            atomicCAS(p.status, 0u, 0x223u);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t base = smem_u32(smem + (size_t)s * stage_bytes);
                    const uint32_t nk = kb1 - kb < p.kps ? kb1 - kb : p.kps;
                    const uint32_t s_now = s;
                    if (++s == p.stages) {
                        s = 0;
                        parity ^= 1;
                    }
                    if (elect_one()) {
                        if constexpr (kFp4) {
                            const uint32_t sf_s = base + block_bytes, sfa_t = tmem + 256 + s_now * tiles_sf_cols(p.tn);
                            const uint64_t ad = make_smem_desc(base, 16, 1024, kSwizzle128B);
                            const uint64_t bd = make_smem_desc(base + kHalfTileBytes, 16, 1024, kSwizzle128B);
#pragma unroll
                            for (uint32_t w = 0; w < kWords; w++)
                                tmem_cp_32x128b_warpx4<2>(sfa_t + 4 * w, make_smem_desc(sf_s + w * 512, 16, 128, kSwizzleNone));
                            for (uint32_t w = 0; w < kWords * b_halves; w++)
                                tmem_cp_32x128b_warpx4<2>(sfa_t + 16 + 4 * w, make_smem_desc(sf_s + 2048 + w * 512, 16, 128, kSwizzleNone));
                            // a 64-column tile in the upper half of its 128 reads the upper two of a word's four columns
                            const uint32_t sfb_t = sfa_t + 16 + (nb * p.tn % 128) / 32;
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; kk++) {
                                const uint32_t accumulate = (kb != kb0 || kk != 0) ? 1u : 0u;
                                if constexpr (kMx)
                                    mma2_mxf4_bs(d, ad + 2 * kk, bd + 2 * kk, (kk & 1) ? idesc_hi : idesc, sfa_t + 4 * (kk / 2),
                                                 sfb_t + 4 * b_halves * (kk / 2), accumulate);
                                else
                                    mma2_nvf4_bs(d, ad + 2 * kk, bd + 2 * kk, idesc, sfa_t + 4 * kk, sfb_t + 4 * b_halves * kk, accumulate);
                            }
                        }
#pragma unroll
                        for (uint32_t h = 0; h < 2; h++) {
                            if (kFp4 || h >= nk)
                                break;
                            const uint32_t blk = base + h * block_bytes;
                            const uint64_t bd = make_smem_desc(blk + b_at, 16, 1024, kSwizzle128B);
                            auto multiply = [&](uint32_t dd, uint64_t ad) {
#pragma unroll
                                for (uint32_t kk = 0; kk < 4; kk++) {
                                    const uint32_t accumulate = (kb != kb0 || h != 0 || kk != 0) ? 1u : 0u;
                                    if constexpr (DT == CLPK_DT_E4M3 || DT == CLPK_DT_E5M2)
                                        mma2_f8f6f4_ss(dd, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                                    else if constexpr (DT == CLPK_DT_TF32)
                                        mma2_tf32_ss(dd, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                                    else if constexpr (DT == CLPK_DT_I8)
                                        mma2_i8_ss(dd, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                                    else if constexpr (!kFp4)
                                        mma2_f16_ss(dd, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                                }
                            };
                            multiply(d, make_smem_desc(blk, 16, 1024, kSwizzle128B));
                            if constexpr (kRowBlocks == 2)
                                multiply(d + p.tn, make_smem_desc(blk + kHalfTileBytes, 16, 1024, kSwizzle128B));
                        }
                        tc_commit_pair(&sh->empty[s_now], pair_mask);
                    }
                    __syncwarp();
                }
                if (ok && elect_one())
                    tc_commit_pair(&sh->tmem_full[acc], pair_mask);
                __syncwarp();
            }
        }
    } else if (kRaw && warp >= 2 + kEpilogueWarps) {
        if constexpr (kRaw)
            tiles_arrange_scales<kWords>(maps, p, sh, smem, stage_bytes, block_bytes, warp - (2 + kEpilogueWarps), lane, kb0, kb1);
    } else if (p.splits == 1) {
        // ---------------- epilogue, K not split: the two warps of a lane quarter take every other chunk ----------------
        uint32_t tcount = 0;
        for (uint32_t tile = cluster_id; tile < n_tiles; tile += n_clusters, tcount++) {
            uint32_t mb, nb;
            dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
            const uint32_t acc = two_accs ? tcount & 1 : 0, use = two_accs ? tcount >> 1 : tcount;
            if (!warp_wait(&sh->tmem_full[acc], use & 1)) {
                if (lane == 0)
                    atomicCAS(p.status, 0u, 0x224u);
                break;
            }
            tc_fence_after_sync();
            // the row blocks' chunks lie one behind another in tensor memory
            const uint32_t all_chunks = kRowBlocks * n_chunks;
            const uint32_t taddr = tmem + acc * kRowBlocks * p.tn + ((q * 32) << 16);
            const uint32_t row = mb * kRowBlocks * kTilesM + r * 128 + q * 32;
            auto store = [&](uint32_t (&v)[32], uint32_t c) {
                const uint32_t block = kRowBlocks == 2 && c >= n_chunks ? 1 : 0;
                tiles_store_chunk<DT>(v, p.alpha, boxes, n_stored, &maps.c, nb * p.tn + (c - block * n_chunks) * kTilesChunk, row + block * kTilesM, lane);
            };
            auto release = [&]() {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive_cluster_relaxed(&sh->tmem_empty[acc], leader);
            };
            if (half >= all_chunks)
                release();
            for (uint32_t c = half; c < all_chunks; c += 4) {
                // two chunks in flight
                const bool two = c + 2 < all_chunks;
                uint32_t v0[32], v1[32];
                tmem_ld_32x32b_x32(taddr + c * kTilesChunk, v0);
                if (two)
                    tmem_ld_32x32b_x32(taddr + (c + 2) * kTilesChunk, v1);
                tmem_ld_wait();
                if (c + 4 >= all_chunks)
                    release();
                store(v0, c);
                if (two)
                    store(v1, c + 2);
            }
        }
    } else if (!warp_wait(&sh->tmem_full[0], 0)) {
        if (lane == 0)
            atomicCAS(p.status, 0u, 0x225u);
    }

    if (p.splits > 1) {
        // ---------------- K split over the cluster's pairs (one tile per cluster) ----------------
        // Every pair's instructions have retired, so the stages of the ring are free to take partial sums: slot
        // (src, j) of CTA (owner, r) holds pair src's sums of the owner's j-th chunk, src counted without the owner.
        tc_fence_before_sync();
        __syncwarp();
        cluster_sync();
        tc_fence_after_sync();
        const uint32_t slots = (n_chunks + p.splits - 1) / p.splits;
        const uint32_t taddr = tmem + ((q * 32) << 16), my_row = q * 32 + lane;
        const bool epilogue = warp >= 2 && warp < 2 + kEpilogueWarps;
        if (epilogue) {
            for (uint32_t c = half; c < n_chunks; c += 2) {
                const uint32_t owner = c % p.splits;
                if (owner == split)
                    continue;
                uint32_t v[32];
                tmem_ld_32x32b_x32(taddr + c * kTilesChunk, v);
                tmem_ld_wait();
                const uint32_t src = split < owner ? split : split - 1;
                const uint32_t dst = cluster_addr(smem + (size_t)(src * slots + c / p.splits) * kTilesChunkBytes + my_row * 16, owner * 2 + r);
#pragma unroll
                for (uint32_t g = 0; g < 8; g++)
                    st_cluster_v4(dst + g * 2048, v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            }
        }
        __syncwarp();
        cluster_sync();
        if (epilogue) {
            uint32_t mb, nb;
            dense_tile_coords(cluster_id, p.tiles_m, p.tiles_n, p.group, mb, nb);
            const uint32_t row = mb * kTilesM + r * 128 + q * 32;
            for (uint32_t j = half; split + j * p.splits < n_chunks; j += 2) {
                const uint32_t c = split + j * p.splits;
                uint32_t own[32], sum[32];
                tmem_ld_32x32b_x32(taddr + c * kTilesChunk, own);
                tmem_ld_wait();
                for (uint32_t src = 0; src < p.splits; src++) {
                    const uint8_t *slot = smem + (size_t)((src < split ? src : src - 1) * slots + j) * kTilesChunkBytes + my_row * 16;
#pragma unroll
                    for (uint32_t g = 0; g < 8; g++) {
                        uint4 v = make_uint4(own[4 * g], own[4 * g + 1], own[4 * g + 2], own[4 * g + 3]);
                        if (src != split)
                            v = *reinterpret_cast<const uint4 *>(slot + g * 2048);
                        const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (uint32_t t = 0; t < 4; t++) {
                            if (src == 0)
                                sum[4 * g + t] = e[t];
                            else if constexpr (DT == CLPK_DT_I8)
                                sum[4 * g + t] += e[t];
                            else
                                sum[4 * g + t] = __float_as_uint(__uint_as_float(sum[4 * g + t]) + __uint_as_float(e[t]));
                        }
                    }
                }
                tiles_store_chunk<DT>(sum, p.alpha, boxes, n_stored, &maps.c, nb * p.tn + c * kTilesChunk, row, lane);
            }
        }
    }
    // the staging boxes must have been read before this CTA's shared memory goes away
    if (warp >= 2 && lane == 0)
        bulk_wait_read<0>();

    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.clock) {
        p.clock[0] = clock64() - clk0;
        p.clock[1] = globaltimer_ns() - ns0;
    }
    if (warp == 1)
        tmem_dealloc<2>(tmem, p.tmem_cols);
}
