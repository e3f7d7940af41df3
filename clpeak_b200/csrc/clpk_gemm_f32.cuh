// The fp32 GEMM on the tensor cores (included by gemm.cu).
//
// An fp32 number is the sum of three bf16 numbers: h is x rounded to bf16, m what is left rounded to bf16, and l what is
// left then, which has no more than eight significand bits -- h + m + l = x exactly, with |m| <= 2^-8 |x| and
// |l| <= 2^-17 |x|.  A product of two fp32 numbers is then nine bf16 products, each exact in fp32; the three smallest
// (m l, l m, l l: at most 2^-24 of the product together, of either sign) are left out, which is no more than the rounding
// that one fp32 operation makes.  Six bf16 instructions per K step at the tensor pipe's 16-bit rate are four times what
// the fp32 pipe does.
//
// bf16 ends where fp32 does, so the pieces of a small x would not exist.  The elements are multiplied by 2^16 on the way, after
// which none has bits below bf16's last one, 2^-133: every finite number up to 2^111, subnormal ones too, is then three bf16
// numbers with m and l as far below h as said above.  (Subnormal bf16 operands and sums are not flushed.)  The sums are multiplied
// by 2^-32 when they leave the registers.  A product that a result of 2^-149 could feel is 2^-117 and more in the accumulator, and
// its last bit 2^-149: results keep their bits down to the end of the fp32 range, with fewer errors there than fused
// multiply-adds, which round each step to 2^-149 (K = 2044, results near 2^-135: at most 2 units of 2^-149 against 56).
// With elements at their own size, tiles with an element or a sum below 2^-100 had to be multiplied again: 40.5 ms for a 4096^3
// product of that kind against 0.62, and 1.05 for one with zeros, for which the same alarm went off.  (m and l at 2^8 and 2^16
// times their size besides, with the accumulator divided between products of different sizes, took two more multiplications of a
// pair and gained nothing.)
//
// The tensor cores cut, not round, what they align to the accumulator, so sums are kept short there: a turn of two chunks of 32
// floats starts from zero, adds the small products first and the h h ones last -- four instructions in which the cut is of
// the sum's size -- and the turn's sum is added to registers with ordinary rounded fp32 additions.  Against the sum in
// 64 bits that is more accurate than a chain of K fused multiply-adds: N(0, 0.02) operands, 2-norm of the error over that
// of the result, 0.9e-7 at K = 256, 1.7e-7 at 4096 and 3.0e-7 at 16384, against 2.9e-7, 1.1e-6 and 2.3e-6.  Sums of one sign, where the
// cuts do not cancel, come out low by 6 to 8.5e-8 of their size at every K; only chains as short as the 128 products of
// eight that the CUDA-core kernels add for 1024 x 65 x 1028 are better there (7.3e-8 against 8.8e-8).
//
//  * Tile 256 x TN per CTA pair (cta_group::2, M = 256), CTA r holding 128 rows of A and of C, and TN / 2 rows of B.
//  * A chunk is 32 floats of K: one 128-byte row per operand row, fetched by TMA as it lies in memory (warp 0).
//  * Two groups of four warps take turns at the chunks: each lane turns a row of A into bf16 and puts it in tensor memory, from
//    where an instruction may take A (from shared memory, whose port it would fill, a chunk of 128 columns takes 1309
//    cycles against 889), and the warps turn B into three planes of 64-byte rows in shared memory.
//  * Warps 1 and 2 of the pair's leader issue a turn each, 24 instructions, into one of two to four accumulators of TN columns.
//  * The last eight warps read an accumulator while others fill, and add it to their sums: 32 rows x TN / 2 columns each.
//  * K over 1, 2 or 4 pairs of a cluster as in gemm_tiles_kernel: partial sums meet in the raw tiles' shared memory and
//    are added in pair order.
//
// What bounds it: the turns of converters, instructions and sums rather than any one of them.  A chunk's 12 instructions take 430
// cycles at TN = 32 and 890 at 128, a whole turn of one chunk 1060: without the arithmetic of the conversion (12 issue slots of an
// SM quarter for a pair of floats) 880, without the additions 1000, with two of the 12 instructions 1000.  The tensor pipe is busy
// for 73 % of the cycles of a 2304 x 4096 x 2048 product, issue slots 54 %; from about 300 us on the power cap takes the clock down to
// 1.4 GHz and with it what is left to gain.  Device time against the CUDA-core kernels: 4096^3 2251 -> 570 to 650 us back to back
// (210 to 240 TFLOPS, by the clock), 690 between inputs that change (199); 2317 x 6252 x 516 338 -> 92, 1636 x 116 x 4084 62 -> 23, 459 x 349 x 4636 70 -> 24; 9019
// random shapes that take this kernel 0.40 in the geometric mean.  Pieces with scales of their own and four conversion stages
// (14 or more slots a pair): 3 % longer at 128 columns, 4 at 96, 7 at 32.
// Earlier forms at 4096^3, TN = 128, with pieces at their own size (658 in the end): hand-overs by .release.cluster arrives and a
// cluster fence 1279; one issuing warp 707; three groups of converters (whose registers the sums then lack) 691; all warps polling for
// themselves 680; turns of one chunk the same, but 953 at TN = 64 against 833.
//
// Numbers that the split cannot serve are multiplied as they are, with fused multiply-adds in K order: a warp whose sums
// are not all finite (an infinity, a NaN, or an overflow on the way, which the scale brings to about 2^96;
// x - h of an infinity is a NaN, so none goes unseen) does its 32 x TN / 2 outputs again, see f32_tile_as_defined.  Whoever
// waits for such a tile waits 0.15 us per element of K at most, under 2.5 s where the operands of more tiles than pairs fill 180 GB.
#pragma once

constexpr uint32_t kF32M = 256;
constexpr uint32_t kF32Chunk = 32;                       // floats of K
constexpr int kF32Threads = 640;
constexpr int kF32Groups = 2;                            // of four converter warps
constexpr int kF32FirstSum = 4 + 4 * kF32Groups;
constexpr int kF32SumWarps = 8;
constexpr uint32_t kF32LaunchRegs = 96;                  // a thread of the block is launched with
constexpr uint32_t kF32BoxLd = 20;                       // floats per row of a warp's 32 x 16 staging box
constexpr float kF32Scale = 0x1p16f;                     // of the elements of A and of B
constexpr float kF32Unscale = 0x1p-32f;                  // of the sums, when they leave the registers

// A wait tells the last two phases of a barrier apart, no more: whoever waits for one has to know that the phase before it is
// complete, and those who take turns know that only of what they have waited for themselves.
//  * A group of converters comes to every second chunk: raw stages in an even number, so that a stage is always the same group's.
//  * Converted stages may be an odd number, since their barriers are not the stage's but come round after kF32Bars chunks.  An issuing
//    warp, whose turns are of one chunk at the end of a range, has waited for a chunk of either group among the six before.
//    Nobody arrives for a chunk before the barrier's phase before is complete: a chunk is converted when the one conv_stages in front
//    has been consumed, whose group had seen the same, and so on back.
//  * An issuing warp waits for an accumulator at every second turn, and all accumulators are given back in the order of the turns.
// With a barrier for each of five (or seven) stages a late load or a late converter let the other group's or warp's wait end a round
// too early.  (160 random shapes: 0.985 of that form's time at 32 and 96 columns, 0.995 at 64, 1.005 at 128; barriers of the raw stages that
// come round after 16 chunks as well 1.01 at 128 and 1.015 at 96.)
constexpr uint32_t kF32Bars = 16;
static_assert(kF32Bars % kF32Groups == 0 && kF32Bars >= 6, "waits that cannot end a round too early");

template <uint32_t TN> struct F32Tile {
    static constexpr uint32_t half_n = TN / 2;
    static constexpr uint32_t a_bytes = 128 * 128;
    static constexpr uint32_t raw_bytes = a_bytes + half_n * 128;
    static constexpr uint32_t plane_bytes = half_n * 64;
    static constexpr uint32_t a_cols = 48;                               // h, m, l of 32 floats: 16 columns each
    static constexpr uint32_t conv_stages = TN == 96 ? 4 : 5;             // what tensor memory has room for
    static constexpr uint32_t accs = TN <= 64 ? 4 : TN == 96 ? 3 : 2;
    static constexpr uint32_t raw_stages = TN <= 64 ? 8 : 6;
    static constexpr uint32_t tmem_cols = accs * TN + conv_stages * a_cols > 256 ? 512 : 256;
    static_assert(accs * TN + conv_stages * a_cols <= 512, "tensor memory");
    static_assert(raw_stages % kF32Groups == 0 && 2 * conv_stages <= kF32Bars, "see kF32Bars");
    static constexpr uint32_t box_bytes = 32 * kF32BoxLd * 4;
    // registers a thread of the issuing, the converting and the adding warps; at 64 columns 72 and 152 take 7 % longer
    static constexpr uint32_t issue_regs = 32, converter_regs = 80, sum_regs = 144;
    static_assert(128 * issue_regs + 128 * kF32Groups * converter_regs + 32 * kF32SumWarps * sum_regs <= kF32Threads * kF32LaunchRegs,
                  "no share may wait for registers that nobody gives back");
    static constexpr size_t smem_bytes = (size_t)raw_stages * raw_bytes + conv_stages * 3 * plane_bytes + kF32SumWarps * box_bytes + 512 + 1024;
};

struct F32Smem {
    uint64_t raw_full[8], raw_empty[8];
    uint64_t conv_full[kF32Bars], conv_empty[kF32Bars];
    uint64_t d_full[4], d_empty[4];
    uint32_t tmem_base;
};
static_assert(sizeof(F32Smem) <= 512, "the room that F32Tile leaves for it");

// Parity of a chunk's phase.  Below zero that is the phase in front of a fresh barrier's, which counts as complete.
__device__ __forceinline__ uint32_t chunk_parity(uint32_t chunk) { return chunk / kF32Bars & 1; }

struct F32Maps {
    CUtensorMap a, b;
};
struct F32Params {
    uint32_t m, n, k;
    uint32_t tiles_m, tiles_n, group;
    uint32_t chunks, splits;
    const float *a, *b;
    float *c;
    float alpha;
    uint32_t *status;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&b);
}
// (h - x) of a bf16 pair and two floats
__device__ __forceinline__ void bf16x2_minus(uint32_t h, float x0, float x1, float &d0, float &d1)
{
    asm("{\n\t"
        ".reg .b16 lo, hi;\n\t"
        "mov.b32 {lo, hi}, %2;\n\t"
        "sub.rn.f32.bf16 %0, lo, %3;\n\t"
        "sub.rn.f32.bf16 %1, hi, %4;\n\t"
        "}"
        : "=f"(d0), "=f"(d1)
        : "r"(h), "f"(x0), "f"(x1));
}
// two floats times a power of two, of either sign
__device__ __forceinline__ void scale_pair(float &x0, float &x1, float by)
{
    asm("{\n\t"
        ".reg .b64 x, f;\n\t"
        "mov.b64 x, {%0, %1};\n\t"
        "mov.b64 f, {%2, %2};\n\t"
        "mul.rn.f32x2 x, x, f;\n\t"
        "mov.b64 {%0, %1}, x;\n\t"
        "}"
        : "+f"(x0), "+f"(x1)
        : "f"(by));
}

// Two floats -> the three bf16 pairs h, -m and l of their products with kF32Scale (bf16x2_minus leaves the other sign).
__device__ __forceinline__ void split_bf16x3(float x0, float x1, uint32_t &h, uint32_t &minus_m, uint32_t &l)
{
    float r0, r1, s0, s1;
    scale_pair(x0, x1, kF32Scale);
    h = pack_bf16x2(x0, x1);
    bf16x2_minus(h, x0, x1, r0, r1);
    minus_m = pack_bf16x2(r0, r1);
    bf16x2_minus(minus_m, r0, r1, s0, s1);
    l = pack_bf16x2(s0, s1);
}

// D = A B or D + A B
__device__ __forceinline__ void mma2_bf16_ts(uint32_t d, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(d),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate ? 1 : 0)
        : "memory");
}

template <bool INC, uint32_t N>
__device__ __forceinline__ void set_max_registers()
{
    if constexpr (INC)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    else
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// 2-D tile load into this CTA's shared memory, its bytes counted by this CTA's barrier
__device__ __forceinline__ void tma_load_own(void *smem_dst, const CUtensorMap *tmap, int32_t x, int32_t y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

template <int THREADS>
__device__ __forceinline__ void named_barrier(uint32_t barrier)
{
    asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(barrier), "n"(THREADS) : "memory");
}

// Lane 0 waits for one barrier, lane 1 for another, and the warp for both.  (A poll costs the shared-memory pipe as many
// turns as lanes take part.)
__device__ __forceinline__ bool warp_wait_two(uint64_t *bar0, uint32_t parity0, uint64_t *bar1, uint32_t parity1)
{
    const uint32_t lane = threadIdx.x & 31;
    uint64_t t0 = 0;                                                     // a read of the timer costs as much as the wait
    for (uint32_t spins = 1;; spins++) {
        uint32_t ok = 1;
        if (lane < 2)
            ok = mbar_try_wait(lane == 0 ? bar0 : bar1, lane == 0 ? parity0 : parity1);
        if (__all_sync(0xffffffffu, ok))
            return true;
        if ((spins & 0x3ff) == 0) {
            const uint64_t now = globaltimer_ns();
            if (t0 == 0)
                t0 = now;
            if (__any_sync(0xffffffffu, now - t0 > kWaitBudgetNs))
                return false;
        }
    }
}
__device__ __forceinline__ bool warp_wait_one(uint64_t *bar, uint32_t parity) { return warp_wait_two(bar, parity, bar, parity); }

// The first warp of a team has waited for all of it; the others stand at a barrier meanwhile, where they take no issue slots
// from the converters (with 20 warps polling a chunk took twice as long).
template <int THREADS>
__device__ __forceinline__ bool team_agrees(uint32_t barrier, bool ok)
{
    uint32_t all;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.aligned.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(all)
        : "r"(ok ? 1u : 0u), "r"(barrier), "n"(THREADS)
        : "memory");
    return all != 0;
}

// The sums of the warps with AGAIN once more, as they are defined: fused multiply-adds over k0 ... k1 in order.  All the warps
// that hold sums call this at the same time and bring their CTA's rows of A and B, eight k at a time, into their boxes (`room`): [k][row of A], [k][row of B],
// four floats between.  A lane computes eight rows x pairs of columns 16 apart of its warp's 32 x TN / 2 sums and hands them to the
// lanes that hold the rows through the warp's box, 16 columns at a time.  A sum that is a NaN stays one, and a tile without
// others ends early.  Beyond K are zeros on both sides; what lies beyond C is computed and not stored.
//
// Bound by latency: two warps per scheduler, the fp32 pipe half busy; 128 x 128 x 4096 take 620 us, 500 where few warps take part.
// Before, each lane streamed its own row of A, again for every second column: 4096^3 with one NaN in A 5.0 -> 1.1 ms, one in every
// 128 rows 23.8 -> 4.1, A all NaN 40.4 -> 0.6, results beyond the range (now 2^96) throughout 40.4 -> 4.9; the CUDA-core kernel takes 2.3 for each.
// Fragments loaded one k ahead, steps of 16 k and fewer polls by the waiting warps changed nothing, scalar multiply-adds
// took 1.3 times as long.
template <uint32_t TN, bool AGAIN>
__device__ __forceinline__ void f32_tile_as_defined(float (&sum)[TN / 2], float *room, const F32Params &p, uint32_t row0, uint32_t col0, uint32_t k0, uint32_t k1)
{
    constexpr uint32_t kStep = 8, kLdA = 128 + 4, kLdB = TN + 4, kBuffer = kStep * (kLdA + kLdB), kPairs = TN / 32;
    static_assert(2 * kBuffer * sizeof(float) <= kF32SumWarps * F32Tile<TN>::box_bytes, "two steps fit the boxes");
    uint32_t t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));                       // read here, so that nothing below is kept in registers before
    t -= 32 * kF32FirstSum;
    const uint32_t line = t >> 1, part = 4 * (t & 1);
    const uint32_t warp = t >> 5, lane = t & 31, lane_row = lane >> 3, lane_col = lane & 7;
    const bool in_a = row0 + line < p.m, in_b = line < TN && col0 + line < p.n;
    const float *pa = p.a + (uint64_t)(in_a ? row0 + line : 0) * p.k + part, *pb = p.b + (uint64_t)(in_b ? col0 + line : 0) * p.k + part;
    float4 xa, xb;
    auto fetch = [&](uint32_t k) {
        const bool in_k = k + part < k1;                                  // K is a multiple of 4
        xa = in_a && in_k ? *reinterpret_cast<const float4 *>(pa + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        xb = in_b && in_k ? *reinterpret_cast<const float4 *>(pb + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    unsigned long long acc[8][kPairs];
#pragma unroll
    for (uint32_t i = 0; i < 8; i++)
#pragma unroll
        for (uint32_t j = 0; j < kPairs; j++)
            acc[i][j] = 0ull;
    fetch(k0);
    uint32_t buffer = 0;
    bool settled = !AGAIN;
#pragma unroll 1
    for (uint32_t k = k0; k < k1; k += kStep, buffer ^= 1) {
        if ((k - k0) % (32 * kStep) == kStep) {
            if constexpr (AGAIN) {
                bool nan = true;
#pragma unroll
                for (uint32_t i = 0; i < 8 * kPairs; i++) {
                    float2 v;
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(acc[i / kPairs][i % kPairs]));
                    nan = nan && isnan(v.x) && isnan(v.y);
                }
                settled = __all_sync(0xffffffffu, nan);
            }
            if (team_agrees<32 * kF32SumWarps>(1, settled))
                break;
        }
        float *sa = room + buffer * kBuffer, *sb = sa + kStep * kLdA;
        float *to = sa + part * kLdA + line;
        to[0] = xa.x, to[kLdA] = xa.y, to[2 * kLdA] = xa.z, to[3 * kLdA] = xa.w;
        if (line < TN) {
            to = sb + part * kLdB + line;
            to[0] = xb.x, to[kLdB] = xb.y, to[2 * kLdB] = xb.z, to[3 * kLdB] = xb.w;
        }
        if (k + kStep < k1)
            fetch(k + kStep);
        named_barrier<32 * kF32SumWarps>(1);
        if constexpr (!AGAIN)
            continue;
        const float *fa = sa + 32 * (warp & 3) + 4 * lane_row, *fb = sb + (warp >> 2) * (TN / 2) + 2 * lane_col;
#pragma unroll
        for (uint32_t kk = 0; kk < kStep; kk++) {
            unsigned long long y[kPairs];
#pragma unroll
            for (uint32_t j = 0; j < kPairs; j++)
                y[j] = *reinterpret_cast<const unsigned long long *>(fb + kk * kLdB + 16 * j);
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                const float4 x = *reinterpret_cast<const float4 *>(fa + kk * kLdA + 16 * h);
                const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    unsigned long long xx;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(xs[i]));
#pragma unroll
                    for (uint32_t j = 0; j < kPairs; j++)
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[4 * h + i][j]) : "l"(xx), "l"(y[j]));
                }
            }
        }
    }
    named_barrier<32 * kF32SumWarps>(1);                                  // the boxes are the warps' own again
    if constexpr (!AGAIN)
        return;
    float *box = room + warp * (F32Tile<TN>::box_bytes / 4);
#pragma unroll
    for (uint32_t j = 0; j < kPairs; j++) {
#pragma unroll
        for (uint32_t i = 0; i < 8; i++)
            *reinterpret_cast<unsigned long long *>(box + (4 * lane_row + 16 * (i >> 2) + (i & 3)) * kF32BoxLd + 2 * lane_col) = acc[i][j];
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const float4 v = *reinterpret_cast<const float4 *>(box + lane * kF32BoxLd + 4 * i);
            sum[16 * j + 4 * i] = v.x, sum[16 * j + 4 * i + 1] = v.y, sum[16 * j + 4 * i + 2] = v.z, sum[16 * j + 4 * i + 3] = v.w;
        }
        __syncwarp();
    }
}

template <uint32_t TN>
__global__ void __launch_bounds__(kF32Threads, 1) gemm_f32_kernel(const __grid_constant__ F32Maps maps, F32Params p)
{
    using T = F32Tile<TN>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *planes = smem + (size_t)T::raw_stages * T::raw_bytes;
    uint8_t *boxes = planes + (size_t)T::conv_stages * 3 * T::plane_bytes;
    F32Smem *sh = reinterpret_cast<F32Smem *>(boxes + kF32SumWarps * T::box_bytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank(), r = rank & 1, leader = rank & ~1u, split = rank >> 1;
    const uint32_t cluster_id = blockIdx.x / (2 * p.splits), n_clusters = gridDim.x / (2 * p.splits);
    const uint32_t n_tiles = p.tiles_m * p.tiles_n;
    const uint32_t c0 = (uint32_t)((uint64_t)split * p.chunks / p.splits), c1 = (uint32_t)((uint64_t)(split + 1) * p.chunks / p.splits);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < T::raw_stages; s++) {
            mbar_init(&sh->raw_full[s], 1);
            mbar_init(&sh->raw_empty[s], 4);
        }
        for (uint32_t i = 0; i < kF32Bars; i++) {
            mbar_init(&sh->conv_full[i], 2 * 4);
            mbar_init(&sh->conv_empty[i], 1);
        }
        for (uint32_t d = 0; d < T::accs; d++) {
            mbar_init(&sh->d_full[d], 1);
            mbar_init(&sh->d_empty[d], 2 * kF32SumWarps);
        }
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1)
        tmem_alloc<2>(&sh->tmem_base, T::tmem_cols);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    tc_fence_after_sync();
    const uint32_t tmem = sh->tmem_base;
    griddep_wait();                        // see join_previous_launch
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *p.status = 0u;
    griddep_launch_dependents();
    auto give_up = [&](uint32_t code) {
        if (lane == 0)
            atomicCAS(p.status, 0u, code);
    };

    if (warp < 4)
        set_max_registers<false, T::issue_regs>();
    if (warp == 0) {
        // ---------------- TMA producer ----------------
        uint32_t s = 0, parity = 1;
        bool ok = true;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            uint32_t mb, nb;
            dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
            const int32_t row_a = (int32_t)(mb * kF32M + r * 128), row_b = (int32_t)(nb * TN + r * T::half_n);
            for (uint32_t c = c0; c < c1; c++) {
                if (!warp_wait_one(&sh->raw_empty[s], parity)) {
                    give_up(0x231u);
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    uint8_t *st = smem + (size_t)s * T::raw_bytes;
                    mbar_expect_tx(&sh->raw_full[s], T::raw_bytes);
                    tma_load_own(st, &maps.a, (int32_t)(c * 128), row_a, &sh->raw_full[s]);
                    tma_load_own(st + T::a_bytes, &maps.b, (int32_t)(c * 128), row_b, &sh->raw_full[s]);
                }
                __syncwarp();
                if (++s == T::raw_stages) {
                    s = 0;
                    parity ^= 1;
                }
            }
        }
    } else if (warp < 3) {
        // ---------------- MMA issuers (the pair's leader), every other turn each ----------------
        if (r == 0) {
            const uint32_t idesc = make_idesc(256, TN, kFmtBF16, kFmtBF16, kAccF32), idesc_minus = idesc | kNegateA;
            const uint16_t pair_mask = (uint16_t)(3u << leader);
            uint32_t turn = 0, chunk = 0;
            bool ok = true;
            for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
                for (uint32_t c = c0; c < c1; c += 2, turn++, chunk += 2) {
                    const bool two = c + 1 < c1;
                    if ((turn & 1) == (uint32_t)warp - 1) {
                        const uint32_t d = turn % T::accs, s0 = chunk % T::conv_stages, s1 = (chunk + 1) % T::conv_stages;
                        const uint32_t bar0 = chunk % kF32Bars, bar1 = (chunk + 1) % kF32Bars;
                        // a fresh barrier's preceding phase counts as complete
                        if (!warp_wait_two(&sh->d_empty[d], (turn / T::accs + 1) & 1, &sh->conv_full[bar0], chunk_parity(chunk)) ||
                            (two && !warp_wait_one(&sh->conv_full[bar1], chunk_parity(chunk + 1)))) {
                            give_up(0x233u);
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        if (elect_one()) {
                            const uint32_t acc = tmem + d * TN;
                            // plane pa of A times plane pb of B of the chunk in stage s
                            auto multiply = [&](uint32_t s, uint32_t pa, uint32_t pb, bool accumulate = true) {
                                const uint32_t a = tmem + T::accs * TN + s * T::a_cols + 16 * pa;
                                const uint64_t b = make_smem_desc(smem_u32(planes + (size_t)s * 3 * T::plane_bytes), 16, 512, kSwizzle64B) +
                                                   pb * T::plane_bytes / 16;
                                const uint32_t desc = (pa == 1) != (pb == 1) ? idesc_minus : idesc;        // one factor is -m
                                mma2_bf16_ts(acc, a, b, desc, accumulate);
                                mma2_bf16_ts(acc, a + 8, b + 2, desc, true);
                            };
                            // the smallest products first, those of full size last
                            multiply(s0, 2, 0, false);
                            multiply(s0, 0, 2);
                            multiply(s0, 1, 1);
                            if (two) {
                                multiply(s1, 2, 0);
                                multiply(s1, 0, 2);
                                multiply(s1, 1, 1);
                            }
                            multiply(s0, 1, 0);
                            multiply(s0, 0, 1);
                            if (two) {
                                multiply(s1, 1, 0);
                                multiply(s1, 0, 1);
                            }
                            multiply(s0, 0, 0);
                            tc_commit_pair(&sh->conv_empty[bar0], pair_mask);
                            if (two) {
                                multiply(s1, 0, 0);
                                tc_commit_pair(&sh->conv_empty[bar1], pair_mask);
                            }
                            tc_commit_pair(&sh->d_full[d], pair_mask);
                        }
                        __syncwarp();
                    }
                    if (!two)
                        chunk--;                                          // the turn had one chunk
                }
            }
        }
    } else if (warp >= 4 && warp < kF32FirstSum) {
        // ---------------- converters: groups of four warps that take turns at the chunks; a row of A per lane, and eight floats of
        // B per lane and step ----------------
        set_max_registers<false, T::converter_regs>();
        const uint32_t cw = (uint32_t)warp & 3, group = (uint32_t)(warp - 4) >> 2;
        const uint32_t full0 = cluster_addr(&sh->conv_full[0], leader);
        uint32_t count = 0;
        bool ok = true;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            for (uint32_t c = c0; c < c1; c++, count++) {
                if (count % kF32Groups != group)
                    continue;
                const uint32_t raw = count % T::raw_stages, s = count % T::conv_stages;
                const bool there = cw != 0 || warp_wait_two(&sh->raw_full[raw], (count / T::raw_stages) & 1,
                                                            &sh->conv_empty[(count - T::conv_stages) % kF32Bars], chunk_parity(count - T::conv_stages));
                if (!team_agrees<128>(2 + group, there)) {
                    give_up(0x234u);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint8_t *st = smem + (size_t)raw * T::raw_bytes;
                uint8_t *dst = planes + (size_t)s * 3 * T::plane_bytes;
                // warp cw takes the 32 steps of eight floats of B cw, cw + 4
                constexpr uint32_t kSteps = T::half_n / 8;
                const uint32_t g = lane & 3;
                auto step_row = [&](uint32_t i) { return ((cw + 4 * i) * 32 + lane) >> 2; };
                float4 xb[2][2];
#pragma unroll
                for (uint32_t i = 0; i < 2; i++)
                    if (4 * i < kSteps && cw + 4 * i < kSteps) {
                        const uint8_t *src = st + T::a_bytes + step_row(i) * 128;
                        xb[i][0] = *reinterpret_cast<const float4 *>(src + (((2 * g) ^ (step_row(i) & 7)) << 4));
                        xb[i][1] = *reinterpret_cast<const float4 *>(src + (((2 * g + 1) ^ (step_row(i) & 7)) << 4));
                    }
                const uint32_t row = cw * 32 + lane;
#pragma unroll
                for (uint32_t kk = 0; kk < 2; kk++) {
                    float4 xa[4];
#pragma unroll
                    for (uint32_t j = 0; j < 4; j++)
                        xa[j] = *reinterpret_cast<const float4 *>(st + row * 128 + (((4 * kk + j) ^ (row & 7)) << 4));
                    if (4 * kk < kSteps && cw + 4 * kk < kSteps) {
                        uint4 h, m, l;
                        split_bf16x3(xb[kk][0].x, xb[kk][0].y, h.x, m.x, l.x);
                        split_bf16x3(xb[kk][0].z, xb[kk][0].w, h.y, m.y, l.y);
                        split_bf16x3(xb[kk][1].x, xb[kk][1].y, h.z, m.z, l.z);
                        split_bf16x3(xb[kk][1].z, xb[kk][1].w, h.w, m.w, l.w);
                        uint8_t *at = dst + step_row(kk) * 64 + ((g ^ ((step_row(kk) >> 1) & 3)) << 4);
                        *reinterpret_cast<uint4 *>(at) = h;
                        *reinterpret_cast<uint4 *>(at + T::plane_bytes) = m;
                        *reinterpret_cast<uint4 *>(at + 2 * T::plane_bytes) = l;
                    }
                    uint32_t h[8], m[8], l[8];
#pragma unroll
                    for (uint32_t j = 0; j < 4; j++) {
                        split_bf16x3(xa[j].x, xa[j].y, h[2 * j], m[2 * j], l[2 * j]);
                        split_bf16x3(xa[j].z, xa[j].w, h[2 * j + 1], m[2 * j + 1], l[2 * j + 1]);
                    }
                    const uint32_t taddr = tmem + T::accs * TN + s * T::a_cols + 8 * kk + ((cw * 32) << 16);
                    tmem_st_32x32b_x8(taddr, h);
                    tmem_st_32x32b_x8(taddr + 16, m);
                    tmem_st_32x32b_x8(taddr + 32, l);
                }
                tmem_st_wait();
                tc_fence_before_sync();
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sh->raw_empty[raw]);
                    mbar_arrive_remote(full0 + 8 * (count % kF32Bars));
                }
            }
        }
    }

    if (warp < kF32FirstSum) {
        if (p.splits > 1) {                // the two meetings of the sum warps' exchange
            __syncwarp();
            cluster_sync();
            cluster_sync();
        }
    } else {
        // ---------------- sums: 32 rows x TN / 2 columns per warp ----------------
        set_max_registers<true, T::sum_regs>();
        const uint32_t q = (uint32_t)warp & 3, half = (uint32_t)(warp - kF32FirstSum) >> 2;
        float *box = reinterpret_cast<float *>(boxes + (size_t)(warp - kF32FirstSum) * T::box_bytes);
        const uint32_t own4 = T::half_n / 4 / p.splits;                   // groups of four columns that this pair stores
        auto owner_of = [&](uint32_t g) { return g * p.splits / (T::half_n / 4); };
        uint32_t count = 0;
        bool ok = true;
        for (uint32_t tile = cluster_id; tile < n_tiles && ok; tile += n_clusters) {
            uint32_t mb, nb;
            dense_tile_coords(tile, p.tiles_m, p.tiles_n, p.group, mb, nb);
            const uint32_t row0 = mb * kF32M + r * 128 + q * 32, col0 = nb * TN + half * T::half_n;
            float sum[T::half_n];
#pragma unroll
            for (uint32_t i = 0; i < T::half_n; i++)
                sum[i] = 0.0f;
            for (uint32_t c = c0; c < c1; c += 2, count++) {              // a turn
                const uint32_t d = count % T::accs;
                const bool there = warp != kF32FirstSum || warp_wait_one(&sh->d_full[d], (count / T::accs) & 1);
                if (!team_agrees<32 * kF32SumWarps>(1, there)) {
                    give_up(0x236u);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t taddr = tmem + d * TN + half * T::half_n + ((q * 32) << 16);
                auto add16 = [&](uint32_t g, const uint32_t (&v)[16]) {
#pragma unroll
                    for (uint32_t i = 0; i < 16; i++)
                        sum[16 * g + i] += __uint_as_float(v[i]);
                };
                auto release = [&]() {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster_relaxed(&sh->d_empty[d], leader);
                };
                // all at once
                constexpr uint32_t kLoads = T::half_n / 16, kRound = kLoads;
#pragma unroll
                for (uint32_t g = 0; g < kLoads; g += kRound) {
                    uint32_t v[kRound][16];
#pragma unroll
                    for (uint32_t i = 0; i < kRound; i++)
                        if (g + i < kLoads)
                            tmem_ld_32x32b_x16(taddr + 16 * (g + i), v[i]);
                    tmem_ld_wait();
                    if (g + kRound >= kLoads)
                        release();
#pragma unroll
                    for (uint32_t i = 0; i < kRound; i++)
                        if (g + i < kLoads)
                            add16(g + i, v[i]);
                }
            }
            if (ok) {
                float probe = 0.0f;                                       // not finite: 0 x = NaN
#pragma unroll
                for (uint32_t i = 0; i < T::half_n; i++) {
                    probe = fmaf(sum[i], 0.0f, probe);
                    sum[i] *= kF32Unscale;
                }
                if (!team_agrees<32 * kF32SumWarps>(1, probe == 0.0f)) {
                    const uint32_t k1 = c1 * kF32Chunk < p.k ? c1 * kF32Chunk : p.k;
                    const uint32_t first_row = mb * kF32M + r * 128;
                    if (__any_sync(0xffffffffu, probe != 0.0f))
                        f32_tile_as_defined<TN, true>(sum, reinterpret_cast<float *>(boxes), p, first_row, nb * TN, c0 * kF32Chunk, k1);
                    else
                        f32_tile_as_defined<TN, false>(sum, reinterpret_cast<float *>(boxes), p, first_row, nb * TN, c0 * kF32Chunk, k1);
                }
            }
            if (p.splits > 1) {
                // Every pair's instructions have retired and its raw tiles are read, so their room takes partial sums:
                // [pair that sends, without the owner][half][group of four columns][128 rows][4 floats]
                __syncwarp();
                cluster_sync();
                const uint32_t at = (q * 32 + lane) * 16;
#pragma unroll
                for (uint32_t g = 0; g < T::half_n / 4; g++) {
                    const uint32_t owner = owner_of(g);
                    if (owner != split) {
                        const uint32_t src = split < owner ? split : split - 1;
                        const uint32_t slot = ((src * 2 + half) * own4 + g - owner * own4) * 2048 + at;
                        st_cluster_v4(cluster_addr(smem, owner * 2 + r) + slot, __float_as_uint(sum[4 * g]), __float_as_uint(sum[4 * g + 1]),
                                      __float_as_uint(sum[4 * g + 2]), __float_as_uint(sum[4 * g + 3]));
                    }
                }
                __syncwarp();
                cluster_sync();
#pragma unroll
                for (uint32_t g = 0; g < T::half_n / 4; g++) {
                    if (owner_of(g) == split) {
                        float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        for (uint32_t src = 0; src < p.splits; src++) {
                            float4 v = make_float4(sum[4 * g], sum[4 * g + 1], sum[4 * g + 2], sum[4 * g + 3]);
                            if (src != split)
                                v = *reinterpret_cast<const float4 *>(smem + (((src < split ? src : src - 1) * 2 + half) * own4 + g - split * own4) * 2048 + at);
                            t = src == 0 ? v : make_float4(t.x + v.x, t.y + v.y, t.z + v.z, t.w + v.w);
                        }
                        sum[4 * g] = t.x;
                        sum[4 * g + 1] = t.y;
                        sum[4 * g + 2] = t.z;
                        sum[4 * g + 3] = t.w;
                    }
                }
            }
            if (ok) {
                // 16 columns at a time through the warp's box, so that a row's 64 bytes leave together: in four pieces where rows
                // of C are aligned for that, else element by element
                const bool vec = p.n % 4 == 0;
                const uint32_t rr = vec ? lane >> 2 : lane >> 4, cc = vec ? 4 * (lane & 3) : lane & 15;
                float *out = p.c + (uint64_t)(row0 + rr) * p.n + col0 + cc;
#pragma unroll
                for (uint32_t g = 0; g < T::half_n / 16; g++) {
                    __syncwarp();
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++) {
                        const float *v = sum + 16 * g + 4 * i;
                        *reinterpret_cast<float4 *>(box + lane * kF32BoxLd + 4 * i) = make_float4(v[0] * p.alpha, v[1] * p.alpha, v[2] * p.alpha, v[3] * p.alpha);
                    }
                    __syncwarp();
                    const bool mine = col0 + 16 * g + cc < p.n && owner_of(4 * g + cc / 4) == split;
                    if (vec) {
                        float4 v[4];
#pragma unroll
                        for (uint32_t i = 0; i < 4; i++)
                            v[i] = *reinterpret_cast<const float4 *>(box + (8 * i + rr) * kF32BoxLd + cc);
#pragma unroll
                        for (uint32_t i = 0; i < 4; i++)
                            if (mine && row0 + 8 * i + rr < p.m)
                                *reinterpret_cast<float4 *>(out + (uint64_t)(8 * i) * p.n + 16 * g) = v[i];
                    } else {
#pragma unroll 4
                        for (uint32_t i = 0; i < 16; i++)
                            if (mine && row0 + 2 * i + rr < p.m)
                                out[(uint64_t)(2 * i) * p.n + 16 * g] = box[(2 * i + rr) * kF32BoxLd + cc];
                    }
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    if (warp == 1)
        tmem_dealloc<2>(tmem, T::tmem_cols);
}
