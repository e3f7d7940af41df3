// Seeded operand generation, format conversion and block-scaled FP4 quantisation.
//
// Eight consecutive elements per thread and step, moved with the widest access their type and alignment allow.  The
// elements in front of the first aligned address, and those left over at the end, go one at a time.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <math.h>

#include "../clpk_internal.h"
#include "../clpk_ptx.cuh"
#include "../clpk_rng_fast.cuh"
#include "../clpk_formats.h"

namespace clpk {

constexpr int kFillThreads = 256;

// every kernel here is launched behind the one before it in the stream (launch_behind)
__device__ __forceinline__ void join_stream()
{
    griddep_wait();
    griddep_launch_dependents();
}

// Which way the CTAs of a kernel that reads an array walk it.  What stands in front has just written or read the same array
// in rising order, and its end is what the L2 (126 MB) still holds: from the end, arrays beyond the cache are read from
// there as far as it reaches.  14997 x 2432 (146 MB) NVFP4 operands 144 -> 138 us, bf16 123 -> 117, 8192 x 8192 (268 MB) 257 ->
// 251 and 222 -> 216.  What fits lies there whichever way it is read, and rising is up to 2 % faster (67 MB: to tf32 57.4
// against 58.6 us).
constexpr uint64_t kFallingFrom = 100ull << 20;
static bool falling_order(uint64_t bytes) { return bytes >= kFallingFrom; }
__device__ __forceinline__ uint64_t ordered_cta(bool falling) { return falling ? gridDim.x - 1 - blockIdx.x : blockIdx.x; }

// An array cut at the first address that is aligned for the wide access: `head` elements, `whole` steps, the rest.  The
// kernels get the aligned address and count from there (with the head added to every index in the loop the normal fill
// took 167 instead of 162 us, aligned or not), so that the head has the indices -head ... -1.  The elements outside the
// steps are fewer than two steps' and go to one thread each of CTA 0 (a loop over them cost int8 0.3 us a launch).
struct Split {
    uint64_t whole;
    uint32_t head, singles;

    __device__ bool has_single() const { return blockIdx.x == 0 && threadIdx.x < singles; }
    // this thread's, in steps of `per`
    __device__ int64_t single(uint32_t per) const
    {
        const int64_t j = (int64_t)threadIdx.x - head;
        return j < 0 ? j : j + (int64_t)(per * whole);
    }
};

struct __align__(32) Float8 {
    float v[8];
};

// 32 bytes, 32-byte aligned: one 256-bit access.  absmax and the quantiser ask for the lines of arrays beyond the cache
// as the first to leave it (FIRST), so that those which come from DRAM do not push out, before they are read, those that the
// kernel in front has left: 8192 x 8192 (268 MB) normal fill with NVFP4 229 -> 220 us, with MXFP4 185 -> 180, 4096 x 8192
// 116 -> 111 and 93 -> 90.  (Conversions gain 1 %, and only through this access.  Letting the fill's first stores go first as well:
// 223; keeping what absmax reads last for the quantiser: 219 to 222.)
template <bool FIRST>
__device__ __forceinline__ Float8 ld_float8x32(const float *p)
{
    unsigned long long w[4];
    if constexpr (FIRST)
        asm volatile("ld.global.L1::no_allocate.L2::evict_first.v4.b64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                     : "l"(p)
                     : "memory");
    else
        asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]) : "l"(p) : "memory");
    Float8 r;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        r.v[2 * i] = lo_of(w[i]);
        r.v[2 * i + 1] = hi_of(w[i]);
    }
    return r;
}

// eight floats from an address that is a multiple of ALIGN bytes
template <int ALIGN, bool FIRST = false>
__device__ __forceinline__ Float8 ld_float8(const float *p)
{
    if constexpr (ALIGN == 32) {
        return ld_float8x32<FIRST>(p);
    } else {
        Float8 r;
        if constexpr (ALIGN == 16) {
            const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
            r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
            r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++)
                r.v[i] = p[i];
        }
        return r;
    }
}

// the first PER of the eight
template <int PER, int ALIGN>
__device__ __forceinline__ Float8 ld_floats(const float *p)
{
    if constexpr (PER == 8) {
        return ld_float8<ALIGN>(p);
    } else {
        static_assert(PER == 4, "four or eight");
        Float8 r = {};
        if constexpr (ALIGN >= 16) {
            const float4 a = *reinterpret_cast<const float4 *>(p);
            r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
        } else {
#pragma unroll
            for (int i = 0; i < PER; i++)
                r.v[i] = p[i];
        }
        return r;
    }
}

__device__ __forceinline__ void st_float8(float *p, f32x2 a, f32x2 b, f32x2 c, f32x2 d)
{
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// Bound by arithmetic: see clpk_rng_fast.cuh.  Eight elements per thread and step, and two steps where the array is long
// enough to fill the chip all the same: at 2^28 floats 536 against 548 us (normal) and 191 against 268 (uniform, bound by the
// start of CTAs with one step), the same at 2^22, and one step is better below (normal, 2^20: 3.4 against 4.3).  8192 x 8192:
// normal 160 -> 136 us, uniform 62 -> 49 (the stores alone would take 41), int8 55 -> 47.
constexpr int kFillF32Threads = 128;
constexpr uint64_t kTwoStepsFrom = 1 << 19;

template <int DIST>
__global__ void __launch_bounds__(kFillF32Threads, 8) fill_f32_kernel(float *dst, Split part, uint64_t base, uint32_t steps, float mean, float stdv)
{
    griddep_launch_dependents();                               // the stores wait, the values need no memory
    // the 2 P values of the words
    auto values = [&](const auto &hi, const auto &lo, auto &out) {
        constexpr int P = sizeof(out) / sizeof(f32x2);
        if constexpr (DIST == CLPK_DIST_NORMAL)
            normal01<P>(hi, lo, out);
#pragma unroll
        for (int j = 0; j < P; j++) {
            const f32x2 u = pk((float)(hi[2 * j] >> 8), (float)(hi[2 * j + 1] >> 8));
            if constexpr (DIST == CLPK_DIST_NORMAL)
                out[j] = fma2(pk(stdv), out[j], pk(mean));
            else if constexpr (DIST == CLPK_DIST_UNIFORM01)
                out[j] = mul2(u, pk(5.9604644775390625e-08f));
            else
                out[j] = add2(mul2(u, pk(1.1920928955078125e-07f)), pk(-1.0f));
        }
    };
    uint64_t g = (uint64_t)blockIdx.x * (steps * kFillF32Threads) + threadIdx.x;
#pragma unroll 1
    for (uint32_t step = 0; step < steps && g < part.whole; step++, g += kFillF32Threads) {
        uint32_t hi[8], lo[8];
        random_words<8>(base + 8 * g, hi, lo);
        f32x2 v[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t hi4[4] = {hi[4 * h], hi[4 * h + 1], hi[4 * h + 2], hi[4 * h + 3]}, lo4[4] = {lo[4 * h], lo[4 * h + 1], lo[4 * h + 2], lo[4 * h + 3]};
            f32x2 o[2];
            values(hi4, lo4, o);
            v[2 * h] = o[0];
            v[2 * h + 1] = o[1];
        }
        griddep_wait();
        st_float8(dst + 8 * g, v[0], v[1], v[2], v[3]);
    }
    if (part.has_single()) {
        const int64_t i = part.single(8);
        uint32_t hi[2], lo[2];
        random_words<2>(base + i, hi, lo);
        f32x2 v[1];
        values(hi, lo, v);
        griddep_wait();
        dst[i] = lo_of(v[0]);
    }
}

__global__ void __launch_bounds__(kFillThreads) fill_i8_kernel(int8_t *dst, Split part, uint64_t base)
{
    griddep_launch_dependents();                               // the stores wait, the values need no memory
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t g = first; g < part.whole; g += stride) {
        uint32_t w[4], hi[16], lo[16];
        random_words<16>(base + 16 * g, hi, lo);
        // The top nibble of each word minus 8, four at a time: n + 0x78 carries out of no byte, and its top bit flipped is n - 8.
        // The kernel is bound by its instructions: 8192 x 8192 48.8 -> 47.0 us against a shift, a subtraction and a mask per byte.
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t top = __byte_perm(__byte_perm(hi[4 * j], hi[4 * j + 1], 0x0073), __byte_perm(hi[4 * j + 2], hi[4 * j + 3], 0x0073), 0x5410);
            w[j] = ((top >> 4 & 0x0F0F0F0Fu) + 0x78787878u) ^ 0x80808080u;
        }
        griddep_wait();
        *reinterpret_cast<uint4 *>(dst + 16 * g) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (part.has_single()) {
        const int64_t i = part.single(16);
        uint32_t hi[1], lo[1];
        random_words<1>(base + i, hi, lo);
        griddep_wait();
        dst[i] = (int8_t)((int)(hi[0] >> 28) - 8);
    }
}

// One element in its narrow format, as bits.
template <int DT>
__device__ __forceinline__ uint64_t narrow(float x)
{
    if constexpr (DT == CLPK_DT_F16) {
        return __half_as_ushort(__float2half_rn(x));
    } else if constexpr (DT == CLPK_DT_BF16) {
        return __bfloat16_as_ushort(__float2bfloat16_rn(x));
    } else if constexpr (DT == CLPK_DT_E4M3) {
        return __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
    } else if constexpr (DT == CLPK_DT_E5M2) {
        return __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E5M2);
    } else if constexpr (DT == CLPK_DT_TF32) {
        // nearest even at bit 13 in integer arithmetic (infinities and NaNs keep their class)
        uint32_t b = __float_as_uint(x);
        if ((b & 0x7F800000u) != 0x7F800000u)
            b += 0xFFFu + ((b >> 13) & 1u);
        return b & 0xFFFFE000u;
    } else if constexpr (DT == CLPK_DT_F64) {
        return (uint64_t)__double_as_longlong((double)x);
    } else if constexpr (DT == CLPK_DT_I8) {
        const int v = __float2int_rn(x);
        return (uint8_t)(int8_t)(v < -128 ? -128 : (v > 127 ? 127 : v));
    } else {
        return clpk_e2m1_encode(x);
    }
}

// two neighbours; the 8-bit floats have an instruction for that
template <int DT>
__device__ __forceinline__ uint64_t narrow2(float x0, float x1)
{
    if constexpr (DT == CLPK_DT_E4M3 || DT == CLPK_DT_E5M2)
        return __nv_cvt_float2_to_fp8x2(make_float2(x0, x1), __NV_SATFINITE, DT == CLPK_DT_E4M3 ? __NV_E4M3 : __NV_E5M2);
    else
        return 0;
}

template <int DT> struct Narrow {
    static constexpr int bits = DT == CLPK_DT_F64 ? 64 : DT == CLPK_DT_TF32 ? 32 : DT == CLPK_DT_F16 || DT == CLPK_DT_BF16 ? 16 : DT == CLPK_DT_E2M1 ? 4 : 8;
    // elements of a step: eight, or four of 64 bits (a step of eight is two 32-byte stores, and behind 4-byte loads took
    // 8.9 us for 2048 x 2048 in L2 against 6.0; aligned 6.35 against 6.1)
    static constexpr int per = bits == 64 ? 4 : 8;
};

// Bound by memory: 4 bytes in and bits / 8 out per element.  8192 x 8192: to fp8 122 -> 50 us (6.7 TB/s), 16 bits
// 129 -> 60, tf32 147 -> 82.
template <int DT, int SRC_ALIGN>
__global__ void __launch_bounds__(kFillThreads) convert_kernel(void *dst, const float *src, Split part, bool falling)
{
    join_stream();
    constexpr int bits = Narrow<DT>::bits, kPer = Narrow<DT>::per;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = ordered_cta(falling) * blockDim.x + threadIdx.x;
    for (uint64_t g = first; g < part.whole; g += stride) {
        const auto x = ld_floats<kPer, SRC_ALIGN>(src + kPer * g);
        constexpr int kWords = (kPer * bits + 63) / 64;
        uint64_t w[kWords];
#pragma unroll
        for (int j = 0; j < kWords; j++)
            w[j] = 0;
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            if constexpr (DT == CLPK_DT_E4M3 || DT == CLPK_DT_E5M2) {
                if ((i & 1) == 0)
                    w[0] |= narrow2<DT>(x.v[i], x.v[i + 1]) << (8 * i);
            } else {
                w[i * bits / 64] |= narrow<DT>(x.v[i]) << (i * bits % 64);
            }
        }
        uint8_t *p = static_cast<uint8_t *>(dst) + g * (kPer * bits / 8);
        if constexpr (bits == 4) {
            *reinterpret_cast<uint32_t *>(p) = (uint32_t)w[0];
        } else if constexpr (bits == 8) {
            *reinterpret_cast<uint64_t *>(p) = w[0];
        } else if constexpr (bits == 16) {
            *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(w[0], w[1]);
        } else {
#pragma unroll
            for (int j = 0; j < kWords; j += 4)
                st_float8(reinterpret_cast<float *>(p + 8 * j), w[j], w[j + 1], w[j + 2], w[j + 3]);
        }
    }
    if constexpr (bits == 4) {
        // two elements a byte: an even number of them, on both sides
        if (part.has_single() && threadIdx.x % 2 == 0) {
            const int64_t i = part.single(kPer);
            static_cast<uint8_t *>(dst)[i / 2] = (uint8_t)(narrow<DT>(src[i]) | (narrow<DT>(src[i + 1]) << 4));
        }
    } else if (part.has_single()) {
        const int64_t i = part.single(kPer);
        const uint64_t v = narrow<DT>(src[i]);
        if constexpr (bits == 8)
            static_cast<uint8_t *>(dst)[i] = (uint8_t)v;
        else if constexpr (bits == 16)
            static_cast<uint16_t *>(dst)[i] = (uint16_t)v;
        else if constexpr (bits == 32)
            static_cast<uint32_t *>(dst)[i] = (uint32_t)v;
        else
            static_cast<uint64_t *>(dst)[i] = v;
    }
}

// Bound by memory (8192 x 8192: 111 -> 40 us, 6.6 TB/s, from any address); a CTA takes four accesses per thread of one
// contiguous range (8 Ki floats), so that the chip walks the array in address order.  SINGLE: one CTA reads everything and
// writes the result itself; otherwise the CTAs meet in an atomicMax on a word that has been cleared.
constexpr int kAbsmaxLoads = 4;

template <bool SINGLE, bool FALLING>
__global__ void __launch_bounds__(kFillThreads) absmax_kernel(float *out, const float *src, Split part)
{
    join_stream();
    float m = 0.0f;
    const uint64_t step = (uint64_t)gridDim.x * kFillThreads * kAbsmaxLoads;
    for (uint64_t g = ordered_cta(FALLING) * kFillThreads * kAbsmaxLoads + threadIdx.x; g < part.whole; g += step) {
        Float8 x[kAbsmaxLoads];
#pragma unroll
        for (int u = 0; u < kAbsmaxLoads; u++)
            x[u] = g + u * kFillThreads < part.whole ? ld_float8x32<FALLING>(src + 8 * (g + u * kFillThreads)) : Float8{};
#pragma unroll
        for (int u = 0; u < kAbsmaxLoads; u++)
#pragma unroll
            for (int i = 0; i < 8; i++)
                m = fmaxf(m, fabsf(x[u].v[i]));
    }
    if (part.has_single())
        m = fmaxf(m, fabsf(src[part.single(8)]));
    // |x| >= 0, so the float ordering equals the ordering of the bit patterns.
    uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    __shared__ uint32_t warp_top[kFillThreads / 32];
    if ((threadIdx.x & 31) == 0)
        warp_top[threadIdx.x >> 5] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < kFillThreads / 32; w++)
            top = max(top, warp_top[w]);
        if (SINGLE)
            *reinterpret_cast<uint32_t *>(out) = top;
        else
            atomicMax(reinterpret_cast<uint32_t *>(out), top);
    }
}

// ---- block-scaled FP4 -------------------------------------------------------------------------------------------------
//
// BLOCK elements share a scale; UE8M0 selects the scale format (power-of-two MX scale) against ue4m3 (NVFP4 scale,
// after the tensor scale).  A lane takes 16 neighbouring elements -- an NVFP4 block -- and BLOCK / 16 lanes share a
// scale.  Bound by memory (4.6 bytes an element) once the two quotients of an element, x / tensor scale and that /
// block scale, are no IEEE division each: both divisors are shared, so each is a multiplication by the divisor's
// reciprocal with the residual correction of clpk_rng_fast.cuh -- done twice for the first, whose exact rounding
// decides ties later; the block scale has four significand bits, so one correction leaves nothing to a tie.  That
// holds while nothing under- or overflows: magnitudes and tensor scales within 2^+-60.  A warp that meets any other
// block (zeros, NaN, infinities) takes the divisions.  NVFP4 codes come from one product with the reciprocal of both divisors, taken
// a little too small and a little too large; a warp for which the two disagree anywhere (an element within 2^-20 of a tie)
// does the quotients.  8192 x 8192: NVFP4 171 -> 44 to 47 us, MXFP4 270 -> 40 to 43; 4096 x 4096, in the L2, with quotients throughout and two
// codes converted at a time 11.2 and 9.5, now 9.2 and 7.2 to 7.8.

// divisor and reciprocal for the whole tensor; plain: outside the range above
struct TensorScale {
    float scale, inv;
    bool plain;
};

__device__ __forceinline__ uint32_t e2m1x2(float x0, float x1)
{
    uint32_t r;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(r)
        : "f"(x0), "f"(x1));
    return r & 0xFFu;
}

// eight of them, the first in the lowest four bits
__device__ __forceinline__ uint32_t e2m1x8(const f32x2 (&x)[4])
{
    uint32_t r;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(r)
        : "f"(lo_of(x[0])), "f"(hi_of(x[0])), "f"(lo_of(x[1])), "f"(hi_of(x[1])), "f"(lo_of(x[2])), "f"(hi_of(x[2])), "f"(lo_of(x[3])), "f"(hi_of(x[3])));
    return r;
}

// x / b from inv = RN(1 / b), correctly rounded (see above)
__device__ __forceinline__ float shared_quotient(float x, float b, float inv)
{
    float q = __fmul_rn(x, inv);
    q = __fmaf_rn(__fmaf_rn(-b, q, x), inv, q);
    return __fmaf_rn(__fmaf_rn(-b, q, x), inv, q);
}

template <bool UE8M0>
__device__ __forceinline__ uint8_t fp4_block_scale(float amax, float *decoded)
{
    uint8_t s;
    if (UE8M0) {
        s = clpk_ue8m0_for_absmax(amax);
        *decoded = clpk_ue8m0_decode(s);
    } else {
        s = __nv_cvt_float_to_fp8(__fdiv_rn(amax, 6.0f), __NV_SATFINITE, __NV_E4M3);
        *decoded = clpk_e4m3_decode(s);
    }
    return s;
}

constexpr int kQuantPerLane = 16;

// eight bytes to any address; the addresses of a launch are all aligned alike
__device__ __forceinline__ void st_codes(uint8_t *p, uint64_t codes)
{
    if ((uintptr_t)p % 8 == 0) {
        *reinterpret_cast<uint64_t *>(p) = codes;
    } else if ((uintptr_t)p % 4 == 0) {
        reinterpret_cast<uint32_t *>(p)[0] = (uint32_t)codes;
        reinterpret_cast<uint32_t *>(p)[1] = (uint32_t)(codes >> 32);
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++)
            p[i] = (uint8_t)(codes >> (8 * i));
    }
}

// ALIGN: 32 when the source is aligned to that and the codes to 8 bytes, else what the source is aligned to, 16 or 4.  The
// blocks lie where they lie, so there is no head to cut off: 8192 x 8192 from a source 16 bytes off 45 to 49 us, 4 bytes
// off 122 (each of 16 loads touches 32 sectors) against 168 to 349 with one thread per block.
template <int BLOCK, bool UE8M0, int ALIGN, bool FIRST>
__global__ void __launch_bounds__(kFillThreads) quantize_fp4_kernel(uint8_t *packed, uint8_t *scales, const float *src, uint64_t n16, TensorScale ts, bool falling)
{
    join_stream();
    constexpr int kLanes = BLOCK / kQuantPerLane;              // lanes of one block
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    // whole warps step together: n16 is a multiple of 4, so a block's lanes are inside or outside as one
    for (uint64_t g0 = ordered_cta(falling) * blockDim.x + (threadIdx.x & ~31u); g0 < n16; g0 += stride) {
        const uint64_t g = g0 + lane;
        const bool inside = g < n16;
        float x[kQuantPerLane] = {};
        if (inside) {
            const Float8 a = ld_float8<ALIGN, FIRST>(src + 16 * g), b = ld_float8<ALIGN, FIRST>(src + 16 * g + 8);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                x[i] = a.v[i];
                x[8 + i] = b.v[i];
            }
        }
        uint32_t top = 0;                                      // largest magnitude's bits; NaNs come out largest
#pragma unroll
        for (int i = 0; i < kQuantPerLane; i++)
            top = max(top, __float_as_uint(x[i]) & 0x7FFFFFFFu);
#pragma unroll
        for (int o = 1; o < kLanes; o *= 2)
            top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        const bool tame = top - 0x21800000u <= 0x5D800000u - 0x21800000u;      // 2^-60 ... 2^60
        uint64_t codes = 0;
        uint8_t sbyte;
        float sdec;
        if (!ts.plain && __all_sync(0xffffffffu, tame || !inside)) {
            float sinv, amax = __uint_as_float(top);
            if (UE8M0) {
                sbyte = clpk_ue8m0_for_absmax(amax);
                sdec = 1.0f;
                sinv = __uint_as_float((254u - sbyte) << 23);  // a power of two's reciprocal is exact (2^-58 ... 2^62)
            } else {
                // rounding is monotone: the quotient of the largest is the largest quotient
                amax = shared_quotient(amax, ts.scale, ts.inv);
                sbyte = __nv_cvt_float_to_fp8(shared_quotient(amax, 6.0f, 0x1.555556p-3f), __NV_SATFINITE, __NV_E4M3);
                sdec = __half2float(__half(__nv_cvt_fp8_to_halfraw(sbyte, __NV_E4M3)));
                sinv = rcp_approx(sdec);
                sinv = __fmaf_rn(__fmaf_rn(-sdec, sinv, 1.0f), sinv, sinv);
            }
            // 16 products with a factor
            auto codes_times = [&](float factor) {
                uint32_t half[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    f32x2 q[4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        q[i] = mul2(pk(x[8 * h + 2 * i], x[8 * h + 2 * i + 1]), pk(factor));
                    half[h] = e2m1x8(q);
                }
                return (uint64_t)half[1] << 32 | half[0];
            };
            if (UE8M0) {
                codes = codes_times(sinv);
            } else {
                // Between a factor that is certainly too small and one that is certainly too large (the two quotients and the
                // factor itself are within 2^-21) nearly every element has one code, and rounding is monotone.
                const float factor = __fmul_rn(ts.inv, sinv);
                codes = codes_times(__fmul_rn(factor, 1.0f - 0x1p-20f));
                const bool sure = codes == codes_times(__fmul_rn(factor, 1.0f + 0x1p-20f));
                if (!__all_sync(0xffffffffu, sure)) {
                    codes = 0;
#pragma unroll
                    for (int i = 0; i < kQuantPerLane; i += 2) {
                        const f32x2 xx = pk(x[i], x[i + 1]);
                        f32x2 q = mul2(xx, pk(ts.inv));
                        q = fma2(fma2(pk(-ts.scale), q, xx), pk(ts.inv), q);
                        const f32x2 v = fma2(fma2(pk(-ts.scale), q, xx), pk(ts.inv), q);
                        q = mul2(v, pk(sinv));
                        q = fma2(fma2(pk(-sdec), q, v), pk(sinv), q);
                        // the sign is x's, also where a residual lost that of a zero
                        const float q0 = __uint_as_float(((uint32_t)q & 0x7FFFFFFFu) | (__float_as_uint(x[i]) & 0x80000000u));
                        const float q1 = __uint_as_float(((uint32_t)(q >> 32) & 0x7FFFFFFFu) | (__float_as_uint(x[i + 1]) & 0x80000000u));
                        codes |= (uint64_t)e2m1x2(q0, q1) << (4 * i);
                    }
                }
            }
            if (!UE8M0 && sdec == 0.0f)
                codes = 0;
        } else {
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < kQuantPerLane; i++) {
                if (!UE8M0)
                    x[i] = __fdiv_rn(x[i], ts.scale);
                amax = fmaxf(amax, fabsf(x[i]));
            }
#pragma unroll
            for (int o = 1; o < kLanes; o *= 2)
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            sbyte = fp4_block_scale<UE8M0>(amax, &sdec);
            if (sdec > 0.0f)
#pragma unroll
                for (int i = 0; i < kQuantPerLane; i++)
                    codes |= (uint64_t)clpk_e2m1_encode(__fdiv_rn(x[i], sdec)) << (4 * i);
        }
        if (inside) {
            if constexpr (ALIGN == 32)
                reinterpret_cast<uint64_t *>(packed)[g] = codes;
            else
                st_codes(packed + 8 * g, codes);
            if (lane % kLanes == 0)
                scales[g / kLanes] = sbyte;
        }
    }
}

__global__ void flush_kernel(uint4 *p, uint64_t n16, uint32_t tag)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride)
        p[i] = make_uint4(tag, tag, tag, tag);
}

// One step of one thread per item: CTAs start in address order as others end, which keeps the chip inside a few MiB of
// memory and has no last round of a few CTAs (a grid of 8 CTAs per SM, of which 6 are resident, ran the normal
// deviates at 57 % of the warps).
static unsigned fill_grid(uint64_t items)
{
    const uint64_t want = (items + kFillThreads - 1) / kFillThreads;
    return (unsigned)(want == 0 ? 1 : want < 0x7FFFFFFFull ? want : 0x7FFFFFFFull);
}

static bool aligned(const void *p, size_t bytes) { return ((uintptr_t)p % bytes) == 0; }

// One element at a time is bound by how fast CTAs start, whatever the type: 8192 x 8192 from an address 4 bytes off,
// uniform 270 us, normal 292, int8 269, absmax 129; cut at the boundary 64, 161, 56 and 42, as from an aligned one.
static Split split_at(const void *p, uint32_t align, uint32_t element_bits, uint32_t per, uint64_t n)
{
    const uint32_t head = (align - (uint32_t)((uintptr_t)p % align)) % align * 8 / element_bits;
    if (head >= n)
        return {0, (uint32_t)n, (uint32_t)n};
    const uint64_t whole = (n - head) / per;
    return {whole, head, (uint32_t)(n - per * whole)};
}

// Cut where the destination is aligned; the source's alignment there picks the loads.  A warp's narrow loads find the rest
// of their lines in L1, its narrow stores would be partial writes.  8192 x 8192 from a source 16 bytes off: to bf16
// 58 us, fp8 49, as from an aligned one; 4 bytes off 72 and 67 (one element at a time, bound by the start of CTAs, 272).
template <int DT>
static int launch_convert(void *d_dst, const float *d_src, uint64_t n, cudaStream_t s)
{
    constexpr uint32_t bits = Narrow<DT>::bits, per = Narrow<DT>::per, step_bytes = per * bits / 8;
    const Split part = split_at(d_dst, step_bytes < 32 ? step_bytes : 32, bits, per, n);
    void *dst = static_cast<uint8_t *>(d_dst) + (uint64_t)part.head * bits / 8;
    const float *src = d_src + part.head;
    const unsigned grid = fill_grid(part.whole);
    if (per == 8 && aligned(src, 32))
        return launch_behind(convert_kernel<DT, 32>, "launch convert", grid, kFillThreads, 0, s, dst, src, part, falling_order(4 * n));
    if (aligned(src, 16))
        return launch_behind(convert_kernel<DT, 16>, "launch convert", grid, kFillThreads, 0, s, dst, src, part, falling_order(4 * n));
    return launch_behind(convert_kernel<DT, 4>, "launch convert", grid, kFillThreads, 0, s, dst, src, part, falling_order(4 * n));
}

template <int BLOCK, bool UE8M0>
static int launch_quantize(uint8_t *d_packed, uint8_t *d_scales, const float *d_src, uint64_t n, float tensor_scale, cudaStream_t s)
{
    const TensorScale ts = {tensor_scale, 1.0f / tensor_scale, !UE8M0 && !(tensor_scale >= 0x1p-60f && tensor_scale <= 0x1p60f)};
    const uint64_t n16 = n / kQuantPerLane;
    const unsigned grid = fill_grid(n16);
    // an NVFP4 tensor's maximum has been taken in front, in falling order: its beginning was read last
    const bool falling = UE8M0 && falling_order(4 * n);
    if (aligned(d_src, 32) && aligned(d_packed, 8)) {
        if (falling_order(4 * n))
            return launch_behind(quantize_fp4_kernel<BLOCK, UE8M0, 32, true>, "launch quantize_fp4", grid, kFillThreads, 0, s, d_packed, d_scales, d_src, n16, ts, falling);
        return launch_behind(quantize_fp4_kernel<BLOCK, UE8M0, 32, false>, "launch quantize_fp4", grid, kFillThreads, 0, s, d_packed, d_scales, d_src, n16, ts, falling);
    }
    if (aligned(d_src, 16))
        return launch_behind(quantize_fp4_kernel<BLOCK, UE8M0, 16, false>, "launch quantize_fp4", grid, kFillThreads, 0, s, d_packed, d_scales, d_src, n16, ts, falling);
    return launch_behind(quantize_fp4_kernel<BLOCK, UE8M0, 4, false>, "launch quantize_fp4", grid, kFillThreads, 0, s, d_packed, d_scales, d_src, n16, ts, falling);
}

} // namespace clpk

using namespace clpk;

extern "C" {

int clpk_fill_f32(float *d_dst, uint64_t n, uint64_t seed, int dist, float mean, float std,
                  void *stream)
{
    CLPK_REQUIRE(d_dst || n == 0, "d_dst is NULL");
    CLPK_REQUIRE(dist >= 0 && dist <= 2, "unknown distribution %d", dist);
    if (n == 0)
        return CLPK_OK;
    const Split part = split_at(d_dst, 32, 32, 8, n);
    const uint64_t base = rand64_base(seed) + part.head;       // the generator's index is added to it
    d_dst += part.head;
    const uint32_t steps = part.whole >= kTwoStepsFrom ? 2 : 1;
    const unsigned grid = (unsigned)((part.whole + steps * kFillF32Threads - 1) / (steps * kFillF32Threads));
    cudaStream_t s = as_stream(stream);
    if (dist == CLPK_DIST_UNIFORM01)
        return launch_behind(fill_f32_kernel<CLPK_DIST_UNIFORM01>, "launch fill_f32", grid > 0 ? grid : 1, kFillF32Threads, 0, s, d_dst, part, base, steps, mean, std);
    if (dist == CLPK_DIST_UNIFORM_PM1)
        return launch_behind(fill_f32_kernel<CLPK_DIST_UNIFORM_PM1>, "launch fill_f32", grid > 0 ? grid : 1, kFillF32Threads, 0, s, d_dst, part, base, steps, mean, std);
    return launch_behind(fill_f32_kernel<CLPK_DIST_NORMAL>, "launch fill_f32", grid > 0 ? grid : 1, kFillF32Threads, 0, s, d_dst, part, base, steps, mean, std);
}

int clpk_fill_i8(int8_t *d_dst, uint64_t n, uint64_t seed, void *stream)
{
    CLPK_REQUIRE(d_dst || n == 0, "d_dst is NULL");
    if (n == 0)
        return CLPK_OK;
    const Split part = split_at(d_dst, 16, 8, 16, n);
    return launch_behind(fill_i8_kernel, "launch fill_i8", fill_grid(part.whole), kFillThreads, 0, as_stream(stream), d_dst + part.head,
                         part, rand64_base(seed) + part.head);
}

int clpk_convert_f32(void *d_dst, const float *d_src, uint64_t n, int dtype, void *stream)
{
    CLPK_REQUIRE((d_dst && d_src) || n == 0, "NULL buffer");
    CLPK_REQUIRE(dtype == CLPK_DT_F16 || dtype == CLPK_DT_BF16 || dtype == CLPK_DT_E4M3 ||
                     dtype == CLPK_DT_E5M2 || dtype == CLPK_DT_I8 || dtype == CLPK_DT_TF32 || dtype == CLPK_DT_E2M1 ||
                     dtype == CLPK_DT_F64,
                 "clpk_convert_f32: dtype %d has no plain conversion", dtype);
    if (n == 0)
        return CLPK_OK;
    CLPK_REQUIRE(dtype != CLPK_DT_E2M1 || n % 2 == 0, "E2M1 packs two elements per byte: n (%llu) must be even", (unsigned long long)n);
    cudaStream_t s = as_stream(stream);
    switch (dtype) {
    case CLPK_DT_F16:  return launch_convert<CLPK_DT_F16>(d_dst, d_src, n, s);
    case CLPK_DT_BF16: return launch_convert<CLPK_DT_BF16>(d_dst, d_src, n, s);
    case CLPK_DT_E4M3: return launch_convert<CLPK_DT_E4M3>(d_dst, d_src, n, s);
    case CLPK_DT_E5M2: return launch_convert<CLPK_DT_E5M2>(d_dst, d_src, n, s);
    case CLPK_DT_I8:   return launch_convert<CLPK_DT_I8>(d_dst, d_src, n, s);
    case CLPK_DT_TF32: return launch_convert<CLPK_DT_TF32>(d_dst, d_src, n, s);
    case CLPK_DT_F64:  return launch_convert<CLPK_DT_F64>(d_dst, d_src, n, s);
    default:           return launch_convert<CLPK_DT_E2M1>(d_dst, d_src, n, s);
    }
}

int clpk_absmax_f32(float *d_absmax, const float *d_src, uint64_t n, void *stream)
{
    CLPK_REQUIRE(d_absmax, "d_absmax is NULL");
    cudaStream_t s = as_stream(stream);
    const Split part = split_at(d_src, 32, 32, 8, n);
    // up to 32 Ki floats one CTA reads in the time that clearing the word would take
    if (n > 0 && n <= 32768 && d_src)
        return launch_behind(absmax_kernel<true, false>, "launch absmax", 1, kFillThreads, 0, s, d_absmax, d_src + part.head, part);
    CLPK_CUDA(cudaMemsetAsync(d_absmax, 0, sizeof(float), s));
    if (n == 0)
        return CLPK_OK;
    CLPK_REQUIRE(d_src, "d_src is NULL");
    const unsigned grid = fill_grid(part.whole / kAbsmaxLoads + 1);
    if (falling_order(4 * n))
        return launch_behind(absmax_kernel<false, true>, "launch absmax", grid, kFillThreads, 0, s, d_absmax, d_src + part.head, part);
    return launch_behind(absmax_kernel<false, false>, "launch absmax", grid, kFillThreads, 0, s, d_absmax, d_src + part.head, part);
}

int clpk_quantize_fp4(uint8_t *d_packed, uint8_t *d_scales, const float *d_src, uint64_t rows,
                      uint64_t cols, int dtype, float tensor_scale, void *stream)
{
    CLPK_REQUIRE(d_packed && d_scales && d_src, "NULL buffer");
    const bool mx = (dtype == CLPK_DT_MXF4 || dtype == CLPK_DT_MXF4_B64);
    CLPK_REQUIRE(mx || dtype == CLPK_DT_NVF4 || dtype == CLPK_DT_NVF4_B32, "dtype must be an MXF4 or NVF4 variant");
    CLPK_REQUIRE(cols % 64 == 0, "cols (%llu) must be a multiple of 64", (unsigned long long)cols);
    CLPK_REQUIRE(mx || tensor_scale > 0.0f, "tensor_scale must be positive");
    const uint64_t n = rows * cols;
    if (n == 0)
        return CLPK_OK;
    cudaStream_t s = as_stream(stream);
    switch (dtype) {
    case CLPK_DT_MXF4:     return launch_quantize<32, true>(d_packed, d_scales, d_src, n, 1.0f, s);
    case CLPK_DT_MXF4_B64: return launch_quantize<64, true>(d_packed, d_scales, d_src, n, 1.0f, s);
    case CLPK_DT_NVF4:     return launch_quantize<16, false>(d_packed, d_scales, d_src, n, tensor_scale, s);
    default:               return launch_quantize<32, false>(d_packed, d_scales, d_src, n, tensor_scale, s);
    }
}

int clpk_flush_l2(void *d_scratch, size_t bytes, void *stream)
{
    CLPK_REQUIRE(d_scratch, "d_scratch is NULL");
    static unsigned tag = 0;
    flush_kernel<<<num_sms() > 0 ? num_sms() * 8 : 1024, kFillThreads, 0, as_stream(stream)>>>(reinterpret_cast<uint4 *>(d_scratch),
                                                            bytes / 16, ++tag);
    CLPK_LAUNCH_CHECK("flush_l2");
    return CLPK_OK;
}

} // extern "C"
