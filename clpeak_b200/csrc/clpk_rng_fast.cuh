// The generators of clpk_rng.h for whole arrays on the device: the same values bit for bit, in fewer instructions.
//
//  * Two elements at a time in sm_100's packed fp32 pairs (fma / mul / add.rn.f32x2, two IEEE operations per issued
//    instruction): every rounding of clpk_rng.h is kept, in its order.  Factors that are powers of two round to nothing and
//    are moved to where they cost nothing: into a polynomial's coefficients, or into the constants of a fused step.
//  * Quotient and square root are correctly rounded by a residual correction of a hardware approximation (P. Markstein,
//    "Computation of elementary functions on the IBM RISC System/6000", 1990): q = a y with y ~ 1/b, q + (a - q b) y; and
//    s = x y with y ~ 1/sqrt(x), s + (x - s s) y / 2.  Both were compared with the IEEE operations over everything they can
//    meet here: the radius has 2^23 arguments, the angle 2^24.  (y needs no refinement of its own for that.)
//  * Integers become floats by adding them to the bits of 2^23 (exact below 2^23; the hardware conversion runs at a
//    quarter of the fp32 rate), and the quadrant is two bits of the random word.
//  * Consecutive elements share what stands above bit 30 of the generator's first step (random_words).
//
// What bounds the normal deviates: a packed instruction takes two issue slots' worth of register reads (56 issued
// instructions a deviate, 17 of them packed: 73 of the 75 cycles a deviate takes a scheduler), so that what counts is the
// number of operations, 40 of fp32 and 30 others.  8192 x 8192 158 -> 138 us against the form with a refined reciprocal,
// 44 fp32 operations and the whole first step for every element.  Tried: everything scalar 155 (with the logarithm's
// polynomial alone scalar 2 us faster than all packed, as here); one polynomial for sine and cosine with coefficients
// from shared memory 141; constants held in registers 176, since three operands of a pair do not come out of the register
// banks in two cycles.
#pragma once

#include "clpk_rng.h"

namespace clpk {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 pk(float v) { return pk(v, v); }
__device__ __forceinline__ float lo_of(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// clpk_rand64 of a seed is a function of this plus the index
__host__ __device__ inline uint64_t rand64_base(uint64_t seed) { return clpk_mix64(seed) + 0x9E3779B97F4A7C15ull; }

// The words of N consecutive elements, z their first one's index + rand64_base: clpk_mix64's steps, with the high half as it is
// before the last of them, which changes its lowest bit only (no generator takes that).
//
// z ^ (z >> 30) of z, z + 1, ...: while nothing is carried into bit 30, z >> 30 is the same for all of them and with it the
// high word, whose part of the product is computed once.  That leaves an addition, an exclusive or and two multiply-adds
// of nine instructions; one in 2^27 threads meets a carry and goes the long way.  8192 x 8192 normal deviates 146 -> 138 us.
template <int N>
__device__ __forceinline__ void random_words(uint64_t z, uint32_t (&hi)[N], uint32_t (&lo)[N])
{
    constexpr uint64_t c1 = 0xBF58476D1CE4E5B9ull, c2 = 0x94D049BB133111EBull;
    uint64_t p[N];
    const uint32_t z_lo = (uint32_t)z, z_hi = (uint32_t)(z >> 32);
    if ((z_lo & 0x3FFFFFFFu) <= 0x3FFFFFFFu - (N - 1)) {
        const uint32_t low = (uint32_t)(z >> 30), from_high = (z_hi ^ (z_hi >> 30)) * (uint32_t)c1;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t w = (z_lo + i) ^ low;
            p[i] = (uint64_t)w * (uint32_t)c1 + ((uint64_t)from_high << 32) + ((uint64_t)(w * (uint32_t)(c1 >> 32)) << 32);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i++)
            p[i] = ((z + i) ^ ((z + i) >> 30)) * c1;
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint64_t q = (p[i] ^ (p[i] >> 27)) * c2;
        hi[i] = (uint32_t)(q >> 32);
        lo[i] = (uint32_t)(q ^ (q >> 31));
    }
}

// The steps below run over P pairs side by side, so that a constant is brought into a register pair once for all of
// them (with one pair at a time a third of the instructions were that).
#define CLPK_PAIRS _Pragma("unroll") for (int j = 0; j < P; j++)

// a * b + c for a constant c, as two instructions that carry c with them
__device__ __forceinline__ f32x2 fma_each(f32x2 a, f32x2 b, float c)
{
    return pk(__fmaf_rn(lo_of(a), lo_of(b), c), __fmaf_rn(hi_of(a), hi_of(b), c));
}

// -sqrt(-2 ln u1), u1 = n 2^-23 with n = 1 ... 2^23, for the 2 P values of n = n1 + 1
template <int P>
__device__ __forceinline__ void minus_radius(const uint32_t (&n1)[2 * P], f32x2 (&out)[P])
{
    // n as a float is m 2^e; u1 has the same significand.  The significand is taken from (sqrt(1/2), sqrt(2)]: one
    // above 1.41421354 (0x3FB504F3) is halved, which is adding 0x3F800000 - 0x3F3504F4 to the bits and reading the
    // exponent there.  The complement of that exponent is the power of two that makes 2 m of n.
    f32x2 t[P], p[P], s[P], e[P];
    CLPK_PAIRS
    {
        const f32x2 n = add2(pk(__uint_as_float(0x4B000000u + n1[2 * j]), __uint_as_float(0x4B000000u + n1[2 * j + 1])), pk(-8388607.0f));
        const uint32_t b0 = (uint32_t)n + (0x3F800000u - 0x3F3504F4u), b1 = (uint32_t)(n >> 32) + (0x3F800000u - 0x3F3504F4u);
        const f32x2 scale = pk(__uint_as_float(~b0 & 0x7F800000u), __uint_as_float(~b1 & 0x7F800000u));
        e[j] = add2(pk(__uint_as_float(0x4B000000u + (b0 >> 23)), __uint_as_float(0x4B000000u + (b1 >> 23))), pk(-(8388608.0f + 127.0f + 23.0f)));
        const f32x2 a = fma2(n, scale, pk(-2.0f)), b = fma2(n, scale, pk(2.0f));
        const f32x2 y = pk(rcp_approx(-lo_of(b)), rcp_approx(-hi_of(b)));
        const f32x2 q = mul2(a, y);
        t[j] = fma2(fma2(b, q, a), y, q);                     // -(m - 1) / (m + 1)
        s[j] = mul2(t[j], t[j]);
    }
    // minus four times the series, so that its product with t is 2 ln m, and x minus the radicand
    CLPK_PAIRS p[j] = fma_each(s[j], pk(-4.0f * 0.0909090936f), -4.0f * 0.111111112f);
    CLPK_PAIRS p[j] = fma_each(p[j], s[j], -4.0f * 0.142857149f);
    CLPK_PAIRS p[j] = fma_each(p[j], s[j], -4.0f * 0.2f);
    CLPK_PAIRS p[j] = fma_each(p[j], s[j], -4.0f * 0.333333343f);
    CLPK_PAIRS p[j] = fma_each(p[j], s[j], -4.0f);
    CLPK_PAIRS
    {
        const f32x2 x = fma2(e[j], pk(2.0f * 0.693147182f), mul2(t[j], p[j]));
        // ln 1 = 0 (n = 2^23) must not meet an infinite reciprocal; the next radicand, 2.4e-7, does not notice
        const f32x2 above = add2(x, pk(-1e-30f));
        const f32x2 z = pk(rsqrt_approx(-lo_of(above)), rsqrt_approx(-hi_of(above)));
        const f32x2 r = mul2(x, z);
        out[j] = fma2(fma2(r, r, x), mul2(pk(0.5f), z), r);
    }
}

// -cos(2 pi k 2^-24) for 2 P values of k, the low 24 bits of k[]: clpk_det_cos2pi's fold and both of its polynomials
template <int P>
__device__ __forceinline__ void minus_cos2pi(const uint32_t (&k)[2 * P], f32x2 (&out)[P])
{
    f32x2 th[P], s[P], c[P], n[P];
    CLPK_PAIRS
    {
        // the fraction of the quadrant, 22 bits, as a significand: 1 + half of it
        const f32x2 f = pk(__uint_as_float(0x3F800000u | (k[2 * j] & 0x3FFFFFu)), __uint_as_float(0x3F800000u | (k[2 * j + 1] & 0x3FFFFFu)));
        th[j] = fma2(f, pk(2.0f * 1.57079637f), pk(-2.0f * 1.57079637f));
        s[j] = mul2(th[j], th[j]);
    }
    CLPK_PAIRS c[j] = fma2(pk(-1.14707454e-11f), s[j], pk(2.08767570e-09f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(-2.75573192e-07f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(2.48015876e-05f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(-1.38888892e-03f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(4.16666679e-02f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(-0.5f));
    CLPK_PAIRS c[j] = fma2(c[j], s[j], pk(1.0f));
    CLPK_PAIRS n[j] = fma2(pk(-7.64716373e-13f), s[j], pk(1.60590438e-10f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(-2.50521084e-08f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(2.75573188e-06f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(-1.98412701e-04f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(8.33333377e-03f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(-0.166666672f));
    CLPK_PAIRS n[j] = fma2(n[j], s[j], pk(1.0f));
    auto pick = [](uint32_t kk, float cos_v, float sin_v) {
        // quadrant (bits 23, 22) 0: cos, 1: -sin, 2: -cos, 3: sin; here with the other sign, which the upper bit of the
        // quadrant's successor says
        const uint32_t next = kk * 256u + 0x40000000u;
        return __uint_as_float(__float_as_uint((kk & 0x400000u) ? sin_v : cos_v) ^ (~next & 0x80000000u));
    };
    CLPK_PAIRS
    {
        const f32x2 sn = mul2(n[j], th[j]);
        out[j] = pk(pick(k[2 * j], lo_of(c[j]), lo_of(sn)), pick(k[2 * j + 1], hi_of(c[j]), hi_of(sn)));
    }
}

// clpk_normal01 of 2 P random words
template <int P>
__device__ __forceinline__ void normal01(const uint32_t (&hi)[2 * P], const uint32_t (&lo)[2 * P], f32x2 (&out)[P])
{
    uint32_t n1[2 * P];
#pragma unroll
    for (int i = 0; i < 2 * P; i++)
        n1[i] = hi[i] >> 9;
    f32x2 r[P], c[P];
    minus_radius<P>(n1, r);
    minus_cos2pi<P>(lo, c);
    CLPK_PAIRS out[j] = mul2(r[j], c[j]);
}
#undef CLPK_PAIRS

} // namespace clpk
