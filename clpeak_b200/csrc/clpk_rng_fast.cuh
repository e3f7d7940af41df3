// The generators of clpk_rng.h for whole arrays on the device: the same values bit for bit, in fewer instructions.
//
//  * Two elements at a time in sm_100's packed fp32 pairs (fma / mul / add.rn.f32x2, two IEEE operations per issued
//    instruction): every rounding of clpk_rng.h is kept, in its order.
//  * Quotient and square root are correctly rounded by a residual correction of a hardware approximation (P. Markstein,
//    "Computation of elementary functions on the IBM RISC System/6000", 1990): y ~ 1/b refined once, q = a y,
//    q + (a - q b) y; and s = x y with y ~ 1/sqrt(x), s + (x - s s) y / 2.  Both were compared with the IEEE
//    operations over everything they can meet here: the radius has 2^23 arguments, the angle 2^24.
//  * Integers become floats by adding them to the bits of 2^23 (exact below 2^23; the hardware conversion runs at a
//    quarter of the fp32 rate), and the quadrant is two bits of the random word.
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

// clpk_rand64 with the seed's own mixing done once
__device__ __forceinline__ uint64_t rand64_at(uint64_t mixed_seed, uint64_t idx) { return clpk_mix64(mixed_seed + idx); }

// The steps below run over P pairs side by side, so that a constant is brought into a register pair once for all of
// them (with one pair at a time a third of the instructions were that).
#define CLPK_PAIRS _Pragma("unroll") for (int j = 0; j < P; j++)

// -sqrt(-2 ln u1), u1 = n 2^-23 with n = 1 ... 2^23, for 2 P values of n
template <int P>
__device__ __forceinline__ void minus_radius(const uint32_t (&n)[2 * P], f32x2 (&out)[P])
{
    // n as a float is m 2^e; u1 has the same significand.  The significand is taken from (sqrt(1/2), sqrt(2)]: one
    // above 1.41421354 (0x3FB504F3) is halved, which is adding 0x3F800000 - 0x3F3504F4 to the bits and reading the
    // exponent there.
    f32x2 t[P], p[P], s[P], e[P];
    CLPK_PAIRS
    {
        const f32x2 nf = add2(pk(__uint_as_float(0x4B000000u + n[2 * j]), __uint_as_float(0x4B000000u + n[2 * j + 1])), pk(-8388608.0f));
        const uint32_t b0 = (uint32_t)nf + (0x3F800000u - 0x3F3504F4u), b1 = (uint32_t)(nf >> 32) + (0x3F800000u - 0x3F3504F4u);
        t[j] = pk(__uint_as_float((b0 & 0x007FFFFFu) + 0x3F3504F4u), __uint_as_float((b1 & 0x007FFFFFu) + 0x3F3504F4u));
        e[j] = add2(pk(__uint_as_float(0x4B000000u + (b0 >> 23)), __uint_as_float(0x4B000000u + (b1 >> 23))), pk(-(8388608.0f + 127.0f + 23.0f)));
    }
    CLPK_PAIRS
    {
        const f32x2 m = t[j], a = add2(m, pk(-1.0f)), b = add2(m, pk(1.0f)), minus_b = fma2(m, pk(-1.0f), pk(-1.0f));
        f32x2 y = pk(rcp_approx(lo_of(b)), rcp_approx(hi_of(b)));
        y = fma2(y, fma2(minus_b, y, pk(1.0f)), y);
        const f32x2 q = mul2(a, y);
        t[j] = fma2(fma2(minus_b, q, a), y, q);               // (m - 1) / (m + 1)
        s[j] = mul2(t[j], t[j]);
    }
    CLPK_PAIRS p[j] = fma2(pk(0.0909090936f), s[j], pk(0.111111112f));
    CLPK_PAIRS p[j] = fma2(p[j], s[j], pk(0.142857149f));
    CLPK_PAIRS p[j] = fma2(p[j], s[j], pk(0.2f));
    CLPK_PAIRS p[j] = fma2(p[j], s[j], pk(0.333333343f));
    CLPK_PAIRS p[j] = fma2(p[j], s[j], pk(1.0f));
    CLPK_PAIRS
    {
        const f32x2 ln = fma2(e[j], pk(0.693147182f), mul2(add2(t[j], t[j]), p[j]));
        const f32x2 x = add2(ln, ln);                         // minus the radicand
        // ln 1 = 0 (n = 2^23) must not meet an infinite reciprocal; the next radicand is 2.4e-7
        const f32x2 z = pk(rsqrt_approx(fmaxf(-lo_of(x), 1e-30f)), rsqrt_approx(fmaxf(-hi_of(x), 1e-30f)));
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
        // the fraction of the quadrant, 22 bits, as a significand
        const f32x2 f = add2(pk(__uint_as_float(0x3F800000u | ((k[2 * j] & 0x3FFFFFu) << 1)), __uint_as_float(0x3F800000u | ((k[2 * j + 1] & 0x3FFFFFu) << 1))),
                             pk(-1.0f));
        th[j] = mul2(f, pk(1.57079637f));
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
        // quadrant (bits 23, 22) 0: cos, 1: -sin, 2: -cos, 3: sin; here with the other sign
        const uint32_t w = kk << 8;
        return __uint_as_float(__float_as_uint((w & 0x40000000u) ? sin_v : cos_v) ^ (~(w ^ (w << 1)) & 0x80000000u));
    };
    CLPK_PAIRS
    {
        const f32x2 sn = mul2(n[j], th[j]);
        out[j] = pk(pick(k[2 * j], lo_of(c[j]), lo_of(sn)), pick(k[2 * j + 1], hi_of(c[j]), hi_of(sn)));
    }
}

// clpk_normal01 of 2 P random words
template <int P>
__device__ __forceinline__ void normal01(const uint64_t (&h)[2 * P], f32x2 (&out)[P])
{
    uint32_t n[2 * P], k[2 * P];
#pragma unroll
    for (int i = 0; i < 2 * P; i++) {
        n[i] = (uint32_t)(h[i] >> 41) + 1u;
        k[i] = (uint32_t)h[i];
    }
    f32x2 r[P], c[P];
    minus_radius<P>(n, r);
    minus_cos2pi<P>(k, c);
    CLPK_PAIRS out[j] = mul2(r[j], c[j]);
}
#undef CLPK_PAIRS

} // namespace clpk
