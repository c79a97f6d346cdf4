// fgc_softdiv.cuh -- correctly rounded FP64 reciprocals and quotients on the
// integer pipe.
//
// An FP64 instruction holds its SM quarter's FP64 pipe for 64 cycles a warp, an
// integer one for 2, and the kernels that divide (vertex stage, primitive
// setup) are bound by that pipe: a correctly rounded reciprocal there is a
// chain of some eight FP64 instructions, here some forty integer ones.
//
// Method: Newton's iteration for 1/d in fixed point, from an FP32 seed, then
// rounding by the exact remainder. With d = x 2^63 in [2^63, 2^64) (x the
// significand in [1, 2)):
//   seed     Y0 = 2^31 / x to within 2^-20 of it (FP32 reciprocal of x truncated
//            to 24 bits: 2^-23 and 2 ulp)
//   step 1   with the upper 32 bits of d: |x Y1 2^-31 - 1| <= 2^-29 (the square
//            of the seed's error, one unit of Y1 <= 2^-30, 2^-31 for d's lower
//            half)
//   step 2   with all of d: Y2 = 2^62 / x to within 2^-57 (2^-58 and the cut of
//            the residual's last three bits, 2^-59)
//   round    q = Y2 rounded to the result's 53 bits is off by at most 0.55 units
//            in the last place, so the exact remainder (below one divisor, known
//            from its low 64 bits) moves it by at most one. Neither a reciprocal
//            nor a quotient of two doubles lies halfway between two others, but
//            for results below the normal range.
// Operands or results outside the normal range take CUDA's functions.
// tests/test_softdiv.py compares every form with the CPU's division.
#pragma once

#include <cmath>

#include "fgc_fpjump.cuh"

namespace fgc {

FGC_HD uint64_t sd_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// The seed for a significand whose 23 fraction bits are f: 1 / x in FP32.
FGC_HD float sd_seed(uint32_t f) {
#ifdef __CUDA_ARCH__
    return __fdividef(1.0f, __uint_as_float(0x3f800000u | f));
#else
    uint32_t b = 0x3f800000u | f;
    float x;
    memcpy(&x, &b, 4);
    return 1.0f / x;
#endif
}

// 2^62 / x to within 2^-57, m = x 2^52 in [2^52, 2^53), from a seed in
// [0.5 - 2^-21, 1 + 2^-21].
FGC_HD uint64_t sd_recip(uint64_t m, float seed) {
    uint32_t sb;
#ifdef __CUDA_ARCH__
    sb = __float_as_uint(seed);
#else
    memcpy(&sb, &seed, 4);
#endif
    const uint64_t d = m << 11;
    const uint32_t dh = (uint32_t)(d >> 32), dl = (uint32_t)d;
    const uint32_t y0 = ((sb & 0x7fffffu) | 0x800000u) << ((sb >> 23) - 119u);  // seed 2^31: exponents 125 .. 127
    const int64_t e1 = (int64_t)((1ull << 62) - (uint64_t)dh * y0);
    const int64_t c1 = ((int64_t)y0 * (int32_t)(e1 >> 12)) >> 50;
    const uint32_t y1 = y0 + (uint32_t)(int32_t)c1;
    const uint64_t p = (uint64_t)dh * y1 + (((uint64_t)dl * y1) >> 32);
    const int64_t e2 = (int64_t)((1ull << 62) - p);
    return ((uint64_t)y1 << 31) + (uint64_t)(((int64_t)y1 * (int32_t)(e2 >> 3)) >> 28);
}

// A divisor: its reciprocal's 62 bits, where it is a normal number.
struct SoftRcp {
    uint64_t m, y;  // significand in [2^52, 2^53), 2^62 / x
    uint64_t sign;
    int e;          // biased exponent
    bool normal;
};

FGC_HD SoftRcp soft_rcp(double w) {
    SoftRcp r;
    const uint64_t b = fj_bits(w);
    r.sign = b & 0x8000000000000000ull;
    r.e = (int)((b >> 52) & 0x7ff);
    r.normal = (unsigned)(r.e - 1) < 2046u;
    r.m = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    r.y = sd_recip(r.m, sd_seed((uint32_t)(b >> 29) & 0x7fffffu));
    return r;
}

// q moved to the nearest of the exact quotient n / m, rem = n - q m.
FGC_HD uint64_t sd_round(uint64_t q, uint64_t m, int64_t rem) {
    const int64_t t = 2 * rem;
    if (t > (int64_t)m) q++;
    if (t < -(int64_t)m) q--;
    return q;
}

// 1 / w
FGC_HD double rcp_of(double w, const SoftRcp& r) {
    if (!r.normal || r.e > 2044) {
#ifdef __CUDA_ARCH__
        return __drcp_rn(w);
#else
        return 1.0 / w;
#endif
    }
    const uint64_t q = (r.y + 256) >> 9;  // 2^105 / m
    return fj_double(r.sign + ((uint64_t)(2044 - r.e) << 52) + sd_round(q, r.m, (int64_t)(0 - q * r.m)));
}
FGC_HD double rcp_i(double w) { return rcp_of(w, soft_rcp(w)); }

// x / w
FGC_HD double div_of(double x, double w, const SoftRcp& r) {
    const uint64_t b = fj_bits(x);
    const int ex = (int)((b >> 52) & 0x7ff);
    const uint64_t mx = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const bool ge = mx >= r.m;                      // the quotient's significand is 1 or more
    const int e = ex - r.e + (ge ? 1023 : 1022);
    if (!r.normal || (unsigned)(ex - 1) >= 2046u || (unsigned)(e - 1) >= 2045u) {
        if ((b << 1) == 0 && r.normal) return fj_double((b ^ r.sign) & 0x8000000000000000ull);  // a zero
#ifdef __CUDA_ARCH__
        return __ddiv_rn(x, w);
#else
        return x / w;
#endif
    }
    const uint64_t p = sd_mulhi(mx << 11, r.y);     // the quotient 2^61
    const int s = ge ? 9 : 8;
    const uint64_t q = (p + (1ull << (s - 1))) >> s;
    const int64_t rem = (int64_t)((mx << (ge ? 52 : 53)) - q * r.m);
    return fj_double(((b ^ r.sign) & 0x8000000000000000ull) + ((uint64_t)(e - 1) << 52) + sd_round(q, r.m, rem));
}

// ---- square root: Newton's iteration for 1 / sqrt(f) from an FP32 seed, one
// step of Heron's on sqrt(f), rounding by the exact remainder. f in [1, 4) is
// the significand with the exponent's parity, A = f 2^62.

// 1 / sqrt(f) in FP32 for the 24 bits after f's leading one (odd: f >= 2).
FGC_HD float sd_rseed(uint32_t f, bool odd) {
    const uint32_t b = (odd ? 0x40000000u : 0x3f800000u) | f;
#ifdef __CUDA_ARCH__
    return rsqrtf(__uint_as_float(b));
#else
    float x;
    memcpy(&x, &b, 4);
    return 1.0f / std::sqrt(x);
#endif
}

// sqrt(f) 2^61 to within 2^-55, from a seed in (0.5 - 2^-21, 1 + 2^-21].
FGC_HD uint64_t sd_sqrt(uint64_t A, float seed) {
    uint32_t sb;
#ifdef __CUDA_ARCH__
    sb = __float_as_uint(seed);
#else
    memcpy(&sb, &seed, 4);
#endif
    uint32_t y = ((sb & 0x7fffffu) | 0x800000u) << ((sb >> 23) - 119u);  // 2^31 / sqrt(f)
    const uint32_t ah = (uint32_t)(A >> 32), al = (uint32_t)A;
    // 1 - f y^2, in units of 2^-61; y + y of half that
    const uint32_t yy = (uint32_t)(((uint64_t)y * y) >> 31);
    const int64_t e = (int64_t)((1ull << 61) - (uint64_t)ah * yy);
    y += (uint32_t)(int32_t)(((int64_t)y * (int32_t)(e >> 12)) >> 50);
    // s = f y, in units of 2^-61, and s + (f - s^2) y / 2
    const uint64_t s = (uint64_t)ah * y + (((uint64_t)al * y) >> 32);
    const int64_t r = (int64_t)((A >> 4) - sd_mulhi(s, s));  // 2^-58
    return s + (uint64_t)(((int64_t)(int32_t)(r >> 3) * (int64_t)y) >> 26);
}

// RN(sqrt(x)); subnormal, infinite, NaN and negative arguments and zeros take
// CUDA's function.
FGC_HD double sqrt_seeded(double x, float seed) {
    const uint64_t b = fj_bits(x);
    const uint32_t e = (uint32_t)(b >> 52);
    const bool odd = (e & 1) == 0;  // the unbiased exponent's parity
    const uint64_t m = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const uint64_t s = sd_sqrt(m << (odd ? 11 : 10), seed);
    uint64_t q = (s + 256) >> 9;
    const int64_t rem = (int64_t)((m << (odd ? 53 : 52)) - q * q);  // f 2^104 - q^2
    if (rem > (int64_t)q) q++;
    if (rem <= -(int64_t)q) q--;
    return fj_double(((uint64_t)((e + 1021u) >> 1) << 52) + q);
}
FGC_HD double sqrt_i(double x) {
    const uint64_t b = fj_bits(x);
    const uint32_t e = (uint32_t)(b >> 52);
    if (e - 1u >= 2046u) {
#ifdef __CUDA_ARCH__
        return __dsqrt_rn(x);
#else
        return std::sqrt(x);
#endif
    }
    return sqrt_seeded(x, sd_rseed((uint32_t)(b >> 29) & 0x7fffffu, (e & 1) == 0));
}

}  // namespace fgc
