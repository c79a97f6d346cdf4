// fgc_fpjump.cuh -- the k-fold serial FP64 sum in O(binades) steps.
//
// rasterize (context.go:184-278) builds every edge value by repeated
// addition: w += a once per pixel along a row, w00 += b12 once per row. The
// result after k steps, t_k = RN(t_{k-1} + a), depends on every rounding on
// the way, so it is not s + k*a. It can still be computed without k steps:
// while t stays in one binade [2^E, 2^(E+1)) of width ulp u = 2^(E-52), t is
// a multiple of u and t + a = (m + q + f) u with integer m = t/u, q and
// fraction f of a/u fixed; round-to-nearest-even adds the same integer
// q + round(f) every step (a tie, |f| = 1/2, settles after one step on the
// even neighbour and then adds a constant too). So the sequence moves
// through a binade with one integer multiply-add, and real FP64 adds are
// only taken where it crosses into another binade (or near zero, or when
// |a| is not below the binade). repeat_add returns exactly the bits of the
// k-step loop, for every input including signed zeros, subnormals,
// infinities and NaN (the last three by plain steps).
//
// Host and device share this code: tests compare it with the plain loop.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FGC_HD __host__ __device__ __forceinline__
#else
#define FGC_HD inline
#endif

namespace fgc {

// The bit pattern of x. On the device it passes through an opaque move:
// given a plain bit cast, the compiler turns masks, sign flips and compares of
// the bits back into FP64 abs, negate and NaN tests (DADD / DSETP), which
// issue on the FP64 pipe at the FP64 rate -- the pipe these helpers keep free.
FGC_HD uint64_t fj_bits(double x) {
#ifdef __CUDA_ARCH__
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return (uint64_t)b;
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}

FGC_HD double fj_double(uint64_t b) {
#ifdef __CUDA_ARCH__
    double x;
    asm("mov.b64 %0, %1;" : "=d"(x) : "l"((unsigned long long)b));
    return x;
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}

FGC_HD double fj_add(double x, double y) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(x, y);
#else
    volatile double r = x + y;  // one IEEE binary64 round-to-nearest add
    return r;
#endif
}

// Whether x * y <= z, without overflow.
FGC_HD bool fj_mul_fits(uint64_t x, uint64_t y, uint64_t z) {
#ifdef __CUDA_ARCH__
    return __umul64hi(x, y) == 0 && x * y <= z;
#else
    return (unsigned __int128)x * y <= z;
#endif
}

// x / y where the quotient is below 2^20 (x < 2^54, 0 < y < 2^54). The FP32
// quotient is within one of it -- two rounded operands and a rounded division,
// 3 * 2^-24 relative -- and two exact products settle it; a 64-bit division is
// a subroutine of some 100 instructions in the middle of every jump's chain
// (the close-up frame of 1.55 M pixels: row starts 320 -> 260 us).
FGC_HD uint64_t fj_div_small(uint64_t x, uint64_t y) {
    uint64_t c = (uint64_t)((float)x / (float)y);
    if (c * y > x) c--;
    if ((c + 1) * y <= x) c++;
    return c;
}

// t = s; repeat k times: t = RN(t + a). Returns t.
FGC_HD double repeat_add(double s, double a, uint64_t k) {
    const uint64_t kSign = 0x8000000000000000ull;
    const uint64_t kExp = 0x7ff0000000000000ull;
    const uint64_t kFrac = 0x000fffffffffffffull;
    const uint64_t kHidden = 0x0010000000000000ull;  // 2^52
    const uint64_t kTop = 0x0020000000000000ull;     // 2^53
    const uint64_t ab = fj_bits(a);
    if ((ab & kExp) == kExp || (ab << 1) == 0) {
        // a infinite, NaN or zero: one step reaches a fixed point
        return k ? fj_add(s, a) : s;
    }
    const int ea = (int)((ab >> 52) & 0x7ff);
    const int el = ea ? ea : 1;  // exponent of a's last place
    const uint64_t Ma = (ab & kFrac) | (ea ? kHidden : 0);
    while (k > 0) {
        s = fj_add(s, a);  // a real step: enters the binade the model then covers
        k--;
        if (k == 0) break;
        const uint64_t sb = fj_bits(s);
        const int es = (int)((sb >> 52) & 0x7ff);
        const int sh = es - el;             // a/u = Ma / 2^sh
        // infinite or NaN: fixed from here; |a| < u/2: t + a rounds back to t
        if (es == 0x7ff || (sh >= 54 && ea < es && (((sb ^ ab) & kSign) == 0 || (sb & kFrac) > 1))) return s;
        // zero, subnormal, or |a| not below the binade: plain steps
        if (es == 0 || ea >= es || sh <= 0 || sh >= 54) continue;
        // work on |t|: it grows when t and a have the same sign
        const bool grow = ((sb ^ ab) & kSign) == 0;
        const uint64_t m = (sb & kFrac) | kHidden;  // |t| / u, in [2^52, 2^53)
        // |t| changes by d = RN(a/u) (in units of u) per step
        const uint64_t half = 1ull << (sh - 1);
        const uint64_t r = Ma + half;
        uint64_t d = r >> sh;
        const uint64_t q = Ma >> sh;
        if ((r & (half + half - 1)) == 0) {
            // tie: the even neighbour. m + q and m - q have the parity of
            // m + q; once m is even (after one tie step) d is constant.
            if ((m & 1) != 0) continue;
            d &= ~1ull;
        }
        // steps that keep every exact sum (before rounding) inside the
        // binade, with one unit of margin at both ends (shrinking from the
        // binade's first value leaves it: finer spacing below): n steps fit
        // when (n - 1) * d <= avail
        const int64_t avail = (int64_t)(grow ? (kTop - 2) - m : m - (kHidden + 1)) - (int64_t)q;
        if (!grow && m <= kHidden + 1) continue;
        if (d == 0) return s;               // t + a rounds back to t from here on
        if (avail < 0) continue;
        // all k remaining steps usually fit: only a jump that reaches the
        // binade's end needs the division
        const uint64_t n = fj_mul_fits(k - 1, d, (uint64_t)avail)
                               ? k : (k <= (1u << 20) ? fj_div_small((uint64_t)avail, d) : (uint64_t)avail / d) + 1;
        const uint64_t nd = n * d;
        k -= n;
        s = fj_double((sb & (kSign | kExp)) | ((grow ? m + nd : m - nd) & kFrac));
    }
    return s;
}

}  // namespace fgc
