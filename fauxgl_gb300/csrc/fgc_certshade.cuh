// fgc_certshade.cuh -- PhongShader.Fragment's colour bytes from FP32 interval
// arithmetic, for the plain (FP64) form.
//
// rasterize stores uint8(clamp(c) * 255) per channel (color.go:56-63), so a
// fragment's FP64 colour matters only through three truncations. cert_shade
// evaluates the shader (shader.go:75-96) in FP32 beside a bound on its
// distance from the FP64 result and returns the bytes when both ends of the
// interval truncate to the same ones; any other fragment is shaded in FP64.
// The stored bytes are the FP64 shader's in every case.
//
// The bounds (u = 2^-24, first-order terms, rounded up; the FP64 result's own
// rounding is 2^-29 of them and lies in the slack):
//   weights   w_k = b_k r_k, b_k >= 0 truncated to FP32 (2u), r_k > 0 rounded
//             (u), product (u): relative error 4u each. The shader divides by
//             their sum, which no direction depends on.
//   normal    n = sum w_k n_k, three FMAs on rounded components: a component
//             is off by at most 8u s S (s the weight sum, S the largest
//             |component|), the vector by sqrt(3) times that, its direction
//             by eN = 15u s S / |n|; normalising adds 8.5u (FP32 rsqrt: 2 ulp).
//   camera    d = s eye - sum w_k p_k: 9u s (E + P) a component (E, P the
//             largest |component| of eye and positions), direction
//             eC = 17u s (E + P) / |d| + 8.5u.
//   N.L       eD = |L| (eN + 5u).
//   specular  (camera . reflected) = 2 (N.L)(c.N) - c.L: off by
//             eS = |L| (4 eN + 3 eC + 24u) and second-order terms (5 %).
//   power     an integer p by repeated squaring, relative error (p - 1) u,
//             monotone in its base: the interval's ends go through it.
//   channel   colour * (ambient + diffuse N.L + specular s^p) * 255, all
//             factors >= 0: 8 roundings, widened by 12u and 1e-6.
//   vertex colours  sum w c / sum w from truncated FP64 weights, every term >=
//             0: 13u; the channel is widened by 28u instead of 12u. Their alpha
//             stays FP64.
// The bounds are relative, so they hold where nothing that matters nears the
// ends of FP32's range. A fragment is therefore left to FP64
//   - when n or d is not between 1e-15 and 1e18 long: n.n and d.d of a shorter
//     vector are subnormal and lose bits (normals need not be unit vectors);
//   - when the light reaches 1e14: a weight below FP32's normal range is off by
//     up to 1.4e-45, a vertex colour by 3.6e-22 (weights from 1e-15, colours to
//     1e6), which the light may multiply up to the 1e-6 that a channel is widened.
// A fragment with |N.L| <= eD is left to FP64 (the specular term switches on
// there); N.L < -eD is the ambient colour, formed once per draw in FP64.
//
// Host and device share the code: tests/certshade_check.cpp compares every
// certified byte with an FP64 evaluation on the CPU.
#pragma once

#include "fgc_intconv.cuh"

#include <cmath>

namespace fgc {

constexpr float kCertU = 5.9604644775390625e-8f;  // 2^-24
constexpr int kCertPowerMax = 128;                // largest SpecularPower certified

// A draw's shader parameters for cert_shade (filled on the host; `on` only
// when every precondition of the bounds holds).
struct CertParams {
    int32_t on;            // every fragment's colour is ObjectColor's
    int32_t vertex;        // the vertices' colours take its place (on is 0)
    int32_t power;         // SpecularPower, an integer in [2, kCertPowerMax]
    uint32_t unlit;        // NRGBA of a fragment facing away from the light
    float light[3], ln;    // LightDirection and an upper bound on its length
    float eye[3], emax;    // CameraPosition and its largest |component|
    float ambient[3], diffuse[3], specular[3];
    float color255[3];     // ObjectColor * 255
    float powtol;          // relative error bound of the power
};

FGC_HD float cs_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}
FGC_HD float cs_rsqrt(float x) {
#ifdef __CUDA_ARCH__
    return rsqrtf(x);
#else
    const float y = (float)(1.0 / std::sqrt((double)x));  // off by 2 ulp, as the device function may be
    uint32_t b;
    memcpy(&b, &x, 4);
    return y * (1.0f + ((b & 1) ? 2.0f : -2.0f) * 2.0f * kCertU);
#endif
}
FGC_HD float cs_max(float a, float b) { return fmaxf(a, b); }
FGC_HD float cs_dot(const float* a, const float* b) { return cs_fma(a[2], b[2], cs_fma(a[1], b[1], a[0] * b[0])); }
// Largest |component| of three vectors (a NaN is dropped: the weighted sum
// it also enters rejects the fragment).
FGC_HD float cs_max9(const float* a, const float* b, const float* c) {
    float m = 0.0f;
    for (int k = 0; k < 3; k++) m = cs_max(m, cs_max(fabsf(a[k]), cs_max(fabsf(b[k]), fabsf(c[k]))));
    return m;
}
FGC_HD float cs_pow(float x, int p) {
    if (p == 32) {
        x = x * x;
        x = x * x;
        x = x * x;
        x = x * x;
        return x * x;
    }
    float r = 1.0f;
    for (int i = p; i != 0; i >>= 1) {
        if (i & 1) r = r * x;
        x = x * x;
    }
    return r;
}
// uint8 of a channel bound already scaled by 255.
FGC_HD uint32_t cs_u8(float v) {
    if (!(v > 0.0f)) return 0u;
    return v >= 255.0f ? 255u : (uint32_t)v;
}

// b (a barycentric in [0, 2], +-0 included) truncated to FP32; anything else
// gives a value above 2, which cert_shade rejects.
FGC_HD float cert_bary(double b) { return f32_trunc_pos(fj_bits(b) & 0x7fffffffffffffffull); }

// The shader from weights w* (their sum s; each within 4u), positions p* and
// normals n* of the three vertices and the fragment's colour * 255 (within
// tol - 12u). A fragment facing away from the light has the bytes of C.unlit,
// or those of its own colour when it has one (vertex). alpha: the top byte.
FGC_HD bool cert_light(const CertParams& C, float w0, float w1, float w2, float s, const float* p0, const float* p1,
                       const float* p2, const float* n0, const float* n1, const float* n2, const float* col255,
                       float tol, bool vertex, uint32_t alpha, uint32_t* out) {
    float n[3], d[3];
    for (int k = 0; k < 3; k++) n[k] = cs_fma(w2, n2[k], cs_fma(w1, n1[k], w0 * n0[k]));
    const float rn = cs_rsqrt(cs_dot(n, n));
    const float eN = 15.0f * kCertU * s * cs_max9(n0, n1, n2) * rn + 8.5f * kCertU;
    if (!(eN < 0.01f && rn > 1e-18f && rn < 1e15f)) return false;
    for (int k = 0; k < 3; k++) n[k] = n[k] * rn;
    const float nl = cs_dot(n, C.light);
    const float eD = C.ln * (eN + 5.0f * kCertU) * 1.01f;
    float nlo = 0.0f, nhi = 0.0f, lo = 0.0f, hi = 0.0f;
    if (nl < -eD) {
        if (!vertex) {
            *out = C.unlit;
            return true;
        }
    } else {
        if (!(nl > eD)) return false;
        for (int k = 0; k < 3; k++) d[k] = cs_fma(C.eye[k], s, -cs_fma(w2, p2[k], cs_fma(w1, p1[k], w0 * p0[k])));
        const float rd = cs_rsqrt(cs_dot(d, d));
        const float eC = 17.0f * kCertU * s * (C.emax + cs_max9(p0, p1, p2)) * rd + 8.5f * kCertU;
        if (!(eC < 0.01f && rd > 1e-18f && rd < 1e15f)) return false;
        const float cl = cs_dot(d, C.light) * rd, cn = cs_dot(d, n) * rd;
        const float sp = cs_fma(2.0f * nl, cn, -cl);
        const float eS = C.ln * (4.0f * eN + 3.0f * eC + 24.0f * kCertU) * 1.05f;
        hi = cs_pow(cs_max(sp + eS, 0.0f), C.power) * (1.0f + C.powtol);
        lo = cs_pow(cs_max(sp - eS, 0.0f), C.power) * (1.0f - C.powtol);
        nlo = nl - eD;
        nhi = nl + eD;
    }
    uint32_t v = alpha;
    bool same = true;
    for (int k = 0; k < 3; k++) {
        const float a = cs_fma(C.specular[k], lo, cs_fma(C.diffuse[k], nlo, C.ambient[k])) * col255[k];
        const float most = cs_fma(C.specular[k], hi, cs_fma(C.diffuse[k], nhi, C.ambient[k]));
        const float b = most * col255[k];
        const uint32_t ia = cs_u8(a * (1.0f - tol) - 1e-6f);
        const uint32_t ib = cs_u8(b * (1.0f + tol) + 1e-6f);
        same = same && ia == ib && a <= b && most < 1e14f;  // a <= b is false for a NaN
        v |= ia << (8 * k);
    }
    if (!same) return false;
    *out = v;
    return true;
}

// b*: truncated barycentrics, r*: FP32 1/W of the three vertices, p*/n*: their
// FP32 positions and normals. Returns whether *out holds the fragment's bytes
// (alpha in C.unlit's top byte).
FGC_HD bool cert_shade(const CertParams& C, float b0, float b1, float b2, float r0, float r1, float r2,
                       const float* p0, const float* p1, const float* p2, const float* n0, const float* n1,
                       const float* n2, uint32_t* out) {
    if (!(b0 <= 2.0f && b1 <= 2.0f && b2 <= 2.0f && r0 > 1e-15f && r1 > 1e-15f && r2 > 1e-15f && r0 < 1e15f &&
          r1 < 1e15f && r2 < 1e15f))
        return false;
    const float w0 = b0 * r0, w1 = b1 * r1, w2 = b2 * r2;
    const float s = w0 + w1 + w2;
    if (!(s > 1e-18f)) return false;
    return cert_light(C, w0, w1, w2, s, p0, p1, p2, n0, n1, n2, C.color255, 12.0f * kCertU, false,
                      C.unlit & 0xff000000u, out);
}

// The same with the vertices' colours c* (r, g, b) in place of ObjectColor, from
// FP64 weights truncated to FP32 (2u each). The colour is sum w c / sum w, every
// term >= 0: weights, colours and roundings 13u in all. alpha: its byte, from
// FP64 (255 times a product of the weights' sum and its rounded reciprocal, which
// decides between 254 and 255), in the top byte.
FGC_HD bool cert_shade_vertex(const CertParams& C, float w0, float w1, float w2, const float* p0, const float* p1,
                              const float* p2, const float* n0, const float* n1, const float* n2, const float* c0,
                              const float* c1, const float* c2, uint32_t alpha, uint32_t* out) {
    const float s = w0 + w1 + w2;
    if (!(w0 >= 0.0f && w1 >= 0.0f && w2 >= 0.0f && s > 1e-15f && s < 1e15f)) return false;
    const float inv = 255.0f / s;
    float col[3];
    bool ok = true;
    for (int k = 0; k < 3; k++) {
        // 0 or far from FP32's ends, where a bound relative to the value holds
        ok = ok && (c0[k] == 0.0f || (c0[k] > 1e-12f && c0[k] < 1e6f)) &&
             (c1[k] == 0.0f || (c1[k] > 1e-12f && c1[k] < 1e6f)) && (c2[k] == 0.0f || (c2[k] > 1e-12f && c2[k] < 1e6f));
        col[k] = cs_fma(w2, c2[k], cs_fma(w1, c1[k], w0 * c0[k])) * inv;
    }
    if (!ok) return false;
    return cert_light(C, w0, w1, w2, s, p0, p1, p2, n0, n1, n2, col, 28.0f * kCertU, true, alpha, out);
}

}  // namespace fgc
