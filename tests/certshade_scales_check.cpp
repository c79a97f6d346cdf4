// Checks cert_shade and cert_shade_vertex (fauxgl_gb300/csrc/fgc_certshade.cuh)
// against an FP64 evaluation of PhongShader.Fragment in the reference's
// operation order (shader.go:75-96, color.go:56-63) where the magnitudes reach
// the ends of FP32's range: the lengths of normals, the size of the scene, W,
// the light's length and the colour factors are drawn over the whole exponent
// range, together or for each vertex, one after the other and combined. Every
// certified NRGBA word must be the FP64 one.
// Prints "ok <certified share>" or the first mismatch of each form and the
// number of mismatches.
// usage: certshade_scales_check N   build: g++ -O2 -ffp-contract=off -std=c++17
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../fauxgl_gb300/csrc/fgc_certshade.cuh"

static uint64_t g_state = 0x2545f4914f6cdd1dull;
static uint64_t next64() {
    uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double uni() { return (double)(next64() >> 11) / 9007199254740992.0; }
static double sym() { return 2 * uni() - 1; }
static double mag(double lo, double hi) { return std::pow(10.0, lo + (hi - lo) * uni()); }

static uint32_t u8(double c) {
    if (!(c == c)) return 0;
    c = c < 0 ? 0 : c > 1 ? 1 : c;
    return (uint32_t)(c * 255.0);
}
static double min1(double v) { return v < 1 || v != v ? v : 1; }

// Go's math.Pow for an integer power: repeated squaring of the Frexp mantissa.
static double go_pow(double x, int p) {
    if (x == 0 || x == 1 || std::isinf(x)) return x;
    int xe;
    double x1 = std::frexp(x, &xe), a1 = 1;
    long long ae = 0, e = xe;
    for (int i = p; i != 0; i >>= 1) {
        if (e < -4096 || e > 4096) {
            ae += e;
            break;
        }
        if (i & 1) {
            a1 *= x1;
            ae += e;
        }
        x1 *= x1;
        e <<= 1;
        if (x1 < .5) {
            x1 += x1;
            e--;
        }
    }
    return std::ldexp(a1, (int)(ae < -100000 ? -100000 : ae > 100000 ? 100000 : ae));
}

enum { kNormals = 1, kScene = 2, kW = 4, kLight = 8, kFactors = 16, kWeights = 32, kForms = 64 };

int main(int argc, char** argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 100000;
    long certified = 0, wrong[kForms] = {}, total = 0;
    for (long it = 0; it < cases; it++) {
        // one kind of scale at a time, every other case any combination
        const int form = (next64() & 1) ? (int)(next64() % kForms) : 1 << (int)(next64() % 6);
        double L[3], eye[3], amb[3], dif[3], spec[3], col[3], l2 = 0, em = 0;
        const double ls = form & kLight ? mag(-3, 6) : 1;
        for (int k = 0; k < 3; k++) L[k] = sym();
        const double l0 = std::sqrt(L[0] * L[0] + L[1] * L[1] + L[2] * L[2]);
        for (int k = 0; k < 3; k++) {
            L[k] = L[k] / l0 * ls;
            l2 += L[k] * L[k];
            eye[k] = sym();
        }
        const double e0 = std::sqrt(eye[0] * eye[0] + eye[1] * eye[1] + eye[2] * eye[2]);
        // one scale for positions and camera, or one for each
        double sc[4];
        sc[3] = form & kScene ? mag(-44, 6) : 1;
        for (int v = 0; v < 3; v++) sc[v] = form & kScene && (it & 3) == 1 ? mag(-44, 38) : sc[3];
        for (int k = 0; k < 3; k++) {
            eye[k] *= (2 + 3 * uni()) / e0 * sc[3];
            em = std::fmax(em, std::fabs(eye[k]));
        }
        const bool wide = form & kFactors;
        for (int k = 0; k < 3; k++) {
            amb[k] = wide ? (next64() & 3 ? mag(-12, 6) : 0.0) : 0.2;
            dif[k] = wide ? (next64() & 3 ? mag(-12, 6) : 0.0) : 0.8;
            spec[k] = wide ? (next64() & 3 ? mag(-12, 6) : 0.0) : 1.0;
            col[k] = wide ? (next64() & 3 ? mag(-12, 6) : 0.0) : (double)(next64() % 256) / 255.0;
        }
        fgc::CertParams C;
        memset(&C, 0, sizeof(C));
        C.on = 1;
        C.power = (next64() & 1) ? 32 : 2 + (int)(next64() % 127);
        // what the host asks of a draw before it certifies its fragments
        bool usable = l2 >= 1e-6 && em <= 1e6;
        for (int k = 0; k < 3; k++) {
            const double f[4] = {amb[k], dif[k], spec[k], col[k]};
            for (double v : f) usable = usable && (v == 0 || (v >= 1e-12 && v <= 1e6));
            usable = usable && std::fabs(L[k]) <= 1e6;
        }
        if (!usable) continue;
        C.ln = (float)(std::sqrt(l2) * 1.0001);
        C.emax = (float)(em * 1.0001);
        C.powtol = (float)((C.power + 8) * 1.05 * fgc::kCertU);
        C.unlit = 0xff000000u;
        for (int k = 0; k < 3; k++) {
            C.light[k] = (float)L[k];
            C.eye[k] = (float)eye[k];
            C.ambient[k] = (float)amb[k];
            C.diffuse[k] = (float)dif[k];
            C.specular[k] = (float)spec[k];
            C.color255[k] = (float)(col[k] * 255.0);
            C.unlit |= u8(min1(col[k] * amb[k])) << (8 * k);
        }
        double n[3][3], p[3][3], r[3], b[3], base[3];
        const double ns = form & kNormals ? mag(-44, 38) : 1, ws = form & kW ? mag(-20, 20) : 1;
        for (int k = 0; k < 3; k++) base[k] = (next64() & 1) ? sym() : eye[k] / e0 / sc[3] + L[k] / ls;
        for (int v = 0; v < 3; v++) {
            const double nv = form & kNormals && (it & 4) ? mag(-44, 38) : ns;
            for (int k = 0; k < 3; k++) {
                n[v][k] = (base[k] + 0.05 * sym()) * nv;
                p[v][k] = sym() * sc[v];
            }
            r[v] = (form & kW && (it & 8) ? mag(-20, 20) : ws) / (0.5 + 4 * uni());
        }
        b[0] = uni();
        b[1] = uni() * (1 - b[0]);
        b[2] = 1 - b[0] - b[1];
        if (form & kWeights) b[next64() % 3] = (next64() & 7) ? mag(-60, 0) : 0;
        // FP64, the reference's order
        double w[4] = {b[0] * r[0], b[1] * r[1], b[2] * r[2], 0};
        w[3] = 1 / (w[0] + w[1] + w[2]);
        double N[3], P[3], c[3], refl[3];
        for (int k = 0; k < 3; k++) {
            N[k] = (((0 + n[0][k] * w[0]) + n[1][k] * w[1]) + n[2][k] * w[2]) * w[3];
            P[k] = (((0 + p[0][k] * w[0]) + p[1][k] * w[1]) + p[2][k] * w[2]) * w[3];
        }
        double q = 1 / std::sqrt(N[0] * N[0] + N[1] * N[1] + N[2] * N[2]);
        for (int k = 0; k < 3; k++) N[k] *= q;
        const double ndl = N[0] * L[0] + N[1] * L[1] + N[2] * L[2];
        const double diffuse = ndl > 0 ? ndl : ndl == ndl ? 0 : ndl;
        double light[3];
        for (int k = 0; k < 3; k++) light[k] = amb[k] + dif[k] * diffuse;
        if (diffuse > 0) {
            for (int k = 0; k < 3; k++) c[k] = eye[k] - P[k];
            q = 1 / std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
            for (int k = 0; k < 3; k++) c[k] *= q;
            const double m = 2 * (N[0] * -L[0] + N[1] * -L[1] + N[2] * -L[2]);
            for (int k = 0; k < 3; k++) refl[k] = -L[k] - N[k] * m;
            const double sp = c[0] * refl[0] + c[1] * refl[1] + c[2] * refl[2];
            if (sp > 0) {
                const double pw = go_pow(sp, C.power);
                for (int k = 0; k < 3; k++) light[k] = light[k] + spec[k] * pw;
            }
        }
        uint32_t want = 0xff000000u;
        for (int k = 0; k < 3; k++) want |= u8(min1(col[k] * light[k])) << (8 * k);
        float pf[3][3], nf[3][3], rf[3], bf[3];
        for (int v = 0; v < 3; v++) {
            for (int k = 0; k < 3; k++) {
                pf[v][k] = (float)p[v][k];
                nf[v][k] = (float)n[v][k];
            }
            rf[v] = (float)r[v];
            bf[v] = fgc::cert_bary(b[v]);
        }
        uint32_t got = 0;
        const bool ok = fgc::cert_shade(C, bf[0], bf[1], bf[2], rf[0], rf[1], rf[2], pf[0], pf[1], pf[2], nf[0], nf[1],
                                        nf[2], &got);
        if (ok && got != want && wrong[form]++ == 0)
            printf("form %d power %d: %08x, FP64 %08x\n", form, C.power, got, want);
        // the same fragment with vertex colours
        double vc[3][3];
        float vf[3][3];
        uint32_t wantv = 0x7b000000u;
        for (int v = 0; v < 3; v++)
            for (int k = 0; k < 3; k++) {
                vc[v][k] = wide ? (next64() & 3 ? mag(-14, 7) : 0.0) : (double)(next64() % 256) / 255.0;
                vf[v][k] = (float)vc[v][k];
            }
        for (int k = 0; k < 3; k++) {
            const double i = (((0 + vc[0][k] * w[0]) + vc[1][k] * w[1]) + vc[2][k] * w[2]) * w[3];
            wantv |= u8(min1(i * light[k])) << (8 * k);
        }
        uint32_t gotv = 0;
        const bool okv = fgc::cert_shade_vertex(C, fgc::f32_trunc(w[0]), fgc::f32_trunc(w[1]), fgc::f32_trunc(w[2]),
                                                pf[0], pf[1], pf[2], nf[0], nf[1], nf[2], vf[0], vf[1], vf[2],
                                                0x7b000000u, &gotv);
        if (okv && gotv != wantv && wrong[form]++ == 0)
            printf("vertex colours, form %d power %d: %08x, FP64 %08x\n", form, C.power, gotv, wantv);
        certified += ok;
        total++;
    }
    long sum = 0;
    for (long x : wrong) sum += x;
    if (sum) {
        printf("%ld certified words differ\n", sum);
        return 1;
    }
    printf("ok %.5f\n", (double)certified / (total ? total : 1));
    return 0;
}
