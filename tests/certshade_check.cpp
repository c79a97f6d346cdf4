// Checks cert_shade (fauxgl_gb300/csrc/fgc_certshade.cuh) against an FP64
// evaluation of PhongShader.Fragment in the reference's operation order
// (shader.go:75-96, color.go:56-63): every certified NRGBA word must be the
// FP64 one. Inputs: smooth, flat, opposing and unnormalised vertex normals,
// near and far cameras, edge-on light, highlights, 8-bit and saturating
// colours, zero weights, and non-finite attributes (which must be refused).
// The FP32 reciprocal square root is perturbed by up to 2 ulp both ways, the
// device function's stated error. Prints "ok <certified share>" or the first
// mismatch. Build: g++ -O2 -ffp-contract=off -std=c++17 certshade_check.cpp
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../fauxgl_gb300/csrc/fgc_certshade.cuh"

static uint64_t g_state = 0x853c49e6748fea9bull;
static uint64_t next64() {
    uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double uni() { return (double)(next64() >> 11) / 9007199254740992.0; }
static double sym() { return 2 * uni() - 1; }

static uint32_t u8(double c) {
    if (!(c == c)) return 0;
    c = c < 0 ? 0 : c > 1 ? 1 : c;
    return (uint32_t)(c * 255.0);
}

// Go's math.Pow for an integer power: repeated squaring of the Frexp mantissa.
static double go_pow(double x, int p) {
    if (x == 0) return 0;
    int xe;
    double x1 = std::frexp(x, &xe), a1 = 1;
    long long ae = 0, e = xe;
    for (int i = p; i != 0; i >>= 1) {
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
    return std::ldexp(a1, (int)(ae < -100000 ? -100000 : ae));
}

int main(int argc, char** argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 100000;
    const int powers[] = {2, 3, 7, 32, 50, 64, 128};
    long certified = 0, ordinary = 0, ordinary_cert = 0, vertex_cert = 0;
    for (long it = 0; it < cases; it++) {
        const int form = (int)(next64() % 8);
        fgc::CertParams C;
        memset(&C, 0, sizeof(C));
        double L[3], eye[3], amb, dif, spec, col[3], ln = 0, em = 0;
        for (int k = 0; k < 3; k++) L[k] = sym();
        const double lscale = form == 5 ? 3 * uni() + 0.1 : 1;
        const double l0 = std::sqrt(L[0] * L[0] + L[1] * L[1] + L[2] * L[2]);
        const double er = form == 6 ? 40 * uni() + 1.2 : 2 + 3 * uni();
        for (int k = 0; k < 3; k++) {
            L[k] = L[k] / l0 * lscale;
            ln += L[k] * L[k];
            eye[k] = sym();
        }
        const double e0 = std::sqrt(eye[0] * eye[0] + eye[1] * eye[1] + eye[2] * eye[2]);
        for (int k = 0; k < 3; k++) {
            eye[k] *= er / e0;
            em = std::fmax(em, std::fabs(eye[k]));
        }
        amb = (next64() & 1) ? 0.2 : uni();
        dif = (next64() & 1) ? 0.8 : uni() * 2;
        spec = (next64() & 1) ? 1.0 : uni();
        for (int k = 0; k < 3; k++) col[k] = (next64() & 3) ? (double)(next64() % 256) / 255.0 : uni() * 1.5;
        C.on = 1;
        C.power = powers[next64() % 7];
        C.ln = (float)(std::sqrt(ln) * 1.0001);
        C.emax = (float)(em * 1.0001);
        C.powtol = (float)((C.power + 8) * 1.05 * fgc::kCertU);
        C.unlit = 0xff000000u;
        for (int k = 0; k < 3; k++) {
            C.light[k] = (float)L[k];
            C.eye[k] = (float)eye[k];
            C.ambient[k] = (float)amb;
            C.diffuse[k] = (float)dif;
            C.specular[k] = (float)spec;
            C.color255[k] = (float)(col[k] * 255.0);
            const double c = col[k] * amb;
            C.unlit |= u8(c < 1 ? c : 1) << (8 * k);
        }
        double n[3][3], p[3][3], r[3], b[3], base[3];
        for (int k = 0; k < 3; k++) base[k] = sym();
        if (form == 2) {  // edge-on light: the base normal nearly perpendicular to it
            double d = 0;
            for (int k = 0; k < 3; k++) d += base[k] * L[k];
            for (int k = 0; k < 3; k++) base[k] -= L[k] * d / ln * (1 - 1e-6 * sym());
        }
        if (form == 3) {  // a highlight: the normal halves eye and light
            for (int k = 0; k < 3; k++) base[k] = eye[k] / er + L[k] / std::sqrt(ln) + 0.05 * sym();
        }
        for (int v = 0; v < 3; v++) {
            double q = 0;
            const double spread = form == 1 ? 0.0 : form == 4 ? 1.5 : 0.05;
            for (int k = 0; k < 3; k++) {
                n[v][k] = base[k] + spread * sym();
                p[v][k] = (v ? p[0][k] + 0.02 * sym() : sym());
                q += n[v][k] * n[v][k];
            }
            if (form != 5)
                for (int k = 0; k < 3; k++) n[v][k] /= std::sqrt(q);
            r[v] = 1 / (0.5 + 4 * uni());
        }
        if (form == 1)
            for (int k = 0; k < 3; k++) n[1][k] = n[2][k] = n[0][k];
        b[0] = uni();
        b[1] = uni() * (1 - b[0]);
        b[2] = 1 - b[0] - b[1];
        if (next64() % 16 == 0) b[next64() % 3] = 0;
        const bool bad = form == 7 && (next64() & 1);
        if (bad) {
            const double evil[] = {NAN, INFINITY, -INFINITY, 1e300};
            const double e = evil[next64() % 4];
            switch (next64() % 3) {
                case 0: n[next64() % 3][next64() % 3] = e; break;
                case 1: p[next64() % 3][next64() % 3] = e; break;
                default: b[next64() % 3] = std::fabs(e); break;
            }
        }
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
        double light = amb + dif * diffuse;
        if (diffuse > 0) {
            for (int k = 0; k < 3; k++) c[k] = eye[k] - P[k];
            q = 1 / std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
            for (int k = 0; k < 3; k++) c[k] *= q;
            const double m = 2 * (N[0] * -L[0] + N[1] * -L[1] + N[2] * -L[2]);
            for (int k = 0; k < 3; k++) refl[k] = -L[k] - N[k] * m;
            const double sp = c[0] * refl[0] + c[1] * refl[1] + c[2] * refl[2];
            if (sp > 0) light = light + spec * go_pow(sp, C.power);
        }
        uint32_t want = 0xff000000u;
        for (int k = 0; k < 3; k++) {
            const double v = col[k] * light;
            want |= u8(v < 1 ? v : v == v ? 1 : v) << (8 * k);
        }
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
        if (ok && got != want) {
            printf("case %ld form %d power %d: %08x, FP64 %08x\n", it, form, C.power, got, want);
            return 1;
        }
        // the same fragment with vertex colours
        double vc[3][3];
        float vf[3][3];
        uint32_t wantv = 0x7b000000u;
        const uint64_t kind = next64();
        for (int v = 0; v < 3; v++)
            for (int k = 0; k < 3; k++) {
                vc[v][k] = kind & 1 ? (double)(next64() % 256) / 255.0 : uni() * 1.5;
                if (kind % 8 == 2 && v) vc[v][k] = vc[0][k];
                if (kind % 64 == 4) vc[v][k] = (next64() & 1) ? 0.0 : -uni();
                vf[v][k] = (float)vc[v][k];
            }
        for (int k = 0; k < 3; k++) {
            const double i = (((0 + vc[0][k] * w[0]) + vc[1][k] * w[1]) + vc[2][k] * w[2]) * w[3];
            const double v = i * light;
            wantv |= u8(v < 1 ? v : v == v ? 1 : v) << (8 * k);
        }
        uint32_t gotv = 0;
        const bool okv = fgc::cert_shade_vertex(C, fgc::f32_trunc(w[0]), fgc::f32_trunc(w[1]), fgc::f32_trunc(w[2]),
                                                pf[0], pf[1], pf[2], nf[0], nf[1], nf[2], vf[0], vf[1], vf[2],
                                                0x7b000000u, &gotv);
        if (okv && gotv != wantv) {
            printf("vertex colours, case %ld form %d power %d: %08x, FP64 %08x\n", it, form, C.power, gotv, wantv);
            return 1;
        }
        certified += ok;
        if (form == 0 || form == 1) {
            ordinary++;
            ordinary_cert += ok;
            vertex_cert += okv;
        }
    }
    if (ordinary_cert < 0.95 * ordinary || vertex_cert < 0.9 * ordinary) {
        printf("only %ld (vertex colours %ld) of %ld ordinary fragments certified\n", ordinary_cert, vertex_cert, ordinary);
        return 1;
    }
    printf("ok %.5f of all, %.5f of ordinary\n", (double)certified / cases, (double)ordinary_cert / ordinary);
    return 0;
}
