// rcp_i, div_of and sqrt_i (fgc_softdiv.cuh) against the CPU's division and
// square root, bit for bit.
// usage: softdiv_check N   prints "ok N" or the first mismatch
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../fauxgl_gb300/csrc/fgc_softdiv.cuh"

using namespace fgc;

static uint64_t st = 88172645463325252ull;
static uint64_t next64() {
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st * 0x9E3779B97F4A7C15ull;
}

// significands near the ends and the middle of the binade, near powers of two, and any
static uint64_t frac() {
    const uint64_t r = next64(), f = next64() & 0x000fffffffffffffull;
    switch (r % 6) {
        case 0: return f >> (r >> 32) % 52;
        case 1: return 0x000fffffffffffffull - (f >> (r >> 32) % 52);
        case 2: return 1ull << (r >> 32) % 52;
        case 3: return (0x0008000000000000ull + (r >> 60) - 8) & 0x000fffffffffffffull;
        default: return f;
    }
}
static double any(bool edge) {
    const uint64_t s = next64() << 63;
    const uint64_t r = next64();
    uint64_t e = edge ? (r & 1 ? r % 4 : 2047 - r % 5) : 1023 - 40 + r % 80;
    if (edge && (r >> 20) % 8 == 0) return fj_double(s | (e << 52));
    return fj_double(s | (e << 52) | frac());
}
static bool same(double a, double b) { return (a != a && b != b) || fj_bits(a) == fj_bits(b); }

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    for (long i = 0; i < n; i++) {
        const bool edge = i % 16 == 0;
        const double w = any(edge);
        double x = any(edge && (next64() & 1));
        if (i % 16 == 1) x = w * (double)(1 + next64() % 1000);        // exact quotients
        if (i % 16 == 2) x = w * (1 + (double)(next64() % 64) * 0x1p-52);  // quotients next to 1
        SoftRcp r = soft_rcp(w);
        if (i & 1) {  // a seed off by as much as the GPU's may be
            uint32_t f = (uint32_t)(fj_bits(w) >> 29) & 0x7fffffu;
            const float seed = sd_seed(f) * (1.0f + (float)(int)(next64() % 9) * 0x1p-23f - 4 * 0x1p-23f);
            r.y = sd_recip(r.m, seed);
        }
        if (!same(rcp_of(w, r), 1.0 / w)) {
            printf("1 / %a: %a, not %a\n", w, rcp_of(w, r), 1.0 / w);
            return 1;
        }
        if (!same(div_of(x, w, r), x / w)) {
            printf("%a / %a: %a, not %a\n", x, w, div_of(x, w, r), x / w);
            return 1;
        }
    }
    for (long i = 0; i < n; i++) {
        double x = std::fabs(any(i % 16 == 0));
        if (i % 16 == 1) x = std::pow(std::fabs(any(false)), 2);      // near squares
        if (i % 16 == 2) {
            const double r = (double)(0x10000000u + next64() % 0x0fffffffu);
            x = r * r + (double)(int)(next64() % 3) - 1;              // squares and their neighbours
        }
        if (!same(sqrt_i(x), std::sqrt(x))) {
            printf("sqrt %a: %a, not %a\n", x, sqrt_i(x), std::sqrt(x));
            return 1;
        }
        const uint32_t e = (uint32_t)(fj_bits(x) >> 52);
        if (e - 1u < 2046u) {
            const float seed = sd_rseed((uint32_t)(fj_bits(x) >> 29) & 0x7fffffu, (e & 1) == 0) *
                               (1.0f + (float)(int)(next64() % 9) * 0x1p-23f - 4 * 0x1p-23f);
            if (!same(sqrt_seeded(x, seed), std::sqrt(x))) {
                printf("sqrt %a, seed %a: %a, not %a\n", x, (double)seed, sqrt_seeded(x, seed), std::sqrt(x));
                return 1;
            }
        }
    }
    printf("ok %ld\n", n);
    return 0;
}
