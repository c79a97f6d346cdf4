// Goes through fit_raster and place_raster (fauxgl_gb300/csrc/fgc_rasterfit.cuh)
// for every fragment cap, bands of many widths, both barycentric sizes and both
// kinds of passes: every array must start on a multiple of its element's size, the
// whole must fit, and the widths that are accepted are those that a buffer of 51
// bytes a fragment beside 10,240 bytes has room for, the cap reduced in steps of
// 128 above 512 and halved above 256. Prints "ok <cases>" or the first fault.
// Build: g++ -O2 -std=c++17 rasterfit_check.cpp
#include <cstdio>

#include "../fauxgl_gb300/csrc/fgc_rasterfit.cuh"

using namespace fgc;

alignas(16) static unsigned char base[1 << 20];

int main() {
    const long per_sm = 233472, optin = 232448, reserved = 1024;  // sm_103a
    long cases = 0;
    for (long stat : {928L, 1056L})
        for (int i = 0; i < 4200; i++) {
            const int cap = i < 4190 ? 256 + i : 0x7fffffff >> (i - 4190) % 3;
            for (int64_t L = 1; L < 60000; L = L < 40 ? L + 1 : L > 25000 && L < 27000 ? L + 13 + i % 7 : L + L / 9 + i % 7)
                for (int bsize : {4, 8})
                    for (bool large : {false, true}) {
                        RasterFit f;
                        const bool fits = fit_raster(per_sm / 2 - reserved - stat, optin - stat, cap, L, L, bsize, large, f);
                        int least = cap < 4096 ? cap : 4096;
                        while (least > 512) least -= 128;
                        while (least > 256) least /= 2;
                        if (fits != (8 * L + 51 * least + 10240 <= 231520)) {
                            printf("cap %d L %lld: %s\n", cap, (long long)L, fits ? "accepted" : "refused");
                            return 1;
                        }
                        if (!fits) continue;
                        RasterArrays a;
                        const unsigned char* end = place_raster(a, base, (int)L, f.F, f.su, f.heads, bsize, f.rounds);
                        const void* eight[] = {a.depth, a.fz, bsize == 8 ? (void*)a.bd : base, a.uw0, a.uw1, a.uw2};
                        const void* four[] = {a.bf, a.fkey, a.uprim, a.urow, a.ux, a.ucnt, a.ufrag};
                        const void* two[] = {a.head, a.nxt};
                        const size_t bytes = (size_t)(end - base);
                        bool good = f.F >= 128 && f.F <= 4096 && f.smem <= (size_t)(optin - stat) && bytes <= f.smem &&
                                    f.smem - bytes < 16 && (f.su == kSpanUnitsMin || f.su == kSpanUnitsMax);
                        for (const void* o : eight) good = good && ((const unsigned char*)o - base) % 8 == 0;
                        for (const void* o : four) good = good && ((const unsigned char*)o - base) % 4 == 0;
                        for (const void* o : two) good = good && ((const unsigned char*)o - base) % 2 == 0;
                        if (!good) {
                            printf("cap %d L %lld bsize %d large %d: F %d, span values at %ld, %zu bytes\n", cap,
                                   (long long)L, bsize, large, f.F, (long)((unsigned char*)a.uw0 - base), bytes);
                            return 1;
                        }
                        cases++;
                    }
        }
    printf("ok %ld\n", cases);
    return 0;
}
