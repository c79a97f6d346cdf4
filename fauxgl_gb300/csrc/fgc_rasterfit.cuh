// fgc_rasterfit.cuh -- the raster kernel's dynamic shared memory: its layout,
// used by the kernel, and the fragment buffer, span arrays and bucket lists
// that a pass's largest band leaves room for, chosen by the host.
// tests/test_rasterfit.py goes through the sizes on the CPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "fgc_fpjump.cuh"

namespace fgc {

// Pixel buckets of the raster kernel's per-chunk fragment lists: as many as a
// band has pixels by default, so that only fragments of one pixel share a
// list; fewer where a row is longer than that and pixels share buckets anyway,
// which leaves 4 KB for fragments (7680 pixels a row: 2.68 -> 2.59 ms).
constexpr int kRasterHeadsMin = 2048;
constexpr int kRasterHeadsMax = 4096;

// (primitive, row) units a chunk of wide primitives holds: kSpanUnitsMax
// (the span arrays then also hold the narrow walk's warp queues) unless
// shared memory cannot hold it, else kSpanUnitsMin. A primitive with more rows in a band than a chunk holds
// (wrap-around rows of a box beyond the frame's sides) is split over chunks.
constexpr int kSpanUnitsMin = 128;
constexpr int kSpanUnitsMax = 256;

// A band's depth (8 bytes a pixel) and 51 bytes for each of the smallest_buffer
// fragments at most; a wider frame is refused. 26,028 pixels with the default
// cap, up to 26,844 with a smaller one.
constexpr int64_t kBandBytesMax = 8 * 26028 + 51 * 256;

// The smallest fragment buffer that the widest frames lead a cap to.
inline int smallest_buffer(int frag_cap) {
    int F = std::max(256, std::min(frag_cap, 4096));
    while (F > 512) F -= 128;
    while (F > 256) F /= 2;
    return F;
}

// Direct rounds (a unit per thread each) a chunk may take before its fragments
// are shaded and resolved; one for frames too wide to hold their units. A
// wireframe overlay leaves 55 fragments of 250 units after the early depth
// test, and the phases after the walk were 40 % of its time: raster stage 5.12
// ms with one round, 4.73 with two, 4.61 with three or four; 1080p dense 280,
// 270, 266, 290 us (four rounds' memory is the L1 cache's).
constexpr int kChunkRounds = 3;

// The raster kernel's dynamic shared memory, for bands of L pixels, a fragment
// buffer of F with barycentrics of bsize bytes, su span units, heads pixel
// buckets and the units of `rounds` rounds. The colour buffer is not staged: the
// band's pixels are read and written in global memory by the CTA that owns them.
struct RasterArrays {
    double* depth;   // [L]
    double* fz;      // [F]
    float* bf;       // [3][F] barycentrics for FP32 shading; or, the same memory,
    double* bd;      // [3][F] for FP64 shading of every fragment (exact)
    int fcap;        // F
    uint32_t* fkey;  // [F] (pixel << 16) | unit
    double* uw0;     // [su] unit -> edge values at its first covered in-band pixel
    double* uw1;
    double* uw2;
    uint32_t* uprim; // [rounds * 256] unit -> primitive
    int32_t* urow;   // [rounds * 256] unit -> row y
    int32_t* ux;     // [su] unit -> first covered in-band x
    uint32_t* ucnt;  // [su] unit -> covered in-band pixels
    uint32_t* ufrag; // [su] unit -> first fragment offset in the chunk
    unsigned short* head;  // [heads] per pixel bucket: last fragment of its list (0xFFFF: none)
    unsigned short* nxt;   // [F] per fragment: the previous fragment in its bucket
    uint8_t* fflag;  // [F] discard / blend / pending flags
};

// Places the arrays from q (16-byte aligned) on and returns their end. With
// barycentrics of 4 bytes those after them are aligned only for an even F
// (fit_raster makes it a multiple of 8).
FGC_HD unsigned char* place_raster(RasterArrays& S, unsigned char* q, int L, int F, int su, int heads, int bsize,
                                   int rounds) {
    S.depth = (double*)q; q += (size_t)L * 8;
    S.fz = (double*)q; q += (size_t)F * 8;
    S.bf = (float*)q;
    S.bd = (double*)q;
    q += (size_t)F * 3 * bsize;
    S.fcap = F;
    S.uw0 = (double*)q; q += (size_t)su * 8;
    S.uw1 = (double*)q; q += (size_t)su * 8;
    S.uw2 = (double*)q; q += (size_t)su * 8;
    S.fkey = (uint32_t*)q; q += (size_t)F * 4;
    S.uprim = (uint32_t*)q; q += (size_t)rounds * 256 * 4;
    S.urow = (int32_t*)q; q += (size_t)rounds * 256 * 4;
    S.ux = (int32_t*)q; q += (size_t)su * 4;
    S.ucnt = (uint32_t*)q; q += (size_t)su * 4;
    S.ufrag = (uint32_t*)q; q += (size_t)su * 4;
    S.head = (unsigned short*)q; q += (size_t)heads * 2;
    S.nxt = (unsigned short*)q; q += (size_t)F * 2;
    S.fflag = (uint8_t*)q;
    return q + F;
}

// Bytes of it.
inline size_t raster_smem_bytes(int64_t L, int F, int su, int heads, int bsize, int rounds) {
    const size_t b = (size_t)L * 8 + (size_t)F * (8 + 3 * bsize + 4 + 2 + 1) + (size_t)su * (8 * 3 + 4 * 3) +
                     (size_t)rounds * 256 * 4 * 2 + (size_t)heads * 2;
    return (b + 15) & ~(size_t)15;
}

struct RasterFit {
    int F, su, heads, rounds;
    size_t smem;
};

// The raster kernel's buffers for bands of up to L pixels within two_cta bytes
// (two CTAs per SM) or else one_cta. Lset: the band that the caller's tuning asks
// for, at least L. large: the pass's primitives cover several pixels and have row
// starts. False when the frame, or the tuning's band, is too wide.
inline bool fit_raster(long two_cta, long one_cta, int frag_cap, int64_t L, int64_t Lset, int bsize, bool large,
                       RasterFit& f) {
    const auto size = [&] { f.smem = raster_smem_bytes(L, f.F, f.su, f.heads, bsize, f.rounds); };
    // primitives of several pixels fill a larger buffer in one round of units
    // (kRowTablePixelsPerElement); small ones do not, and its memory is then
    // better left to the L1 cache (raster stage at twice the cap: 48 mixed
    // thumbnails 2.33 -> 2.13 ms, a close-up 231 -> 218 us; a dense 1080p frame at
    // 1.5 times 295 -> 315 us)
    const int cap = std::min(frag_cap, 4096);
    f.F = std::max(256, std::min(large ? 2 * cap : cap, 4096)) & ~7;
    f.heads = L > kRasterHeadsMax ? kRasterHeadsMin : kRasterHeadsMax;
    f.rounds = kChunkRounds;
    // the larger span arrays first: they also hold the warp queues of the
    // narrow walk, which needs one 32-entry queue per warp (kSpanUnitsMax =
    // the CTA's threads) and is worth more than a larger fragment buffer
    f.su = kSpanUnitsMax;
    size();
    // two CTAs per SM (the register budget allows two) when a smaller
    // fragment buffer makes them fit
    while ((long)f.smem > two_cta && f.F > 512) {
        f.F -= 128;
        size();
    }
    while ((long)f.smem > one_cta && f.F > 256) {
        f.F = f.F / 2 & ~7;
        size();
    }
    if ((long)f.smem > one_cta) {
        f.heads = kRasterHeadsMin;
        f.rounds = 1;
        size();
    }
    if ((long)f.smem > one_cta) {
        // the smaller span arrays (narrow rows then walk thread by thread)
        f.su = kSpanUnitsMin;
        size();
    }
    if ((long)f.smem > one_cta) {
        f.F = smallest_buffer(frag_cap) & ~7;
        size();
    }
    return Lset * 8 + smallest_buffer(frag_cap) * 51 <= kBandBytesMax && (long)f.smem <= one_cta;
}

}  // namespace fgc
