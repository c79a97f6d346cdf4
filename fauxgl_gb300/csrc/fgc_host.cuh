// fgc_host.cuh -- host-side objects of libfauxglcuda shared by the C ABI
// (fgc_api.cu) and the pass engine (fgc_pass.cu): device buffers, the
// mesh / texture / context handles, and the pass interface.
//
// A pass renders any number of draws (a mesh range, state, shader and
// target context each) with one launch per pipeline stage. DrawMesh /
// DrawTriangles / DrawLines run a pass of one draw and wait for it, because
// the reference returns RasterizeInfo by value (context.go:391-439); the
// batch interface runs passes of many draws asynchronously.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <shared_mutex>
#include <string>
#include <vector>

#include "fgc_internal.cuh"

namespace fgc {

// Record msg as the calling thread's last error and return code.
int fail(int code, const std::string& msg);

#define FGC_CUDA(call)                                                                                             \
    do {                                                                                                           \
        cudaError_t e_ = (call);                                                                                   \
        if (e_ != cudaSuccess) return ::fgc::fail(FGC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Device memory comes from stream-ordered pools, three per device: the
// temporaries of the calls that make and edit meshes, the arrays of meshes,
// and everything else (framebuffers, a context's or batch's scratch).
// cudaMalloc and cudaFree (which waits for the device) took most of the time
// of mesh calls, which allocate up to two dozen arrays: LoadSTL of 327,680
// triangles 2.8 ms, SmoothNormals 1.3 ms, a mesh of 81,920 uploaded for one
// draw 1.6 ms; from the pools they take 0.29, 0.26 and 0.28 ms. The first draw
// into a new 1080p context, which allocates its scratch, takes 1.27 ms instead
// of 2.36. Each pool keeps at most kPoolKeep bytes of freed memory (the driver
// returns the rest when a stream synchronises), so that many resident meshes
// or large frames do not take the temporaries' share. When the library's last
// object on the device is released they go back to kPoolIdle bytes, and
// fgc_trim_memory gives back everything unused at any time. The pools are the
// driver's, so threads and streams may use them together: memory freed on one
// stream is handed to another only once that free has taken effect.
constexpr uint64_t kPoolKeep = 1ull << 30;
constexpr uint64_t kPoolIdle = 128ull << 20;
// Frame and scratch buffers from this size on are allocations of their own: a
// pool grows in small pieces, and one that has to grow by several GB takes
// longer than cudaMalloc (first pass over a 7680x4320 frame with a wireframe
// overlay 14.9 -> 11.7 ms).
constexpr size_t kPoolBufMax = 64ull << 20;
enum PoolKind { kPoolTemp, kPoolMesh, kPoolFrame, kPoolKinds };
cudaError_t pool_alloc(PoolKind kind, void** p, size_t bytes, cudaStream_t s);
void pool_free(void* p, cudaStream_t s);
// cudaMalloc, the pools' kept memory given back first where it is in the way.
cudaError_t big_alloc(void** p, size_t bytes);
// The current device's pools reduced to `keep` bytes each, as far as their
// memory is unused.
cudaError_t trim_pools(uint64_t keep);
// An object (context, batch, mesh, texture) on a device; the first member of
// its struct, so that it is destroyed after the buffers.
struct Live {
    int device = -1;
    Live() = default;
    Live(const Live&) = delete;
    Live& operator=(const Live&) = delete;
    void on(int dev);
    ~Live();
};
// A stream of the device for one call (kept for later calls, at most eight)
// and its return. free_stream: the stream on which memory outliving its call
// is freed, once nothing uses it any more.
cudaError_t take_stream(int device, cudaStream_t* s);
void give_stream(int device, cudaStream_t s);
cudaStream_t free_stream();
// Waits for all work of the current device. While a thread captures a stream
// cudaDeviceSynchronize is not permitted to any thread -- it breaks the capture
// --, so batches hold capture_mutex shared while they capture, and this call
// holds it alone.
std::shared_mutex& capture_mutex();
void device_wait();

// Arrays of meshes and their temporaries from this size on are allocations of
// their own as well: a pool that keeps 1 GiB grows and shrinks by the rest on
// every call. Upload of 12 M triangles 22.6 -> 19.0 ms (20.2 with cudaMalloc
// throughout), upload, smoothing, sharp edges and release of 6 M / 12 M / 24 M
// 14.8 / 36 / - -> 13.4 / 29.0 / 61 ms; from 256 MiB on they take 14.7 / 30.2 /
// 64 ms, from 1 GiB on 14.3 / 31.5 / 63, and 3 M triangles, whose arrays are
// smaller than 512 MiB, 5.7 ms (6.7 from 256 MiB on).
constexpr size_t kPoolOwnMin = 512ull << 20;

// n elements of pool memory in the order of stream s: a call's temporary (Kept
// false: freed in that order as well) or an array of a mesh (Kept true).
template <typename T, bool Kept>
struct PoolBuf {
    T* p = nullptr;
    size_t cap = 0;
    cudaStream_t s = nullptr;
    PoolBuf() = default;
    PoolBuf(const PoolBuf&) = delete;
    PoolBuf& operator=(const PoolBuf&) = delete;
    ~PoolBuf() { release(); }
    void release() {
        if (p && cap * sizeof(T) >= kPoolOwnMin) {
            if (!Kept) cudaStreamSynchronize(s);
            cudaFree(p);
        } else if (p) {
            pool_free(p, Kept ? free_stream() : s);
        }
        p = nullptr;
        cap = 0;
    }
    cudaError_t ensure(size_t n, cudaStream_t stream) {
        if (n <= cap && p) return cudaSuccess;
        release();
        s = stream;
        const size_t want = std::max<size_t>(n, 1), bytes = want * sizeof(T);
        const cudaError_t e = bytes >= kPoolOwnMin ? big_alloc((void**)&p, bytes)
                                                   : pool_alloc(Kept ? kPoolMesh : kPoolTemp, (void**)&p, bytes, stream);
        if (e != cudaSuccess) {
            p = nullptr;
            return e;
        }
        cap = want;
        return cudaSuccess;
    }
};
template <typename T>
using TempBuf = PoolBuf<T, false>;
template <typename T>
using MeshBuf = PoolBuf<T, true>;

// A buffer that any stream may use: its allocation has taken effect before it
// is used. Its owner sees to it that nothing uses it any more when it is
// released or grows: contexts and batches wait for their streams, also where a
// call fails, meshes and textures for the device. (Waiting for the device here
// would break the graph capture of another thread, see device_wait.)
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t cap = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) {
            if (cap * sizeof(T) >= kPoolBufMax) cudaFree(p);
            else pool_free(p, free_stream());
        }
        p = nullptr;
        cap = 0;
    }
    // Make room for n elements (contents not preserved when it grows); user: the
    // stream whose work may use the buffer still.
    cudaError_t ensure(size_t n, cudaStream_t user) {
        if (n > cap && p) cudaStreamSynchronize(user);
        return ensure(n);
    }
    cudaError_t ensure(size_t n) {
        if (n <= cap && p) return cudaSuccess;
        release();
        size_t want = std::max<size_t>(n + n / 4, 64);
        cudaError_t e;
        if (want * sizeof(T) >= kPoolBufMax) {
            e = big_alloc((void**)&p, want * sizeof(T));
        } else {
            const cudaStream_t s = free_stream();
            e = pool_alloc(kPoolFrame, (void**)&p, want * sizeof(T), s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        }
        if (e != cudaSuccess) {
            p = nullptr;
            return e;
        }
        cap = want;
        return cudaSuccess;
    }
};

// Page-locked host staging (the table upload and the results of a pass).
struct PinnedBuf {
    unsigned char* p = nullptr;
    size_t cap = 0;
    PinnedBuf() = default;
    PinnedBuf(const PinnedBuf&) = delete;
    PinnedBuf& operator=(const PinnedBuf&) = delete;
    ~PinnedBuf() { release(); }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
    cudaError_t ensure(size_t n) {
        if (n <= cap && p) return cudaSuccess;
        release();
        size_t want = std::max<size_t>(n + n / 4, 4096);
        cudaError_t e = cudaMallocHost((void**)&p, want);
        if (e != cudaSuccess) {
            p = nullptr;
            return e;
        }
        cap = want;
        return cudaSuccess;
    }
};

constexpr int kRasterThreads = 256;

// The look-back of the draw pipeline's ordered allocations and scans: the
// limit on polls of an unpublished predecessor (kSpinLimit) and no withheld
// block, unless fgc_debug_lookback set a test configuration.
extern std::atomic<uint32_t> g_lookback_spin_limit;
extern std::atomic<uint32_t> g_lookback_withhold;
inline Lookback draw_lookback(unsigned long long* tiles, unsigned int* ticket, unsigned int* status,
                              unsigned long long* total) {
    Lookback L{tiles, ticket, status, total};
    L.spin_limit = g_lookback_spin_limit.load(std::memory_order_relaxed);
    L.withhold = g_lookback_withhold.load(std::memory_order_relaxed);
    return L;
}
constexpr int kMaxBands = 24576;

uint32_t pack_nrgba_host(const double c[4]);
int grid_for(uint64_t n, int block, int cap);

// Shared-memory limits of a device and the raster kernels' static usage,
// read once per device.
struct DevLimits {
    int device = -1;
    int sms = 1;
    int smem_per_sm = 0;
    int smem_per_block_optin = 0;
    int smem_reserved_per_block = 0;
    int raster_static[2] = {0, 0};  // plain, mixed
};
int dev_limits(int device, const DevLimits** out);

}  // namespace fgc

struct fgc_texture {
    fgc::Live live;
    int device = 0;
    int32_t w = 0, h = 0;
    fgc::DevBuf<ushort4> texels;
    fgc::DevBuf<double> unit64;  // 4 per texel: the channels as float64(c) / 0xffff
};

struct fgc_mesh {
    fgc::Live live;
    int device = 0;
    uint64_t ntri = 0, nline = 0, nuniq = 0;
    fgc::MeshBuf<double> ux, uy, uz;
    fgc::MeshBuf<uint32_t> corner_uniq;
    fgc::MeshBuf<fgc::APosNrm64> pn64;
    fgc::MeshBuf<fgc::APosNrm32> pn32;
    fgc::MeshBuf<double> tex64, col64;
    fgc::MeshBuf<float> tex32, col32;
    bool has_tex = false, has_col = false;
    bool plain_positions = false;  // no coordinate is -0 or NaN: equal positions have equal bits

    fgc::MeshView view() const {
        fgc::MeshView v;
        v.ntri = ntri;
        v.nline = nline;
        v.nuniq = nuniq;
        v.upos_x = ux.p;
        v.upos_y = uy.p;
        v.upos_z = uz.p;
        v.corner_uniq = corner_uniq.p;
        v.pn64 = pn64.p;
        v.tex64 = has_tex ? tex64.p : nullptr;
        v.col64 = has_col ? col64.p : nullptr;
        v.pn32 = pn32.p;
        v.tex32 = has_tex ? tex32.p : nullptr;
        v.col32 = has_col ? col32.p : nullptr;
        return v;
    }
};

// Weld device corner positions cp (3 doubles per corner) into m and fill its
// position/normal records from nrm (device, or null for zero normals).
int mesh_weld_attrs(fgc_mesh* m, cudaStream_t s, int sms, const double* cp, const double* nrm, uint64_t V);

namespace fgc {

// Pass-wide device counters (one block per pass; the status word is shared by
// all passes of one submission so that a later pass skips its raster stage
// once an earlier one has overflowed).
struct PassCounters {
    unsigned int clip_count;
    unsigned int lclip_count;
    unsigned int band_counter;
    unsigned int tick_setup;
    unsigned int tick_scan;
    unsigned int tick_rscan;
    unsigned long long prim_total;
    unsigned long long pair_total;
    unsigned long long reserved;
    unsigned long long work_total;  // setup work items of the pass
    unsigned long long pad1;
};

// Tunable shapes of a pass; results do not depend on them.
struct PassTuning {
    int64_t band_pixels = 4096;         // pixels per band, rounded to whole rows
    int64_t prims_per_bin_block = 4096; // raster primitives per binning block
    int frag_cap = 1024;                // raster fragment buffer at most, rounded down to a multiple of 8 (twice it for large primitives; 4096)
    int window = 8;                     // accepted and reported; the raster stage sizes its runs itself
};

// One draw of a pass, as the host describes it.
struct PassItem {
    fgc_context* ctx = nullptr;
    const fgc_mesh* mesh = nullptr;
    uint64_t tf = 0, tc = 0, lf = 0, lc = 0;
    StateView sv;
    ShaderView shv;
    bool clear_color = false, clear_depth = false;
    uint32_t clear_color_value = 0;
    double clear_depth_value = 0;
};

// Scratch of the pass pipeline (buffers grow on demand and are reused by the
// passes issued on one stream).
struct PassScratch {
    DevBuf<VClip> vclip;
    DevBuf<double2> vndc;
    DevBuf<VScreen> vscr;
    DevBuf<uint8_t> vout;
    DevBuf<RPrim> prims;
    DevBuf<PBox> pbox;
    DevBuf<float4> rf;
    DevBuf<uint32_t> pspan;
    DevBuf<ClipEntry> clip_list, lclip_list;
    DevBuf<PoolVertex> pool;
    DevBuf<PoolVertex32> pool32;
    DevBuf<ClipPoly> cpoly;        // per clip_list entry: its clipped polygon
    DevBuf<ClipVert> cvert;        // per clip_list entry: the polygon's vertices
    DevBuf<uint32_t> mat, off, bins;
    DevBuf<uint32_t> pnb, prs;     // per primitive: bands it is binned to, first row-start slot
    DevBuf<double> rstart;         // per (primitive, band): edge values at its first row in the band
    DevBuf<unsigned char> table;   // item views + lookup starts + per-draw results + counters + status
    DevBuf<double> dbg;
    DevBuf<PendFrag> pend;         // per raster CTA: fragments awaiting their FP64 colour
    DevBuf<SetupWork> work;        // setup work items (triangles, wireframe edges, lines)
    DevBuf<uint16_t> smeta;        // per element of a setup tile: its setup decision
    DevBuf<uint32_t> cidx;         // per element of a setup tile: its clip_list entry (clipped triangles)
    DevBuf<unsigned long long> tsum;  // per setup tile: its sums, then their exclusive prefix
    PinnedBuf host_in, host_out;
    uint32_t clip_cap = 1024;
    uint64_t bin_cap = 0;
    // the clip kernels run on a second stream beside the setup scan, list
    // writer and emission
    int side_device = -1;
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_clip = nullptr, ev_join = nullptr;
    PassScratch() = default;
    PassScratch(const PassScratch&) = delete;
    PassScratch& operator=(const PassScratch&) = delete;
    ~PassScratch() {
        if (side) cudaStreamSynchronize(side);
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (ev_join) cudaEventDestroy(ev_join);
        if (side) cudaStreamDestroy(side);
    }
};

// The host's record of one issued pass (for reading its results).
struct PassRecord {
    std::vector<uint32_t> items;  // indices into the submission's item list
    size_t in_off = 0;            // offset of its staging in host_in
    size_t out_off = 0;           // offset of its results in host_out
    uint32_t nbands = 0;
    int32_t band_rows = 0;
    uint64_t launches = 0;
};

// A submission: the passes that render a list of draws in order. Draws that
// share a target context or differ in precision go to separate passes.
struct Submission {
    std::vector<PassItem> items;
    std::vector<PassRecord> passes;
    std::vector<fgc_rasterize_info> infos;
    std::vector<std::vector<cudaEvent_t>> events;  // stage boundaries per pass, when timing
    uint32_t cut = 0;             // item that begins a pass of its own accord, or 0
    cudaEvent_t at_cut = nullptr; // recorded before that pass
    fgc_stats stats = {};
    bool timing = false;
    Submission() = default;
    Submission(const Submission&) = delete;
    Submission& operator=(const Submission&) = delete;
    ~Submission();
    void reset();  // before the first issue: clears results, passes and events
};

// Plan the submission's passes and grow the scratch for them (no stream
// work): after it, issue_submission allocates nothing, so it may be captured
// into a CUDA graph.
int prepare_submission(PassScratch& S, const DevLimits& D, const PassTuning& T, const Submission& sub);
// Split items into passes and issue passes [first_pass, end) on stream (no
// host wait), each followed by the copy of its results. The submission's
// status word is zeroed first. An issue that fails has been waited for.
int issue_submission(PassScratch& S, cudaStream_t stream, const DevLimits& D, const PassTuning& T,
                     Submission& sub, size_t first_pass);
// Wait for what a failed issue has left running (nothing while capturing).
void abandon_submission(PassScratch& S, cudaStream_t stream);
// After the stream has drained: read the results of passes [from, end).
// Sets *retry_from = passes.size() when they all succeeded; otherwise grows
// the scratch limits and sets *retry_from to the first pass to re-issue.
int collect_submission(PassScratch& S, Submission& sub, size_t from, size_t* retry_from);
// Wait for passes [from, end) and re-issue failed ones until all succeed.
int finish_submission(PassScratch& S, cudaStream_t stream, const DevLimits& D, const PassTuning& T, Submission& sub,
                      size_t from);
// reset + issue + finish.
int run_submission(PassScratch& S, cudaStream_t stream, const DevLimits& D, const PassTuning& T, Submission& sub);

// Validate a state / shader pair and convert it to device views.
int fill_views(const fgc_state* st, const fgc_shader* sh, StateView& sv, ShaderView& shv);
const char* last_error();

}  // namespace fgc

namespace fgc {
// FGC_ERR_BUSY while a batch has unfinished draws on the context (call with
// the context's mutex held).
int context_ready(const fgc_context* c);
// Allocate the debug buffers the context's flags ask for.
int ensure_debug(fgc_context* c);
}  // namespace fgc

struct fgc_context {
    fgc::Live live;
    int device = 0;
    int sms = 1;
    cudaStream_t stream = nullptr;      // the stream work is issued on
    cudaStream_t own_stream = nullptr;  // the context's own stream
    int32_t W = 0, H = 0;
    int64_t N = 0;
    fgc::DevBuf<uint32_t> color;
    fgc::DevBuf<double> depth;
    bool clear_color_pending = false, clear_depth_pending = false;
    uint32_t clear_color = 0;
    double clear_depth = 1.7976931348623157e308;
    int debug = 0;
    fgc::DevBuf<uint32_t> winner;
    fgc::DevBuf<double> shaded;
    fgc::PassScratch scratch;           // the context's own draws
    fgc::DevBuf<unsigned long long> lohi;
    fgc::DevBuf<uint32_t> ds;
    fgc::DevBuf<uint16_t> gray;
    bool timing = false;
    fgc_stats stats = {};
    const void* busy = nullptr;         // the batch that has unfinished work on this context
    std::mutex mu;
};
