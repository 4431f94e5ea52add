// fg_capi.cu -- the render entry points of the C-ABI: buffer staging, launch planning and the
// whole-image orchestration of render_from_workspace_impl (src/lib.rs:134-173).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/film_grain_gb300.h"
#include "fg_host.h"
#include "fg_kernels.cuh"
#include "fg_internal.h"

namespace fg {

static thread_local unsigned long long g_pw_diag[kPwDiagWords] = {0, 0, 0, 0, 0, 0};

fg_status cuda_error(cudaError_t e, const char *what) {
    return set_error(e == cudaErrorMemoryAllocation ? FG_ERR_NOMEM : FG_ERR_CUDA,
                     std::string("gpu error: ") + what + ": " + cudaGetErrorString(e));
}

#define FG_CUDA(call, what)                                  \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return cuda_error(e_, what);  \
    } while (0)

bool is_device_ptr(const void *p) {
    if (!p) return false;
    cudaPointerAttributes attr;
    cudaError_t e = cudaPointerGetAttributes(&attr, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

static bool cancelled(const volatile int32_t *cancel) { return cancel && *cancel != 0; }

// ------------------------------------------------------------------ a synchronous render's host side
// One 64-byte line of pinned, mapped host memory per synchronous render in flight, from one block kept for
// the life of the process.  Words 0 and 1 are the in-launch cancellation words (cancel_requested): the
// caller's cancel flag is ordinary host memory that the GPU cannot be assumed to reach, so it is mirrored
// into word 0.  The rest receives the diagnostic counters (a copy into pageable memory would block the
// host until the stream reached it).
class HostLines {
  public:
    static HostLines &get() {
        static HostLines s;
        return s;
    }
    int *acquire() {
        std::lock_guard<std::mutex> lock(mu_);
        if (!base_) {
            void *p = nullptr;
            if (cudaHostAlloc(&p, kLines * kLine, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;  // no in-launch polling; the flag is still read between launches
            }
            base_ = static_cast<int *>(p);
            for (int i = kLines - 1; i >= 0; i--) free_.push_back(i);
        }
        if (free_.empty()) return nullptr;
        int *w = base_ + free_.back() * (kLine / sizeof(int));
        free_.pop_back();
        ((volatile int *)w)[0] = 0;
        ((volatile int *)w)[1] = 0;
        return w;
    }
    void release(int *w) {
        std::lock_guard<std::mutex> lock(mu_);
        free_.push_back((int)((w - base_) / (kLine / sizeof(int))));
    }

  private:
    static constexpr int kLines = 256;
    static constexpr size_t kLine = 64;
    static_assert(2 * sizeof(int) + kPwDiagWords * sizeof(unsigned long long) <= kLine, "line too short");
    std::mutex mu_;
    int *base_ = nullptr;
    std::vector<int> free_;
};

// The calling thread waits for its render here, and mirrors the cancel flag while it waits.  (A watcher
// thread that slept 200 us between its looks cost every call its start and up to 200 us in its join: a
// 96 x 64 plane whose launches span 208 us took 432 us.)
class HostSide {
  public:
    HostSide(const volatile int32_t *cancel, cudaStream_t s)
        : cancel_(cancel), stream_(s), line_(HostLines::get().acquire()) {
        if (!cancel || !line_) return;
        void *d = nullptr;
        if (cudaHostGetDevicePointer(&d, line_, 0) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        dev_ = static_cast<int *>(d);
    }
    // An early return waits here once something may be queued: the kernels and the counters' copy write the line.
    // A refused request does not wait for what the caller has on the stream.
    ~HostSide() {
        if (queued_ && !waited_) cudaStreamSynchronize(stream_);
        if (line_) HostLines::get().release(line_);
    }
    HostSide(const HostSide &) = delete;
    HostSide &operator=(const HostSide &) = delete;
    int *cancel_words() const { return dev_; }
    void queued() { queued_ = true; }
    // where the counters' copy lands: pinned when there is a line
    unsigned long long *diag() {
        return line_ ? reinterpret_cast<unsigned long long *>(line_ + 2) : diag_;
    }
    // whether a CTA stopped on the flag
    bool stopped() const { return line_ && ((volatile int *)line_)[1] != 0; }
    // until the work queued so far has finished
    cudaError_t wait() {
        waited_ = true;
        if (!dev_) return cudaStreamSynchronize(stream_);
        for (;;) {
            const cudaError_t e = cudaStreamQuery(stream_);
            if (e != cudaErrorNotReady) return e;
            cudaGetLastError();
            if (*cancel_ != 0) {
                ((volatile int *)line_)[0] = 1;
                return cudaStreamSynchronize(stream_);
            }
            std::this_thread::yield();
        }
    }

  private:
    const volatile int32_t *cancel_;
    cudaStream_t stream_;
    int *line_;
    bool queued_ = false, waited_ = false;
    int *dev_ = nullptr;
    unsigned long long diag_[kPwDiagWords];
};

static fg_status cancelled_error(const HostSide &h) {
    return set_error(FG_ERR_CANCELLED, h.stopped() ? "cancelled (stopped inside a kernel)" : "cancelled");
}

void offset_extents(const float *offs, uint32_t n, float ext[4]) {
    ext[0] = ext[1] = ext[2] = ext[3] = 0.0f;
    for (uint32_t k = 0; k < n; k++) {
        ext[0] = std::fmin(ext[0], offs[2 * k]);
        ext[1] = std::fmax(ext[1], offs[2 * k]);
        ext[2] = std::fmin(ext[2], offs[2 * k + 1]);
        ext[3] = std::fmax(ext[3], offs[2 * k + 1]);
    }
}

fg_status check_render_args(const fg_params *p, const fg_derived *d) {
    if (!p || !d) return set_error(FG_ERR_INVALID, "null params or derived");
    if (d->input_width <= 0 || d->input_height <= 0 || d->output_width <= 0 || d->output_height <= 0)
        return set_error(FG_ERR_INVALID, "plane dimensions must be positive");
    if (d->input_width > (1 << 24) || d->input_height > (1 << 24) || d->output_width > (1 << 24) ||
        d->output_height > (1 << 24) || d->input_width * d->input_height >= (1ll << 31) ||
        d->output_width * d->output_height >= (1ll << 31))
        return set_error(FG_ERR_UNSUPPORTED, "plane larger than 2^31 pixels or 2^24 per side");
    if (p->n_samples == 0 || p->n_samples > 65536) return set_error(FG_ERR_UNSUPPORTED, "n_samples must be in 1..65536");
    if (!(p->zoom > 0.0f) || !(d->delta > 0.0f)) return set_error(FG_ERR_INVALID, "zoom and delta must be positive");
    if (p->radius_dist == FG_RADIUS_LOGNORM && !p->has_log_params)
        return set_error(FG_ERR_INVALID, "missing log-normal parameters");
    return FG_OK;
}

// Pixel-wise launch plan: the largest power-of-two block edge whose staged window fits.
PwPlan plan_pixelwise(const fg_params &p, const fg_derived &d, const float *h_offs_in, int max_block_log2) {
    PwPlan pl;
    offset_extents(h_offs_in, p.n_samples, pl.ext);
    const float rm = d.rm, delta = d.delta;
    int b;
    for (b = max_block_log2; b > -8; b--) {
        float B = std::ldexp(1.0f, b);
        double wc = std::floor((B + 2.0 * rm) / delta) + 4.0;
        if (wc <= kPwEdgeMax && wc * wc <= kPwCellMax) break;
    }
    pl.bsize = std::ldexp(1.0f, b);
    const float inv_zoom = 1.0f / p.zoom;
    float xmin = 0.5f * inv_zoom - pl.ext[1], ymin = 0.5f * inv_zoom - pl.ext[3];
    float xmax = ((float)(d.output_width - 1) + 0.5f) * inv_zoom - pl.ext[0];
    float ymax = ((float)(d.output_height - 1) + 0.5f) * inv_zoom - pl.ext[2];
    pl.bx0 = (int)std::floor(xmin / pl.bsize) - 1;
    pl.by0 = (int)std::floor(ymin / pl.bsize) - 1;
    pl.nbx = (int)std::floor(xmax / pl.bsize) + 1 - pl.bx0 + 1;
    pl.nby = (int)std::floor(ymax / pl.bsize) + 1 - pl.by0 + 1;
    return pl;
}

PixelwiseArgs pixelwise_args(const fg_params &p, const fg_derived &d, const PwPlan &pl, const float *d_lam,
                             const CellParam *d_cells, const float *d_offs_in, float *d_out, unsigned long long *d_diag) {
    PixelwiseArgs a;
    std::memset(&a, 0, sizeof a);
    a.lam = d_lam;
    a.cells = d_cells;
    a.offs = reinterpret_cast<const float2 *>(d_offs_in);
    a.out = d_out;
    a.diag = d_diag;
    a.in_w = (int)d.input_width; a.in_h = (int)d.input_height;
    a.out_w = (int)d.output_width; a.out_h = (int)d.output_height;
    a.n = (int)p.n_samples;
    a.rm = d.rm;
    a.delta = d.delta;
    {
        const double t = d.rm > 0.0f ? 2.0 * (double)d.rm / (double)d.delta + 1.0 : 0.0;
        a.regen_cells = (float)(t * t);
    }
    a.inv_zoom = 1.0f / p.zoom;
    a.zoom = p.zoom;
    a.bsize = pl.bsize;
    a.inv_bsize = 1.0f / pl.bsize;
    a.bx0 = pl.bx0; a.by0 = pl.by0; a.nbx = pl.nbx;
    a.offx_min = pl.ext[0]; a.offx_max = pl.ext[1]; a.offy_min = pl.ext[2]; a.offy_max = pl.ext[3];
    a.seed = p.seed;
    a.lognorm = p.radius_dist == FG_RADIUS_LOGNORM;
    a.radius_mean = p.radius_mean;
    a.log_mu = p.radius_log_mu;
    a.log_sigma = p.radius_log_sigma;
    return a;
}

// Stream-ordered device buffer that frees itself.
struct DevBuf {
    void *p = nullptr;
    cudaStream_t s = nullptr;
    cudaError_t alloc(size_t bytes, cudaStream_t st) {
        s = st;
        return cudaMallocAsync(&p, bytes ? bytes : 16, st);
    }
    ~DevBuf() {
        if (p) cudaFreeAsync(p, s);
    }
};

// The parts of a render's device memory, laid out one after the other in one allocation (each alloc and
// free is some microseconds of host time before the first launch): add() gives a part's byte offset.
struct Layout {
    size_t bytes = 0;
    size_t add(size_t n) {
        const size_t at = bytes;
        bytes = at + ((n + 255) & ~(size_t)255);
        return at;
    }
};

// A pixel-wise plane's scratch: the counters and the deferred list (its header beside them, so that both
// are cleared together), the offsets, the cell table and, last, the sparse pass's bitmask and the stream pass's bits
// (without the bits, the bitmask's part has room for the sparse pass's sorted offsets too).
struct PwScratch {
    PwPlan plan;
    size_t diag, offs, cells, mask, mask_bytes, bits, bits_bytes;
    PwScratch(const fg_params &p, const fg_derived &d, const float *h_offs_in, Layout *l) {
        plan = plan_pixelwise(p, d, h_offs_in, 4);
        const PixelwiseArgs a = pixelwise_args(p, d, plan, nullptr, nullptr, nullptr, nullptr, nullptr);
        diag = l->add(sizeof(PwCounters) + (size_t)plan.nbx * plan.nby * sizeof(int));
        offs = l->add(sizeof(float) * 2 * p.n_samples);
        cells = l->add(sizeof(CellParam) * (size_t)d.input_width * d.input_height);
        mask_bytes = pixelwise_cellmask_bytes(a, plan.nby);
        mask = l->add(mask_bytes);
        bits_bytes = mask_bytes ? pixelwise_stream_bytes(a, plan.nby) : 0;
        bits = l->add(bits_bytes);
    }
    // the layout's allocation: without the bits where that finds no room (the plane takes the sparse pass), and then
    // without the bitmask (the lean pass)
    cudaError_t alloc(DevBuf *b, const Layout &l, cudaStream_t s) {
        cudaError_t e = b->alloc(l.bytes, s);
        if (e == cudaErrorMemoryAllocation && bits_bytes) {
            cudaGetLastError();
            bits_bytes = 0;
            e = b->alloc(bits, s);
        }
        if (e == cudaErrorMemoryAllocation && mask_bytes) {
            cudaGetLastError();
            mask_bytes = 0;
            e = b->alloc(mask, s);
        }
        return e;
    }
    PwBuffers at(void *base) const {
        char *c = static_cast<char *>(base);
        PwBuffers w;
        w.counters = reinterpret_cast<PwCounters *>(c + diag);
        w.offs = reinterpret_cast<float *>(c + offs);
        w.cells = reinterpret_cast<CellParam *>(c + cells);
        w.listed = true;
        w.mask = mask_bytes ? reinterpret_cast<unsigned int *>(c + mask) : nullptr;
        w.bits = bits_bytes ? reinterpret_cast<unsigned int *>(c + bits) : nullptr;
        w.bits_bytes = bits_bytes;
        return w;
    }
};

fg_status enqueue_pixelwise(const float *d_lam, const fg_params &p, const fg_derived &d, const PwPlan &pl,
                            const PwBuffers &w, float *d_out, const EpilogueArgs *colour, cudaStream_t s,
                            int *d_cancel) {
    const int in_w = (int)d.input_width, in_h = (int)d.input_height;
    const int out_w = (int)d.output_width, out_h = (int)d.output_height;
    const long long n_in = (long long)in_w * in_h, n_out = (long long)out_w * out_h;
    // An output that shares memory with lambda (a render in place) is cleared only once the cell table is made.
    const bool in_place = !w.bits && d_out < d_lam + n_in && d_lam < d_out + n_out;
    FG_CUDA(launch_cell_params(d_lam, in_w, in_h, d.delta, w.cells,
                               w.bits ? w.bits : reinterpret_cast<unsigned int *>(d_out),
                               w.bits ? (long long)(w.bits_bytes / sizeof(int)) : (in_place ? 0 : n_out), w.counters, s),
            "cell params");
    if (in_place) FG_CUDA(cudaMemsetAsync(d_out, 0, sizeof(float) * n_out, s), "clear output");
    PixelwiseArgs a = pixelwise_args(p, d, pl, d_lam, w.cells, w.offs, d_out, w.counters->diag);
    a.cancel = d_cancel;
    FG_CUDA(launch_pixelwise(a, pl.nby, w.listed ? w.counters : nullptr, w.mask, w.bits, s), "pixelwise kernel");
    EpilogueArgs e;
    if (colour) e = *colour;
    else std::memset(&e, 0, sizeof e);
    e.plane = d_out;
    e.bits = w.bits;
    e.words = (int)((p.n_samples + 31) / 32);
    e.out_w = out_w; e.out_h = out_h; e.in_w = in_w; e.in_h = in_h;
    e.inv_samples = 1.0f / (float)p.n_samples;
    FG_CUDA(launch_epilogue(e, s), "pixelwise epilogue");
    return FG_OK;
}

// Shared-memory sample-mask words per grain-wise tile (sets the tile edge).  Measured on GB300 with
// N = 128 at zoom 2 (1024^2 plane): 6144 words 29.6 ms, 8192 26.3 ms, 12288 28.7 ms, 16384 31.7 ms.
constexpr int kGrainMaskWords = 8192;
constexpr int kGrainChunkWords = 8;  // mask words of a chunk at most (kGbMaxWords, fg_grainwise.cuh)

GrainwiseArgs grainwise_args(const fg_params &p, const fg_derived &d, const float *h_offs, const float *d_lam,
                             const float *d_offs, unsigned int *d_gmask, int mask_words) {
    GrainwiseArgs a;
    std::memset(&a, 0, sizeof a);
    float ext[4];
    offset_extents(h_offs, p.n_samples, ext);
    a.lam = d_lam;
    a.offs = reinterpret_cast<const float2 *>(d_offs);
    a.gmask = d_gmask;
    a.in_w = (int)d.input_width; a.in_h = (int)d.input_height;
    a.out_w = (int)d.output_width; a.out_h = (int)d.output_height;
    a.n = (int)p.n_samples;
    a.words = (a.n + 31) / 32;
    // chunks of equal width, so that no item is much lighter than the others of its tile
    a.chunks = (a.words + kGrainChunkWords - 1) / kGrainChunkWords;
    a.chunk_words = (a.words + a.chunks - 1) / a.chunks;
    a.chunks = (a.words + a.chunk_words - 1) / a.chunk_words;
    // Input tile: its zoomed rectangle should fill about `mask_words` words of shared memory.
    // floor(x0*zoom + tin*zoom) - floor(x0*zoom) <= ceil(tin*zoom), so that bounds the rectangle.
    auto fit_tile = [&](int words) {
        const int side = std::max(1, (int)std::floor(std::sqrt((double)mask_words / words)));
        const int tin = std::max(1, (int)std::floor(side / p.zoom));
        a.tin_w = std::min(tin, a.in_w);
        a.tin_h = std::min(tin, a.in_h);
        a.rmax_w = std::max(1, std::min(a.out_w, (int)std::ceil(a.tin_w * (double)p.zoom)));
        a.rmax_h = std::max(1, std::min(a.out_h, (int)std::ceil(a.tin_h * (double)p.zoom)));
    };
    // What limits a request: 200 KB for a tile's masks with all samples (the rectangle such a tile would
    // have) beside fixed sizes per offset and filter word, whatever the kernel's own layout and chunks need
    // (grainwise_smem_bytes: at most 12 KB more than this with one chunk, less with several).
    fit_tile(a.words);
    const size_t n = p.n_samples, rect = (size_t)a.rmax_w * a.rmax_h * a.words * sizeof(unsigned int);
    a.request_bytes = rect + (a.chunks > 1 ? n * 20 + 44108
                                           : ((n + 1) & ~(size_t)1) * 8 + 7168 * (size_t)(a.words | 1) +
                                                 ((n + 7) & ~(size_t)7) * 2 + 16);
    fit_tile(a.chunk_words);
    a.rm = d.rm;
    a.zoom = p.zoom;
    // A grain's draws and filter cost about 400 lane-ops, a pair 100, and a grain has
    // n (2 (r zoom + 1/128))^2 of them on average.
    {
        const double n_chunk = std::min<double>(p.n_samples, 32.0 * a.chunk_words);
        const double r2 = (double)p.radius_mean * p.radius_mean + (double)p.radius_stddev * p.radius_stddev;
        const double band = std::min(1.0, 2.0 * (std::sqrt(r2) * p.zoom + 1.0 / 128.0));
        a.grain_cost = (float)(400.0 + 100.0 * n_chunk * band * band);
    }
    a.offx_min = ext[0]; a.offx_max = ext[1]; a.offy_min = ext[2]; a.offy_max = ext[3];
    // Rounding margin of the candidate intervals: each of the three f32 roundings between
    // czx + offx and the bounds() comparison moves a value by at most half an ulp of the largest
    // coordinate M; the fraction arithmetic adds a few 2^-24.
    const double M = (double)std::max(d.output_width, d.output_height) + 8.0 +
                     std::max(std::max(-ext[0], ext[1]), std::max(-ext[2], ext[3])) + d.rm * p.zoom;
    const double U = std::ldexp(1.0, (int)std::floor(std::log2(M)) - 23);
    a.frac_eps = (float)(4.0 * U + std::ldexp(1.0, -20));
    a.seed = p.seed;
    a.lognorm = p.radius_dist == FG_RADIUS_LOGNORM;
    a.radius_mean = p.radius_mean;
    a.log_mu = p.radius_log_mu;
    a.log_sigma = p.radius_log_sigma;
    return a;
}

// A grain-wise plane's scheduler area and a device's SM count for it.
static fg_status grainwise_work_bytes(const GrainwiseArgs &a, size_t *bytes, int *sms) {
    int dev = 0;
    FG_CUDA(cudaGetDevice(&dev), "device");
    FG_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    *bytes = grainwise_work_ints(a, *sms) * sizeof(int);
    return FG_OK;
}

static fg_status check_grainwise(const GrainwiseArgs &a) {
    if (a.request_bytes > 200 * 1024)
        return set_error(FG_ERR_UNSUPPORTED, "n_samples too large for the grain-wise tile");
    return FG_OK;
}

size_t grainwise_mask_bytes(const fg_params &p, const fg_derived &d) {
    return (size_t)d.output_width * d.output_height * ((p.n_samples + 31) / 32) * sizeof(unsigned int);
}

// a.work: the scheduler's area (grainwise_work_bytes)
static fg_status enqueue_grainwise(const GrainwiseArgs &a, int sms, cudaStream_t s) {
    FG_CUDA(cudaMemsetAsync(a.gmask, 0, (size_t)a.out_w * a.out_h * a.words * sizeof(unsigned int), s), "memset mask");
    FG_CUDA(launch_grainwise(a, sms, s), "grainwise kernel");
    return FG_OK;
}

fg_status enqueue_grainwise_epilogue(const GrainwiseArgs &a, float *d_out, int mode, unsigned char *d_rgb8,
                                     const float *d_cb, const float *d_cr, cudaStream_t s) {
    GrainwiseEpilogueArgs e;
    std::memset(&e, 0, sizeof e);
    e.gmask = a.gmask;
    e.out = d_out;
    e.out_rgb8 = d_rgb8;
    e.cb = d_cb;
    e.cr = d_cr;
    e.out_w = a.out_w; e.out_h = a.out_h; e.in_w = a.in_w; e.in_h = a.in_h;
    e.n = a.n;
    e.words = a.words;
    e.mode = mode;
    FG_CUDA(launch_grainwise_epilogue(e, s), "grainwise epilogue");
    return FG_OK;
}

// The stream-ordered pool of the current device keeps its memory between renders (raised release
// threshold), set once per device; safe to call from several threads.
static void keep_pool_memory() {
    static std::atomic<bool> done[128];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) {
        cudaGetLastError();
        return;
    }
    if (done[dev].load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev].load(std::memory_order_relaxed)) return;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t thr = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    cudaGetLastError();
    done[dev].store(true, std::memory_order_release);
}

// Shared body of the synchronous integrator entry points.
static fg_status render_plane_sync(int algo, const float *lambda, const fg_params *params, const fg_derived *derived,
                                   const float *offsets, float *out, const volatile int32_t *cancel, void *stream) {
    fg_status st = check_render_args(params, derived);
    if (st != FG_OK) return st;
    if (!lambda || !offsets || !out) return set_error(FG_ERR_INVALID, "null buffer");
    if (cancelled(cancel)) return set_error(FG_ERR_CANCELLED, "cancelled");
    keep_pool_memory();
    cudaStream_t s = (cudaStream_t)stream;
    const fg_params &p = *params;
    const fg_derived &d = *derived;
    HostSide host(cancel, s);
    const size_t n_in = (size_t)d.input_width * d.input_height, n_out = (size_t)d.output_width * d.output_height;
    const size_t off_bytes = sizeof(float) * 2 * p.n_samples;

    const bool offs_dev = is_device_ptr(offsets), lam_dev = is_device_ptr(lambda), out_dev = is_device_ptr(out);
    std::vector<float> h_copy;
    const float *h_offs = offsets;
    if (offs_dev) {
        h_copy.resize(2 * (size_t)p.n_samples);
        FG_CUDA(cudaMemcpy(h_copy.data(), offsets, off_bytes, cudaMemcpyDeviceToHost), "offsets D2H");
        h_offs = h_copy.data();
    }
    DevBuf b;
    Layout l;
    const size_t at_lam = lam_dev ? 0 : l.add(sizeof(float) * n_in), at_out = out_dev ? 0 : l.add(sizeof(float) * n_out);
    auto planes = [&](const float **d_lam, float **d_out) -> fg_status {
        *d_lam = lambda;
        *d_out = out;
        if (!lam_dev) {
            float *dst = reinterpret_cast<float *>(static_cast<char *>(b.p) + at_lam);
            FG_CUDA(cudaMemcpyAsync(dst, lambda, sizeof(float) * n_in, cudaMemcpyHostToDevice, s), "lambda H2D");
            *d_lam = dst;
        }
        if (!out_dev) *d_out = reinterpret_cast<float *>(static_cast<char *>(b.p) + at_out);
        return FG_OK;
    };
    const float *d_lam;
    float *d_out;
    if (algo == FG_ALGO_PIXEL) {
        PwScratch scratch(p, d, h_offs, &l);
        FG_CUDA(scratch.alloc(&b, l, s), "alloc render");
        host.queued();
        const PwBuffers w = scratch.at(b.p);
        FG_CUDA(cudaMemcpyAsync(w.offs, h_offs, off_bytes, cudaMemcpyHostToDevice, s), "offsets H2D");
        if ((st = planes(&d_lam, &d_out)) != FG_OK) return st;
        st = enqueue_pixelwise(d_lam, p, d, scratch.plan, w, d_out, nullptr, s, host.cancel_words());
        if (st != FG_OK) return st;
        FG_CUDA(cudaMemcpyAsync(host.diag(), w.counters->diag, sizeof g_pw_diag, cudaMemcpyDeviceToHost, s), "diag D2H");
    } else {
        GrainwiseArgs a = grainwise_args(p, d, h_offs, nullptr, nullptr, nullptr, kGrainMaskWords);
        size_t work_bytes;
        int sms;
        if ((st = check_grainwise(a)) != FG_OK) return st;
        if ((st = grainwise_work_bytes(a, &work_bytes, &sms)) != FG_OK) return st;
        const size_t at_offs = l.add(off_bytes), at_work = l.add(work_bytes), at_mask = l.add(grainwise_mask_bytes(p, d));
        FG_CUDA(b.alloc(l.bytes, s), "alloc render");
        host.queued();
        char *base = static_cast<char *>(b.p);
        FG_CUDA(cudaMemcpyAsync(base + at_offs, h_offs, off_bytes, cudaMemcpyHostToDevice, s), "offsets H2D");
        if ((st = planes(&d_lam, &d_out)) != FG_OK) return st;
        a.lam = d_lam;
        a.offs = reinterpret_cast<const float2 *>(base + at_offs);
        a.work = reinterpret_cast<int *>(base + at_work);
        a.gmask = reinterpret_cast<unsigned int *>(base + at_mask);
        a.cancel = host.cancel_words();
        st = enqueue_grainwise(a, sms, s);
        if (st == FG_OK) st = enqueue_grainwise_epilogue(a, d_out, 0, nullptr, nullptr, nullptr, s);
        if (st != FG_OK) return st;
    }
    FG_CUDA(host.wait(), "render");
    if (!out_dev) {
        FG_CUDA(cudaMemcpyAsync(out, d_out, sizeof(float) * n_out, cudaMemcpyDeviceToHost, s), "out D2H");
        FG_CUDA(cudaStreamSynchronize(s), "render");
    }
    if (algo == FG_ALGO_PIXEL) std::memcpy(g_pw_diag, host.diag(), sizeof g_pw_diag);
    if (cancelled(cancel)) return cancelled_error(host);
    clear_error();
    return FG_OK;
}

}  // namespace fg

using namespace fg;

extern "C" {

FG_API fg_status fg_render_pixelwise(const float *lambda, const fg_params *params, const fg_derived *derived,
                                     const float *offsets_input, float *out, const volatile int32_t *cancel,
                                     void *stream) {
    return render_plane_sync(FG_ALGO_PIXEL, lambda, params, derived, offsets_input, out, cancel, stream);
}

FG_API fg_status fg_render_grainwise(const float *lambda, const fg_params *params, const fg_derived *derived,
                                     const float *offsets, float *out, const volatile int32_t *cancel, void *stream) {
    return render_plane_sync(FG_ALGO_GRAIN, lambda, params, derived, offsets, out, cancel, stream);
}

FG_API fg_status fg_render_pixelwise_async(const float *d_lambda, const fg_params *params, const fg_derived *derived,
                                           const float *offsets_input, float *d_out, void *stream) {
    fg_status st = check_render_args(params, derived);
    if (st != FG_OK) return st;
    if (!d_lambda || !offsets_input || !d_out) return set_error(FG_ERR_INVALID, "null buffer");
    if (is_device_ptr(offsets_input)) return set_error(FG_ERR_INVALID, "offsets_input must be host memory");
    keep_pool_memory();
    cudaStream_t s = (cudaStream_t)stream;
    DevBuf b;
    Layout l;
    PwScratch scratch(*params, *derived, offsets_input, &l);
    FG_CUDA(scratch.alloc(&b, l, s), "alloc render");
    const PwBuffers w = scratch.at(b.p);
    FG_CUDA(cudaMemcpyAsync(w.offs, offsets_input, sizeof(float) * 2 * params->n_samples, cudaMemcpyHostToDevice, s),
            "offsets H2D");
    return enqueue_pixelwise(d_lambda, *params, *derived, scratch.plan, w, d_out, nullptr, s, nullptr);
}

FG_API fg_status fg_render_grainwise_async(const float *d_lambda, const fg_params *params, const fg_derived *derived,
                                           const float *offsets, float *d_out, void *stream) {
    fg_status st = check_render_args(params, derived);
    if (st != FG_OK) return st;
    if (!d_lambda || !offsets || !d_out) return set_error(FG_ERR_INVALID, "null buffer");
    if (is_device_ptr(offsets)) return set_error(FG_ERR_INVALID, "offsets must be host memory");
    keep_pool_memory();
    cudaStream_t s = (cudaStream_t)stream;
    const size_t off_bytes = sizeof(float) * 2 * params->n_samples;
    GrainwiseArgs a = grainwise_args(*params, *derived, offsets, d_lambda, nullptr, nullptr, kGrainMaskWords);
    size_t work_bytes;
    int sms;
    if ((st = check_grainwise(a)) != FG_OK) return st;
    if ((st = grainwise_work_bytes(a, &work_bytes, &sms)) != FG_OK) return st;
    DevBuf b;
    Layout l;
    const size_t at_offs = l.add(off_bytes), at_work = l.add(work_bytes),
                 at_mask = l.add(grainwise_mask_bytes(*params, *derived));
    FG_CUDA(b.alloc(l.bytes, s), "alloc render");
    char *base = static_cast<char *>(b.p);
    FG_CUDA(cudaMemcpyAsync(base + at_offs, offsets, off_bytes, cudaMemcpyHostToDevice, s), "offsets H2D");
    a.offs = reinterpret_cast<const float2 *>(base + at_offs);
    a.work = reinterpret_cast<int *>(base + at_work);
    a.gmask = reinterpret_cast<unsigned int *>(base + at_mask);
    st = enqueue_grainwise(a, sms, s);
    if (st == FG_OK) st = enqueue_grainwise_epilogue(a, d_out, 0, nullptr, nullptr, nullptr, s);
    return st;
}

FG_API fg_status fg_render_image(const float *rgb, int64_t width, int64_t height, const fg_params *params,
                                 uint8_t *out_rgb8, fg_render_stats *stats, const volatile int32_t *cancel,
                                 void *stream) {
    if (!rgb || !params || !out_rgb8) return set_error(FG_ERR_INVALID, "null pointer");
    if (width <= 0 || height <= 0) return set_error(FG_ERR_INVALID, "input image is empty");
    if (cancelled(cancel)) return set_error(FG_ERR_CANCELLED, "cancelled");
    const fg_params &p = *params;
    int64_t x0 = 0, y0 = 0, cw = width, ch = height;
    if (p.has_roi) {
        if ((int64_t)p.roi_x1 > width || (int64_t)p.roi_y1 > height)
            return set_error(FG_ERR_INVALID, "ROI exceeds image bounds");
        x0 = p.roi_x0; y0 = p.roi_y0;
        cw = (int64_t)p.roi_x1 - p.roi_x0; ch = (int64_t)p.roi_y1 - p.roi_y0;
        if (cw <= 0 || ch <= 0) return set_error(FG_ERR_INVALID, "ROI width and height must be positive");
    }
    fg_derived d;
    std::vector<float> offs(2 * (size_t)p.n_samples), offs_in(2 * (size_t)p.n_samples);
    fg_status st = derive(p, cw, ch, &d, offs.data(), offs_in.data());
    if (st != FG_OK) return st;
    st = check_render_args(params, &d);
    if (st != FG_OK) return st;
    const int32_t algo = choose_algorithm(p, d);
    const bool luma = p.color_mode == FG_COLOR_LUMA;
    const int nplanes = luma ? 1 : 3;
    const size_t n_in = (size_t)cw * ch, n_out = (size_t)d.output_width * d.output_height;

    keep_pool_memory();
    cudaStream_t s = (cudaStream_t)stream;
    HostSide host(cancel, s);
    // the cropped interleaved RGB to the device, then the colour split, the plane maxima and lambda
    // there (fg_lambda.cu): no host pass over the image
    DevBuf b;
    Layout l;
    const size_t at_rgb = l.add(sizeof(float) * 3 * n_in), at_planes = l.add(sizeof(float) * 3 * n_in),
                 at_max = l.add(sizeof(unsigned int) * 3), at_lam = l.add(sizeof(float) * n_in * nplanes),
                 at_out = l.add(sizeof(float) * n_out * nplanes), at_rgb8 = l.add(3 * n_out);
    const std::vector<float> &used_offs = algo == FG_ALGO_PIXEL ? offs_in : offs;
    const size_t off_bytes = sizeof(float) * 2 * p.n_samples;
    const size_t mask_bytes = algo == FG_ALGO_GRAIN ? grainwise_mask_bytes(p, d) : 0;
    std::unique_ptr<PwScratch> pw;  // one plane after the other in the same scratch
    GrainwiseArgs ga;
    std::memset(&ga, 0, sizeof ga);
    size_t at_offs = 0, at_work = 0, at_mask = 0;
    int sms = 0;
    if (algo == FG_ALGO_PIXEL) {
        pw.reset(new PwScratch(p, d, offs_in.data(), &l));
        at_offs = pw->offs;
        FG_CUDA(pw->alloc(&b, l, s), "alloc render");
    } else {
        ga = grainwise_args(p, d, offs.data(), nullptr, nullptr, nullptr, kGrainMaskWords);
        size_t work_bytes;
        if ((st = check_grainwise(ga)) != FG_OK) return st;
        if ((st = grainwise_work_bytes(ga, &work_bytes, &sms)) != FG_OK) return st;
        at_offs = l.add(off_bytes);
        at_work = l.add(work_bytes);
        at_mask = l.add(mask_bytes * nplanes);
        FG_CUDA(b.alloc(l.bytes, s), "alloc render");
    }
    host.queued();
    char *base = static_cast<char *>(b.p);
    float *d_rgb = reinterpret_cast<float *>(base + at_rgb), *d_planes = reinterpret_cast<float *>(base + at_planes);
    float *d_lam = reinterpret_cast<float *>(base + at_lam), *d_out = reinterpret_cast<float *>(base + at_out);
    unsigned char *d_rgb8 = reinterpret_cast<unsigned char *>(base + at_rgb8);
    FG_CUDA(cudaMemcpyAsync(base + at_offs, used_offs.data(), off_bytes, cudaMemcpyHostToDevice, s), "offsets H2D");
    FG_CUDA(cudaMemcpy2DAsync(d_rgb, sizeof(float) * 3 * (size_t)cw, rgb + 3 * ((size_t)y0 * width + x0),
                              sizeof(float) * 3 * (size_t)width, sizeof(float) * 3 * (size_t)cw, (size_t)ch,
                              cudaMemcpyHostToDevice, s),
            "rgb H2D");
    st = enqueue_split_lambda(d_rgb, (long long)n_in, luma ? 1 : 0, d_planes,
                              reinterpret_cast<unsigned int *>(base + at_max), d.inv_e_pi_r2, d_lam, s);
    if (st != FG_OK) return st;
    float *d_cb = luma ? d_planes + n_in : nullptr, *d_cr = luma ? d_cb + n_in : nullptr;
    for (int c = 0; c < nplanes; c++) {
        if (cancelled(cancel)) {
            host.wait();
            return cancelled_error(host);
        }
        float *d_plane = d_out + (size_t)c * n_out;
        if (algo == FG_ALGO_PIXEL) {
            EpilogueArgs e;
            std::memset(&e, 0, sizeof e);
            if (luma) {
                e.mode = 1; e.out_rgb8 = d_rgb8; e.cb = d_cb; e.cr = d_cr;
            } else if (c == 2) {
                e.mode = 2; e.out_rgb8 = d_rgb8; e.p0 = d_out; e.p1 = d_out + n_out;
            }
            st = enqueue_pixelwise(d_lam + (size_t)c * n_in, p, d, pw->plan, pw->at(base), d_plane, &e, s,
                                   host.cancel_words());
        } else {
            GrainwiseArgs a = ga;
            a.lam = d_lam + (size_t)c * n_in;
            a.offs = reinterpret_cast<const float2 *>(base + at_offs);
            a.work = reinterpret_cast<int *>(base + at_work);
            a.gmask = reinterpret_cast<unsigned int *>(base + at_mask + mask_bytes * c);
            a.cancel = host.cancel_words();
            st = enqueue_grainwise(a, sms, s);
            if (st == FG_OK && c == nplanes - 1) {
                a.gmask = reinterpret_cast<unsigned int *>(base + at_mask);  // all planes' masks, consecutive
                st = enqueue_grainwise_epilogue(a, nullptr, luma ? 1 : 2, d_rgb8, d_cb, d_cr, s);
            }
        }
        if (st != FG_OK) return st;
    }
    FG_CUDA(host.wait(), "render");
    FG_CUDA(cudaMemcpyAsync(out_rgb8, d_rgb8, 3 * n_out, cudaMemcpyDeviceToHost, s), "rgb8 D2H");
    FG_CUDA(cudaStreamSynchronize(s), "render");
    if (cancelled(cancel)) return cancelled_error(host);
    if (stats) fill_stats(p, d, algo, stats);
    clear_error();
    return FG_OK;
}

// Counters of the calling thread's last synchronous pixel-wise render: samples evaluated on the
// per-sample regeneration path, blocks without a staged window, block subdivisions, blocks run.
FG_API void fg_pixelwise_diagnostics(unsigned long long out[4]) {
    for (int i = 0; i < 4; i++) out[i] = g_pw_diag[i];
}

// That render's blocks of the sparse pass, and tiles (or parts of chunks) of the stream pass.
FG_API void fg_pixelwise_sparse_forms(unsigned long long out[2]) {
    out[0] = g_pw_diag[4];
    out[1] = g_pw_diag[5];
}

FG_API fg_status fg_pixelwise_kernel_count(const fg_params *params, const fg_derived *derived,
                                           const float *offsets_input, int32_t *out) {
    if (!params || !derived || !offsets_input || !out) return set_error(FG_ERR_INVALID, "null argument");
    fg_status st = check_render_args(params, derived);
    if (st != FG_OK) return st;
    const PwPlan pl = plan_pixelwise(*params, *derived, offsets_input, 4);
    const PixelwiseArgs a = pixelwise_args(*params, *derived, pl, nullptr, nullptr, nullptr, nullptr, nullptr);
    *out = pixelwise_takes_regen(a) ? 3 : (pixelwise_cellmask_bytes(a, pl.nby) ? 6 : 4);
    clear_error();
    return FG_OK;
}

}  // extern "C"
