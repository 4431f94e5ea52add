// fg_kernels.cuh -- launch descriptors shared by the kernels and the C-ABI layer.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace fg {

// Per input pixel: the Poisson set-up of a pixel-wise cell whose lambda lookup lands on the pixel
// (src/pixelwise.rs:69-82).  `thresh` turns the first Knuth comparison into an integer test on the
// first draw's 53-bit value v: U1 = v * 2^-53 > exp_lambda  <=>  v > floor(exp_lambda * 2^53), so
// v <= thresh means q = 0.  thresh = INT64_MAX means "no grains" (lambda <= 0 or
// lambda*delta*delta <= 0, the cell is skipped without drawing); thresh = -1 marks the rejection
// regime (lambda*delta^2 >= 12), where exp_lambda holds -expected.
struct __align__(16) CellParam {
    long long thresh;
    double exp_lambda;
};

// Shared-memory capacities of the pixel-wise tile kernel.
constexpr int kPwCellMax = 8192;   // staged window cells
// Shared-memory configurations of the pixel-wise block: lean CTAs (256 threads, 4 per SM) take every
// block first and defer the dense ones; fat CTAs (512 threads, 2 per SM) take the deferred blocks
// (and every block of the batched and allocation-free paths).
struct PwLean {
    static constexpr int kThreads = 256, kCtasPerSm = 4, kGrainMax = 1024, kListMax = 2048;
    static constexpr bool kDefers = true;
};
struct PwFat {
    static constexpr int kThreads = 512, kCtasPerSm = 2, kGrainMax = 4096, kListMax = 8192;
    static constexpr bool kDefers = false;
};
constexpr int kPwEdgeMax = 128;    // window cells per axis
constexpr int kPwKChunk = 256;     // offsets per sample-assignment chunk
constexpr int kPwFootMax = 1024;   // per-block output-pixel counters
constexpr int kPwMaxLevel = 3;     // block subdivision depth on grain overflow
// Pixel-wise diagnostic counters (PixelwiseArgs::diag): [0] samples evaluated on the per-sample path,
// [1] blocks without a staged window, [2] block subdivisions, [3] blocks and tiles run, [4] blocks of the sparse
// pass, [5] tiles of the stream pass.
constexpr int kPwDiagWords = 6;

// A pixel-wise plane's counters, and the header of its deferred list: [0] the next entry the fat pass
// takes, [1] the number of entries, which follow in list[2..] where a list is kept.
struct PwCounters {
    unsigned long long diag[kPwDiagWords];
    int tile, unused;  // the next tile of the stream pass
    int list[2];
};
// A block regenerates per sample (no staging) when its samples' reach, in cells, is below
// kPwRegenSparse x its window's cells, or below kPwRegenOverflow x them once the window overflows
// with more than kPwRegenDense of its cells non-empty.
constexpr float kPwRegenSparse = 1.0f;
constexpr float kPwRegenOverflow = 4.0f;
constexpr float kPwRegenDense = 0.4f;
// The per-sample kernel replaces the block kernel for a whole plane when an interior root block's
// samples reach fewer than kPwRegenKernel x its window's cells (and a sample's range fits 64 cells): 700 x 500
// ramps cross at 2.1 to 2.7 (radius 0.05: N 100 at 2.1 runs 2.92 ms against the block passes' 3.40, N 128 at
// 2.7 3.66 against 3.63; radius 0.07: N 64 at 2.6 1.92 against 1.96), blobs at 2.1 (2.29 against 2.27).
constexpr int kPwRegenThreads = 256;
constexpr float kPwRegenKernel = 2.05f;
// Small planes on their own (pixelwise_takes_regen): below kPwRegenSmallVisits cell visits and kPwRegenSmall
// windows.  Ramps of radius 0.1 and 0.2 on the per-sample kernel against the block passes, us of a whole call:
// 96 x 64 N 32 (1.8 million visits) 116 / 257, N 64 119 / 301, 160 x 120 N 64 (11 million) 183 / 385, 256 x 256
// N 64 (38 million) 458 / 550.  The line lies well below where the two meet, so that the small planes on which
// the tests hold the block passes against the oracle stay with them.  kPwRegenWarps: the warps per SM below
// which the kernel splits the samples (96 x 64 N 32 without the split: 226 us).
constexpr double kPwRegenSmallVisits = 4.5e6;
constexpr float kPwRegenSmall = 5.0f;
constexpr double kPwRegenWarps = 64.0;
// The stream pass (fg_pixelwise_stream.cuh): planes of kPwStreamPixels output pixels and more, and the grains per
// output pixel, in multiples of N, above which a segment's samples go to the per-sample kernel -- with ranges of
// up to 4 cells an axis, and wider ones, whose samples look at more cells.  Log-normal 0.025 / 0.01, N 256:
// 1024^2 blobs at 2.2 N 13.4 ms, 3 N 12.3, 4 N 13.1, a 1000^2 ramp 29.3, 24.1, 22.0; radius 0.1 N 32: 1080p at
// 1.3 N 2.19 ms, 2 N 2.10, 3 N 2.02, a 1000^2 ramp 1.68, 1.58, 1.70.
constexpr double kPwStreamPixels = 8192.0;
constexpr float kPwStreamDense = 2.0f, kPwStreamDenseWide = 4.0f;

// In-launch cancellation: `cancel` is null or two words of mapped pinned host memory.  Word 0 is set
// by the waiting host thread once the caller's cancel flag turns non-zero; the persistent passes
// read it once per work item they pull (the block passes once per block, the per-sample kernel once per CTA)
// and stop, and a CTA that stops on it sets word 1.  Reads of host memory go one after the other, about 7 ns
// each, so warps whose items are short look at it by the clock (CancelPoll).
#ifdef __CUDACC__
__device__ __forceinline__ bool cancel_requested(int *cancel) {
    if (!cancel || *(volatile int *)cancel == 0) return false;
    *(volatile int *)(cancel + 1) = 1;
    return true;
}
// A warp's look at the flag every 200 us.  512 x 512, radius 0.1, N 32, with a flag, looking once per item of
// the stream and dense passes: 1.92 ms a call against 0.40 without a flag.
struct CancelPoll {
    static constexpr long long kCycles = 400000;
    long long last;
    __device__ __forceinline__ void begin() { last = clock64(); }
    __device__ __forceinline__ bool requested(int *cancel) {
        if (!cancel || clock64() - last < kCycles) return false;
        last = clock64();
        return cancel_requested(cancel);
    }
};
#endif

struct PixelwiseArgs {
    const float *lam;           // in_w x in_h
    const CellParam *cells;     // in_w x in_h
    const float2 *offs;         // offsets_input [n]
    float *out;                 // out_w x out_h, accumulates hit counts (pre-zeroed)
    unsigned long long *diag;   // [kPwDiagWords] counters
    int in_w, in_h, out_w, out_h;
    int n;
    float rm, delta, inv_zoom, zoom;
    float regen_cells;          // mean cells one sample's own loop visits: (2 rm / delta + 1)^2
    float bsize, inv_bsize;     // block edge in input pixels (power of two) and its inverse
    int bx0, by0, nbx;          // block-grid origin and width
    float offx_min, offx_max, offy_min, offy_max;
    unsigned long long seed;
    int lognorm;
    float radius_mean;
    float log_mu, log_sigma;
    int *cancel;                // null, or the in-launch cancellation words (cancel_requested)
    // null, or the plane's emptiness bitmask (the sparse pass's first_draw_maybe of every cell):
    // cells [cm_gi0, cm_gi0 + cm_gw) x [cm_gj0, cm_gj0 + 32 cm_ghw), word (c, k) = cellmask[k * cm_gw + c]
    // holding rows cm_gj0 + 32k .. + 31 of column cm_gi0 + c
    const unsigned int *cellmask;
    int cm_gi0, cm_gj0, cm_gw, cm_ghw;
};

// Whether the per-sample kernel screens this plane's samples in two steps: ranges of more than 4 cells an axis.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool pixelwise_two_step(const PixelwiseArgs &a) {
    return floor(2.0 * (double)a.rm / (double)a.delta) + 2.0 > 4.0;
}

struct GrainwiseArgs {
    const float *lam;           // in_w x in_h
    const float2 *offs;         // offsets [n]
    unsigned int *gmask;        // out_w x out_h x words sample masks (zeroed before the launch)
    int in_w, in_h, out_w, out_h;
    int n, words;               // words = ceil(n/32)
    int chunk_words, chunks;    // a work item takes the samples of one chunk of chunk_words mask words
    int tin_w, tin_h;           // input tile of one CTA
    int rmax_w, rmax_h;         // bound of the zoomed tile rectangle held in shared memory
    float rm, zoom;
    float offx_min, offx_max, offy_min, offy_max;
    float frac_eps;             // rounding margin of the candidate-offset intervals
    unsigned long long seed;
    int lognorm;
    float radius_mean;
    float log_mu, log_sigma;
    int *work;                  // the tile scheduler's area (grainwise_work_ints)
    float grain_cost;           // lane-ops of a grain in one chunk (the tile scheduler's cost model)
    size_t request_bytes;       // size of the request, for its limit (grainwise_request_bytes)
    int *cancel;                // null, or the in-launch cancellation words (cancel_requested)
};

// popcount / colour epilogue of the grain-wise path.
struct GrainwiseEpilogueArgs {
    const unsigned int *gmask;  // planes x out_w x out_h x words
    float *out;                 // planes x out_w x out_h values (may be null)
    unsigned char *out_rgb8;    // null, or u8 RGB (mode 1 / 2)
    const float *cb, *cr;       // luma: chroma planes at input size
    int out_w, out_h, in_w, in_h;
    int n, words;
    int mode;                   // 0 values of one plane, 1 luma recombination, 2 pack of three planes
};

// Epilogue of the pixel-wise path: counts -> value (and optional colour packing).
struct EpilogueArgs {
    float *plane;               // counts in (unless bits), values out (in place)
    const unsigned int *bits;   // null, or the samples' bits: `words` words a pixel
    int words;
    int out_w, out_h, in_w, in_h;
    float inv_samples;
    unsigned char *out_rgb8;    // null: values only
    int mode;                   // 0 values, 1 luma recombine, 2 rgb pack (plane is channel 2)
    const float *cb, *cr;       // luma: chroma planes at input size
    const float *p0, *p1;       // rgb: rendered channels 0 and 1 (values)
};

// The platform-logf table on the device (fg_lambda.cu platform_logf).
struct LogfTableDev {
    const uint32_t *bucket_start, *keys, *vals;
    uint32_t lo_bits, hi_bits;
    int shift;
};

// The cell table, and n_clear words (the output's floats, or the samples' bits) and the counters set to zero
// beside it.
cudaError_t launch_cell_params(const float *lam, int in_w, int in_h, float delta, CellParam *cells, unsigned int *clear,
                               long long n_clear, PwCounters *counters, cudaStream_t s);
// counters: null (fat CTAs over every block) or cleared, with nbx*nby ints behind them (lean or sparse pass,
// then fat CTAs over the deferred blocks).
// cellmask: null, or pixelwise_cellmask_bytes(a, nby) bytes for the sparse pass's plane bitmask (the
// plane then takes the sparse pass, else the lean pass).
// bits: null, or pixelwise_stream_bytes(a, nby) cleared bytes (with cellmask: the plane takes the stream pass,
// which gives the samples' bits instead of the counts).
cudaError_t launch_pixelwise(const PixelwiseArgs &a, int nby, PwCounters *counters, unsigned int *cellmask,
                             unsigned int *bits, cudaStream_t s);
size_t pixelwise_stream_bytes(const PixelwiseArgs &a, int nby);
// Scratch bytes of the sparse pass's plane bitmask for this plane; 0 when the plane does not take it.
size_t pixelwise_cellmask_bytes(const PixelwiseArgs &a, int nby);
// Whether a plane runs on the per-sample kernel instead of the block kernel: in a batch, and on its own.
bool pixelwise_prefers_regen(const PixelwiseArgs &a);
bool pixelwise_takes_regen(const PixelwiseArgs &a);
size_t pixelwise_smem_bytes();  // the fat configuration (the batched kernel's pixel-wise items)
cudaError_t launch_grainwise(const GrainwiseArgs &a, int sms, cudaStream_t s);
size_t grainwise_smem_bytes(const GrainwiseArgs &a);
int grainwise_tile_count(const GrainwiseArgs &a);
size_t grainwise_work_ints(const GrainwiseArgs &a, int sms);  // the tile scheduler's area (GrainwiseArgs::work)
cudaError_t launch_grainwise_epilogue(const GrainwiseEpilogueArgs &a, cudaStream_t s);
cudaError_t launch_epilogue(const EpilogueArgs &a, cudaStream_t s);
cudaError_t launch_rgb_pack(const float *p0, const float *p1, const float *p2, int n, unsigned char *out,
                            cudaStream_t s);

}  // namespace fg
