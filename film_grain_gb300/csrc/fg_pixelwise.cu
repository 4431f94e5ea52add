// fg_pixelwise.cu -- the pixel-wise coverage estimator (src/pixelwise.rs:11-106) for sm_103a.
//
// The reference loops pixel -> offset sample -> cell -> grain and regenerates every cell's grains
// from its cell_rng each time a sample visits it.  A plane takes one of three ways.  The stream pass
// (fg_pixelwise_stream.cuh) generates each grain once and finds the samples it covers: planes whose grains
// reach less than half an output pixel.  The per-sample kernel keeps that loop, one thread per output pixel
// (pixelwise_regen_pixels in fg_pixelwise.cuh), for planes whose samples reach fewer cells than a
// staged window would hold (small radii, few samples per pixel); the block kernels regroup the work by
// where the samples land: sample (pixel x,y; offset k) has the input-space point
//     xg = ((x + 0.5) * inv_zoom) - offsets_input[k][0]      (same f32 rounding as src/pixelwise.rs:34)
// and belongs to the block of input space [X0,X1) x [Y0,Y1) containing (xg, yg).  One CTA owns a
// block; it
//   A. hashes every cell of the block's window (the cells any owned sample can reach) once and
//      stores its grain count q (the Poisson draw of src/pixelwise.rs:77-82),
//   B. turns the counts into a row-major CSR prefix and regenerates the non-empty cells' grains
//      (centre, radius^2) into shared memory,
//   C. evaluates every owned sample: its exact cell range i0..i1 x j0..j1 (src/pixelwise.rs:55-58)
//      maps to one contiguous CSR interval per cell row; the sample is covered if any grain there
//      passes the reference's disk test dx*dx + dy*dy <= r*r (src/pixelwise.rs:96-99),
//   D. adds per-pixel hit counts (integers, exact in f32) into the output plane.
// Because a cell's grains depend only on (seed, i, j) and coverage is an OR over the grains of the
// sample's cells, the result equals the reference's early-exit loop bit for bit.  A block whose
// window holds more grains than shared memory splits into quadrants (up to kPwMaxLevel levels);
// border blocks (few owned samples), dense overflowing windows, samples whose cell range leaves the
// staged window (never expected) and leaf blocks that still overflow run the reference's per-sample
// regeneration instead, which is exact too.
#include <algorithm>
#include <cmath>

#include "fg_kernels.cuh"
#include "fg_rng.cuh"
#include "fg_color.cuh"
#include "fg_pixelwise.cuh"
#include "fg_pixelwise_sparse.cuh"
#include "fg_pixelwise_stream.cuh"

namespace fg {

// ------------------------------------------------------------------ per-pixel Poisson set-up
// What the later kernels add to -- the output or the bits, and the counters -- is cleared here too: each memset
// of its own was 6 us of the 208 us of a small plane
// between its first and last launch, which are bound by the host's enqueueing.
__global__ void cell_params_kernel(const float *__restrict__ lam, long long n, float delta,
                                   CellParam *__restrict__ cells, unsigned int *__restrict__ clear,
                                   long long n_clear, PwCounters *__restrict__ counters) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (long long)(sizeof(PwCounters) / sizeof(int))) reinterpret_cast<int *>(counters)[i] = 0;
    if (i < n_clear) clear[i] = 0u;
    if (i >= n) return;
    float l = lam[i];
    CellParam c;
    c.thresh = 0x7FFFFFFFFFFFFFFFll;
    c.exp_lambda = 0.0;
    if (l > 0.0f) {
        float expected = FG_FMUL(FG_FMUL(l, delta), delta);  // lambda_cell * delta * delta
        if (expected > 0.0f) {
            double e = (double)expected;
            if (e < 12.0) {
                double el = exp(-e);
                c.exp_lambda = el;
                c.thresh = (long long)FG_DMUL(el, 9007199254740992.0);  // floor(el * 2^53), exact scale
            } else {
                c.thresh = -1;
                c.exp_lambda = -e;
            }
        }
    }
    cells[i] = c;
}

cudaError_t launch_cell_params(const float *lam, int in_w, int in_h, float delta, CellParam *cells, unsigned int *clear,
                               long long n_clear, PwCounters *counters, cudaStream_t s) {
    const long long n = (long long)in_w * in_h;
    const long long grid = (std::max(n, n_clear) + 255) / 256;  // 256 threads and more: all words of the counters
    if (grid <= 0) return cudaSuccess;
    cell_params_kernel<<<(unsigned)grid, 256, 0, s>>>(lam, n, delta, cells, clear, n_clear, counters);
    return cudaGetLastError();
}

size_t pixelwise_smem_bytes() { return sizeof(PwShared<PwFat>); }

// One CTA per root block (block-grid row-major from (bx0, by0)).  With a list (lean pass), the blocks
// left to fat CTAs are appended to it: list[0] = count, list[1..] = block indices.
template <class C>
__global__ void __launch_bounds__(C::kThreads, C::kCtasPerSm)
    pixelwise_kernel(const __grid_constant__ PixelwiseArgs a, int *__restrict__ list) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int id = (int)blockIdx.x;
    const bool deferred = pixelwise_block<C>(a, a.bx0 + (int)(blockIdx.x % (unsigned)a.nbx),
                                             a.by0 + (int)(blockIdx.x / (unsigned)a.nbx), smem_raw, list != nullptr);
    if (deferred && threadIdx.x == 0) list[1 + atomicAdd(list, 1)] = id;
}

// The sparse pass: one CTA per sparse block (grid row-major from (sbx0, sby0)); the fat-grid blocks it
// leaves are appended to the list (list[0] = count, list[1..] = fat-grid block indices).
__global__ void __launch_bounds__(PwSparse::kThreads, PwSparse::kCtasPerSm)
    pixelwise_sparse_kernel(const __grid_constant__ PixelwiseArgs a, const PwSparseGrid g, int nby,
                            int *__restrict__ list) {
    const int sbx = g.sbx0 + (int)(blockIdx.x % (unsigned)g.nsbx), sby = g.sby0 + (int)(blockIdx.x / (unsigned)g.nsbx);
    pixelwise_sparse_root(a, g, sbx, sby, nby, list);
}

// The offsets in ascending x (ties by index: a permutation even with NaNs), for the sparse pass's
// lanes (sparse_sample_pass).  One CTA of kPwKChunk threads; n <= kPwKChunk.
__device__ __forceinline__ unsigned offset_sort_key(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);  // the float order as an unsigned order
}
__global__ void __launch_bounds__(kPwKChunk) sort_offsets_kernel(const float2 *__restrict__ offs, int n,
                                                                 float2 *__restrict__ sorted) {
    const int k = threadIdx.x;
    if (k >= n) return;
    const float2 o = offs[k];
    const unsigned key = offset_sort_key(o.x);
    int rank = 0;
    for (int j = 0; j < n; j++) {
        const unsigned kj = offset_sort_key(offs[j].x);
        rank += (kj < key || (kj == key && j < k)) ? 1 : 0;
    }
    sorted[rank] = o;
}

// The stream pass's tables: block 0 the offsets and their phase masks, the others the dense segments, a warp
// each.
struct StreamSetup {
    int segs, nw;  // nw: words of a mask
    float limit, w_max;
    unsigned char *dense;
    int *count, *list;
    float4 *ent;
    unsigned int *masks;
};
__global__ void __launch_bounds__(kPwKChunk) stream_setup_kernel(const __grid_constant__ PixelwiseArgs a,
                                                                 const __grid_constant__ StreamSetup t) {
    if (blockIdx.x > 0) {
        stream_classify(a, (long long)(blockIdx.x - 1) * (kPwKChunk / 32) + threadIdx.x / 32, t.segs, t.limit, t.dense,
                        t.count, t.list);
        return;
    }
    __shared__ float s_oz[2][kPwKChunk];
    if ((int)threadIdx.x < a.n) {
        const float2 o = a.offs[threadIdx.x];
        const float4 e = make_float4(o.x, o.y, FG_FMUL(o.x, a.zoom), FG_FMUL(o.y, a.zoom));
        t.ent[threadIdx.x] = e;
        s_oz[0][threadIdx.x] = e.z;
        s_oz[1][threadIdx.x] = e.w;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < phase_table_words(t.nw); w += blockDim.x) {
        const int word = w % t.nw, bucket = w / t.nw % kPhaseBuckets, cls = w / t.nw / kPhaseBuckets % kPhaseClasses;
        const int axis = w / t.nw / kPhaseBuckets / kPhaseClasses;
        t.masks[w] = phase_mask_word(s_oz[axis], a.n, bucket, cls, word, t.w_max);
    }
}

// The plane's emptiness bitmask (pixelwise_sparse_block step 0): one thread per mask word, row_ctas CTAs to a
// word row.
constexpr int kMaskThreads = 256;
__global__ void __launch_bounds__(kMaskThreads) cell_mask_kernel(const __grid_constant__ PixelwiseArgs a,
                                                                 const PwSparseGrid g, int row_ctas,
                                                                 unsigned int *__restrict__ cellmask) {
    const int k = (int)(blockIdx.x / (unsigned)row_ctas);
    const int c = (int)(blockIdx.x % (unsigned)row_ctas) * kMaskThreads + (int)threadIdx.x;
    if ((c & ~31) < g.gw) cell_mask_word(a, g, c, k, cellmask);  // whole warps
}

static int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// The window bounds of pixelwise_sparse_block, by the same f32 operations.
static int window_lo(float X0, const PixelwiseArgs &a) { return (int)std::floor((X0 - a.rm) / a.delta); }
static int window_hi(float X1, const PixelwiseArgs &a) { return (int)std::floor((X1 + a.rm) / a.delta); }

// Largest plane bitmask the sparse pass allocates (larger planes take the lean pass).
constexpr double kCellMaskMaxBytes = 16.0 * (1ull << 30);

// The sparse pass's block grid: the largest edge of 4, 2 or 1 fat-grid blocks whose window fits its
// bitmask and whose grid still gives every CTA slot several blocks; false when no edge fits (or N is
// above one offset chunk), and the plane takes the lean pass instead.
static bool plan_sparse(const PixelwiseArgs &a, int nby, int sms, PwSparseGrid *g) {
    if (a.n > kPwKChunk || !(a.rm >= 0.0f)) return false;
    for (int R = 4; R >= 1; R >>= 1) {
        const float bs = a.bsize * (float)R;
        const double edge = std::floor(((double)bs + 2.0 * a.rm) / a.delta) + 3.0;
        const double wpr = (double)sparse_col_stride((int)std::ceil(edge / 32.0));
        if (edge > PwSparse::kRowsMax || wpr * edge > PwSparse::kMaskWords) continue;
        const int sbx0 = floor_div(a.bx0, R), sbx1 = floor_div(a.bx0 + a.nbx - 1, R);
        const int sby0 = floor_div(a.by0, R), sby1 = floor_div(a.by0 + nby - 1, R);
        const long long blocks = (long long)(sbx1 - sbx0 + 1) * (sby1 - sby0 + 1);
        if (R > 1 && blocks < 4LL * sms * PwSparse::kCtasPerSm) continue;
        g->bs = bs;
        g->ratio = R;
        g->sbx0 = sbx0; g->sby0 = sby0;
        g->nsbx = sbx1 - sbx0 + 1; g->nsby = sby1 - sby0 + 1;
        // the bitmask covers every block's window with a two-cell margin
        const int gi0 = window_lo((float)sbx0 * bs, a) - 2, gi1 = window_hi((float)(sbx1 + 1) * bs, a) + 2;
        const int gj0 = window_lo((float)sby0 * bs, a) - 2, gj1 = window_hi((float)(sby1 + 1) * bs, a) + 2;
        g->cellmask = nullptr;
        g->gi0 = gi0;
        g->gj0 = gj0;
        g->gw = gi1 - gi0 + 1;
        g->ghw = (gj1 - gj0 + 1 + 31) / 32 + 1;  // one more word row for the windows' shifted reads
        return (double)g->gw * g->ghw * 4.0 <= kCellMaskMaxBytes;
    }
    return false;
}

static int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                    cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return sms;
}

// The sparse pass's scratch, each part 16-byte aligned: the bitmask, the offsets sorted by x -- or the stream
// pass's: the bitmask, the offsets (float4), their phase masks, the list of dense segments and their flags.
static size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }
static size_t sparse_mask_bytes(const PwSparseGrid &g) { return align16((size_t)g.gw * g.ghw * sizeof(unsigned int)); }
static int stream_words(int n) { return n <= 32 ? 1 : n <= 64 ? 2 : n <= 128 ? 4 : 8; }  // words of the kernel's variant
static size_t stream_masks_at(const PwSparseGrid &g, int n) {
    return sparse_mask_bytes(g) + align16((size_t)n * sizeof(float4));
}
static size_t stream_list_at(const PwSparseGrid &g, int n) {
    return stream_masks_at(g, n) + phase_table_words(stream_words(n)) * sizeof(unsigned int);
}

// The stream pass's plane conditions and tiles.  A grain reaches at most rm * zoom output pixels; the candidate
// pixel of an offset is exact while that reach plus the f32 rounding of the pixel coordinates (eps: a few
// ulps of the largest coordinate) stays below half a pixel, and the rounding to an integer by adding
// 1.5 * 2^23 needs coordinates below 2^22.
// Reach: up to 0.44, which leaves the candidate room for the rounding (500 x 400, constant radius 0.42, N 64: 478 us
// here, 518 us on the sparse pass; at 0.21, zoom 2, N 22 on 276 x 565: 411 and 641).
// Hits: the walk over a grain's hits costs per hit, the block passes per sample of a block, so those win where a
// grain covers many samples.  500 x 400 to 600 x 500, a ramp, here and on the block passes: 36 hits 862 and 968 us,
// 45 hits 1127 and 1423 (radius 0.3) or 747 and 828 (0.38), 55 hits 796 and 794 (0.42), 58 hits 1035 and 881, 72 hits
// 2123 and 1662; 116 hits (400 x 400, radius 0.19, zoom 2, N 256) 4799 and 2885.  Hence 48.
// Planes below kPwStreamPixels stay with the sparse and fat passes, whose forms the tests hold against the oracle
// there.
// Tiles: the largest of 512 .. 32 cells an edge whose footprint's bits leave room for many CTAs an SM and whose
// tiles give every CTA slot several; chunks are split while a warp would get few.
static bool plan_stream(const PixelwiseArgs &a, const PwSparseGrid &g, int sms, PwStreamGrid *t) {
    if ((double)a.out_w * a.out_h < kPwStreamPixels) return false;
    const double ext = std::max({std::fabs(a.offx_min), std::fabs(a.offx_max), std::fabs(a.offy_min),
                                 std::fabs(a.offy_max)});
    const double coord = (double)std::max(a.out_w, a.out_h) + ext * a.zoom + 2.0;
    const double eps = coord * 0x1p-21 + 0x1p-20;
    if (!(coord < 0x1p21) || !((double)a.rm * a.zoom + eps <= 0.44)) return false;
    const double hits = a.n * 3.14 * a.radius_mean * a.radius_mean * a.zoom * a.zoom;
    if (!(hits < 48.0)) return false;
    t->eps = (float)eps;
    // the roundings of xg, of xg +- rm, of the cell's origin and of the divisions: a few ulps of the largest
    // input coordinate
    const double grid = (double)std::max(a.out_w, a.out_h) * a.inv_zoom + ext + a.rm + 2.0;
    t->near_rm = (float)(a.rm - 16.0 * grid * 0x1p-23);
    t->nw = (a.n + 31) / 32;
    if ((double)a.out_w * a.out_h * t->nw * 4.0 > kCellMaskMaxBytes) return false;
    t->gi0 = g.gi0; t->gj0 = g.gj0; t->gw = g.gw; t->ghw = g.ghw;
    t->segs = (a.out_w + 31) / 32;
    for (int T = 512; T >= 32; T >>= 1) {
        auto edge = [&](float lo, float hi) {
            return std::floor(((double)T * a.delta + 2.0 * a.rm + (double)hi - (double)lo) * a.zoom) + 8.0;
        };
        const double words = edge(a.offx_min, a.offx_max) * edge(a.offy_min, a.offy_max) * t->nw;
        t->tile = T;
        t->ntx = (t->gw + T - 1) / T;
        t->nty = (32 * t->ghw + T - 1) / T;
        if (words <= (T == 32 ? 12288.0 : 4096.0) && (T == 32 || (double)t->ntx * t->nty >= 32.0 * sms)) {
            t->fp_words = (int)words;
            // parts of a tile's chunks: one or two for each of its eight warps
            const int chunks = (T / 32) * (T / 32);
            t->sub = chunks >= 16 ? 1 : chunks >= 4 ? 4 : 8;
            t->cols = (t->gw + 31) / 32;
            // no tiles (DIRECT) where they would be this small, unless a grain has many hits to gather
            t->direct = T <= 64 && t->gw < 65536 && 32.0 * t->ghw < 65536.0 &&
                        (double)a.out_w * a.out_h * t->nw < 0x1p31 &&
                        hits < 16.0;
            if (t->direct) t->sub = 8;
            return (double)t->ntx * t->nty < 2.0e9;
        }
    }
    return false;
}

size_t pixelwise_cellmask_bytes(const PixelwiseArgs &a, int nby) {
    if (pixelwise_takes_regen(a)) return 0;
    PwSparseGrid g;
    PwStreamGrid t;
    const int sms = sm_count() > 0 ? sm_count() : 152;  // without a device (planning only): the GB300's 152
    if (!plan_sparse(a, nby, sms, &g)) return 0;
    if (plan_stream(a, g, sms, &t)) return stream_list_at(g, a.n) + (size_t)t.segs * a.out_h * (sizeof(int) + 1);
    return sparse_mask_bytes(g) + (size_t)a.n * sizeof(float2);
}

size_t pixelwise_stream_bytes(const PixelwiseArgs &a, int nby) {
    if (pixelwise_takes_regen(a)) return 0;
    PwSparseGrid g;
    PwStreamGrid t;
    const int sms = sm_count() > 0 ? sm_count() : 152;
    return plan_sparse(a, nby, sms, &g) && plan_stream(a, g, sms, &t) ? (size_t)a.out_w * a.out_h * t.nw * 4 : 0;
}

// The root blocks the lean pass deferred, in fat CTAs: persistent, each CTA taking the next listed
// block from the counter defer[-1] (the word before the list's count).
__global__ void __launch_bounds__(PwFat::kThreads, PwFat::kCtasPerSm)
    pixelwise_deferred_kernel(const __grid_constant__ PixelwiseArgs a, int *__restrict__ defer) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_id;
    const int n = defer[0];
    for (;;) {
        if (threadIdx.x == 0) {
            const int i = atomicAdd(defer - 1, 1);
            s_id = (i < n && !cancel_requested(a.cancel)) ? defer[1 + i] : -1;
        }
        __syncthreads();
        const int id = s_id;
        if (id < 0) break;
        pixelwise_block<PwFat>(a, a.bx0 + id % a.nbx, a.by0 + id / a.nbx, smem_raw);
        __syncthreads();
    }
}

// Per-sample kernel: one thread per output pixel and part of its samples (pixelwise_regen_pixels).
// CTA b covers pixels [256 (c % row_ctas), +256) of row c / row_ctas, c = b / parts, and samples
// [per (b % parts), +per).
template <bool kTwoStep>
__global__ void __launch_bounds__(kPwRegenThreads) pixelwise_regen_kernel(const __grid_constant__ PixelwiseArgs a,
                                                                          int row_ctas, int parts, int per) {
    if (a.cancel && __syncthreads_or(threadIdx.x == 0 && cancel_requested(a.cancel))) return;
    const unsigned c = blockIdx.x / (unsigned)parts;
    const int k0 = (int)(blockIdx.x % (unsigned)parts) * per;
    pixelwise_regen_pixels<kTwoStep>(a, (int)(c % (unsigned)row_ctas) * kPwRegenThreads, (int)(c / (unsigned)row_ctas), k0,
                           min(a.n, k0 + per));
}

// The reach of an interior root block's samples, in windows of cells; infinite where the per-sample kernel cannot
// take the plane, 0 where it has nothing to do.
static double regen_reach(const PixelwiseArgs &a) {
    if (!(a.rm > 0.0f)) return 0.0;  // nothing can cover a sample: the per-sample loop exits at once
    // a sample's range must fit the 64-bit cell mask of pixelwise_pixel_queue
    const double axis = std::floor(2.0 * (double)a.rm / (double)a.delta) + 2.0;
    if (!(axis * axis <= 64.0)) return HUGE_VAL;
    // cell indices of every sample must stay far inside int (the range arithmetic)
    const double reach = (double)std::max(a.out_w, a.out_h) / a.zoom +
                         std::max({std::fabs(a.offx_min), std::fabs(a.offx_max), std::fabs(a.offy_min),
                                   std::fabs(a.offy_max)}) + a.rm + 2.0;
    if (reach / a.delta > 1.0e9) return HUGE_VAL;
    // an interior root block: its samples' reach in cells against its staged window
    const double samples = (double)a.bsize * a.bsize * a.zoom * a.zoom * a.n;
    const double edge = std::floor((a.bsize + 2.0 * a.rm) / a.delta) + 1.0;
    return samples * a.regen_cells / (edge * edge);
}

bool pixelwise_prefers_regen(const PixelwiseArgs &a) { return regen_reach(a) < kPwRegenKernel; }

// The planes that one render gives to the per-sample kernel: besides the ones of pixelwise_prefers_regen, small
// ones, whose block passes are a chain of a few CTAs' latencies (bitmask, sparse blocks, the dense blocks left
// over) while the per-sample kernel spreads their samples over the chip.
bool pixelwise_takes_regen(const PixelwiseArgs &a) {
    if (pixelwise_prefers_regen(a)) return true;
    const double visits = (double)a.out_w * a.out_h * a.n * a.regen_cells;
    return visits < kPwRegenSmallVisits && regen_reach(a) < kPwRegenSmall;
}

static cudaError_t launch_pixelwise_regen(const PixelwiseArgs &a, cudaStream_t s) {
    const long long row_ctas = (a.out_w + kPwRegenThreads - 1) / kPwRegenThreads;
    const long long grid = row_ctas * a.out_h;
    if (grid <= 0) return cudaSuccess;
    // A warp alone on its scheduler takes 3.6 us a sample, most of it waiting: with fewer warps than
    // kPwRegenWarps per SM the samples are split, down to one by one where that is what fills the chip (a
    // part's last round of cells is partly idle, but 96 x 64 N 32 takes 131 us a call in parts of four and
    // 32 warps, 111 us so).
    const int sms = sm_count();
    const double warps = (double)((a.out_w + 31) / 32) * a.out_h;
    const double want = warps > 0 ? kPwRegenWarps * (double)std::max(1, sms) / warps : 1.0;
    const int per = std::max(1, (int)std::ceil(a.n / std::max(1.0, want)));
    const int parts = (a.n + per - 1) / per;
    if (pixelwise_two_step(a))
        pixelwise_regen_kernel<true><<<(unsigned)(grid * parts), kPwRegenThreads, 0, s>>>(a, (int)row_ctas, parts, per);
    else
        pixelwise_regen_kernel<false><<<(unsigned)(grid * parts), kPwRegenThreads, 0, s>>>(a, (int)row_ctas, parts, per);
    return cudaGetLastError();
}

template <class K>
static cudaError_t set_smem(K k, size_t smem) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int NW, bool DIRECT>
static cudaError_t launch_stream_as(const PixelwiseArgs &a, const PwStreamGrid &t, int sms, cudaStream_t s) {
    const size_t smem = sizeof(PwStreamShared<NW>) + (DIRECT ? 0 : (size_t)t.fp_words * sizeof(unsigned int));
    cudaError_t e = set_smem(pixelwise_stream_kernel<NW, DIRECT>, smem);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pixelwise_stream_kernel<NW, DIRECT>, PwStream::kThreads, smem);
    if (e != cudaSuccess) return e;
    const long long work = DIRECT ? (long long)t.cols * t.ghw * t.sub * 32 / PwStream::kThreads + 1 : (long long)t.ntx * t.nty;
    const long long grid = std::min<long long>(work, (long long)sms * std::max(1, per_sm));
    pixelwise_stream_kernel<NW, DIRECT><<<(unsigned)grid, PwStream::kThreads, smem, s>>>(a, t);
    return cudaGetLastError();
}

template <int NW>
static cudaError_t launch_stream(const PixelwiseArgs &a, const PwStreamGrid &t, int sms, cudaStream_t s) {
    return t.direct ? launch_stream_as<NW, true>(a, t, sms, s) : launch_stream_as<NW, false>(a, t, sms, s);
}

// The plane's bits, its emptiness bitmask (g) written: the tables, the stream pass and the per-sample kernel over
// the dense segments.
static cudaError_t launch_pixelwise_stream(const PixelwiseArgs &a, const PwSparseGrid &g, PwStreamGrid t,
                                           PwCounters *counters, unsigned int *scratch, unsigned int *bits, int sms,
                                           cudaStream_t s) {
    char *base = reinterpret_cast<char *>(scratch);
    const int nw = stream_words(a.n);
    const long long nseg = (long long)t.segs * a.out_h;
    StreamSetup u;
    u.segs = t.segs;
    u.nw = nw;
    u.ent = reinterpret_cast<float4 *>(base + sparse_mask_bytes(g));
    u.masks = reinterpret_cast<unsigned int *>(base + stream_masks_at(g, a.n));
    u.list = reinterpret_cast<int *>(base + stream_list_at(g, a.n));
    u.dense = reinterpret_cast<unsigned char *>(u.list + nseg);
    u.count = &counters->list[1];
    // the per-sample kernel's limits, as pixelwise_prefers_regen
    const bool two = pixelwise_two_step(a);
    u.limit = std::isfinite(regen_reach(a))
                  ? (two ? kPwStreamDenseWide : kPwStreamDense) * (float)a.n * a.zoom * a.zoom
                  : HUGE_VALF;
    u.w_max = FG_FMUL(FG_FMUL(a.rm, a.zoom), 1.000008f) + t.eps;  // (stream_candidates' half-width of radius rm, rounded up)
    t.cellmask = g.cellmask;
    t.ent = u.ent;
    t.masks = u.masks;
    t.class_scale = (float)kPhaseClasses / u.w_max;
    t.bits = bits;
    t.next = &counters->tile;
    t.dense = u.dense;
    t.dense_count = u.count;
    constexpr int kSegs = kPwKChunk / 32;
    stream_setup_kernel<<<(unsigned)(1 + (nseg + kSegs - 1) / kSegs), kPwKChunk, 0, s>>>(a, u);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = nw == 1   ? launch_stream<1>(a, t, sms, s)
        : nw == 2 ? launch_stream<2>(a, t, sms, s)
        : nw == 4 ? launch_stream<4>(a, t, sms, s)
                  : launch_stream<8>(a, t, sms, s);
    if (e != cudaSuccess) return e;
    const long long ctas = std::min<long long>((nseg + 7) / 8, 4LL * std::max(1, sms));
    // Parts of eight samples: the last round of a part's cells is partly idle, which parts of four pay more often
    // (1024^2 log-normal 15.6 ms against 14.9), but where segments are few their warps' latency counts more
    // (256^2 ramp 0.32 ms against 0.35).
    const int part = nseg < 32LL * sms ? 4 : 8;
    auto *dense = two ? pixelwise_dense_kernel<true> : pixelwise_dense_kernel<false>;
    dense<<<(unsigned)ctas, kPwRegenThreads, 0, s>>>(a, bits, t.nw, t.segs, part, &counters->list[0], u.count, u.list);
    return cudaGetLastError();
}

cudaError_t launch_pixelwise(const PixelwiseArgs &a, int nby, PwCounters *counters, unsigned int *cellmask,
                             unsigned int *bits, cudaStream_t s) {
    if (pixelwise_takes_regen(a)) return launch_pixelwise_regen(a, s);
    const size_t lean_smem = sizeof(PwShared<PwLean>), fat_smem = sizeof(PwShared<PwFat>);
    const long long nblocks = (long long)a.nbx * nby;
    if (nblocks <= 0) return cudaSuccess;
    cudaError_t e;
    if (!counters) {
        e = set_smem(pixelwise_kernel<PwFat>, fat_smem);
        if (e != cudaSuccess) return e;
        pixelwise_kernel<PwFat><<<(unsigned)nblocks, PwFat::kThreads, fat_smem, s>>>(a, nullptr);
        return cudaGetLastError();
    }
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    int *list = &counters->list[1];  // the count, then the deferred root blocks
    PwSparseGrid g;
    const bool sparse = cellmask && plan_sparse(a, nby, sms, &g);
    if (sparse) {
        g.cellmask = cellmask;
        const int row_ctas = (g.gw + kMaskThreads - 1) / kMaskThreads;
        cell_mask_kernel<<<(unsigned)((long long)row_ctas * g.ghw), kMaskThreads, 0, s>>>(a, g, row_ctas, cellmask);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        PwStreamGrid t;
        if (bits && plan_stream(a, g, sms, &t)) return launch_pixelwise_stream(a, g, t, counters, cellmask, bits, sms, s);
        PixelwiseArgs as = a;  // the sparse pass reads the offsets sorted by x
        float2 *sorted = reinterpret_cast<float2 *>(reinterpret_cast<char *>(cellmask) + sparse_mask_bytes(g));
        as.offs = sorted;
        sort_offsets_kernel<<<1, kPwKChunk, 0, s>>>(a.offs, a.n, sorted);
        const size_t sparse_smem = sizeof(PwSparseShared);
        e = set_smem(pixelwise_sparse_kernel, sparse_smem);
        if (e != cudaSuccess) return e;
        pixelwise_sparse_kernel<<<(unsigned)((long long)g.nsbx * g.nsby), PwSparse::kThreads, sparse_smem, s>>>(
            as, g, nby, list);
    } else {
        e = set_smem(pixelwise_kernel<PwLean>, lean_smem);
        if (e != cudaSuccess) return e;
        pixelwise_kernel<PwLean><<<(unsigned)nblocks, PwLean::kThreads, lean_smem, s>>>(a, list);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = set_smem(pixelwise_deferred_kernel, fat_smem);
    if (e != cudaSuccess) return e;
    const long long grid = std::min<long long>(nblocks, (long long)std::max(1, sms) * PwFat::kCtasPerSm);
    PixelwiseArgs ad = a;  // after the sparse pass, the fat pass reads cell emptiness from its bitmask
    if (sparse) {
        ad.cellmask = cellmask;
        ad.cm_gi0 = g.gi0;
        ad.cm_gj0 = g.gj0;
        ad.cm_gw = g.gw;
        ad.cm_ghw = g.ghw;
    }
    pixelwise_deferred_kernel<<<(unsigned)grid, PwFat::kThreads, fat_smem, s>>>(ad, list);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ epilogue: counts -> values (+ colour)
__global__ void epilogue_kernel(const EpilogueArgs a) {
    long long n = (long long)a.out_w * a.out_h;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float count;
    if (a.bits) {
        const unsigned int *m = a.bits + i * a.words;
        int c = 0;
        for (int w = 0; w < a.words; w++) c += __popc(m[w]);
        count = (float)c;
    } else {
        count = a.plane[i];
    }
    const float v = FG_FMUL(count, a.inv_samples);  // sum * inv_samples (src/pixelwise.rs:38)
    a.plane[i] = v;
    if (!a.out_rgb8) return;
    unsigned char *o = a.out_rgb8 + 3 * i;
    if (a.mode == 1) {
        int x = (int)(i % a.out_w), y = (int)(i / a.out_w);
        float cbv, crv;
        if (a.in_w == a.out_w && a.in_h == a.out_h) {
            cbv = a.cb[i]; crv = a.cr[i];
        } else {
            float sxs = FG_FDIV((float)a.in_w, (float)a.out_w), sys = FG_FDIV((float)a.in_h, (float)a.out_h);
            long long src = (long long)nearest_src(y, sys, a.in_h) * a.in_w + nearest_src(x, sxs, a.in_w);
            cbv = a.cb[src]; crv = a.cr[src];
        }
        luma_rgb8(v, cbv, crv, o);
    } else if (a.mode == 2) {
        o[0] = to_u8(a.p0[i]); o[1] = to_u8(a.p1[i]); o[2] = to_u8(v);
    }
}

cudaError_t launch_epilogue(const EpilogueArgs &a, cudaStream_t s) {
    long long n = (long long)a.out_w * a.out_h;
    if (n <= 0) return cudaSuccess;
    epilogue_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

__global__ void rgb_pack_kernel(const float *p0, const float *p1, const float *p2, int n, unsigned char *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[3 * i] = to_u8(p0[i]); out[3 * i + 1] = to_u8(p1[i]); out[3 * i + 2] = to_u8(p2[i]);
}
cudaError_t launch_rgb_pack(const float *p0, const float *p1, const float *p2, int n, unsigned char *out,
                            cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    rgb_pack_kernel<<<(n + 255) / 256, 256, 0, s>>>(p0, p1, p2, n, out);
    return cudaGetLastError();
}

}  // namespace fg
