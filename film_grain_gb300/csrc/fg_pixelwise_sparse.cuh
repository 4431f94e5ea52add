// fg_pixelwise_sparse.cuh -- the sparse block pass of the pixel-wise coverage estimator
// (src/pixelwise.rs:11-106): the first pass over every block of a plane whose grains are sparse
// enough to stage a large window in shared memory.  Blocks that turn out denser are left to the fat
// block pass (pixelwise_block<PwFat>), as the fat-grid blocks they cover.
//
// A CTA owns a square block of input space [X0, X1) x [Y0, Y1) (edge a power of two, `ratio` fat-grid
// blocks per side) and evaluates every sample (pixel, offset) whose point xg = ((x + 0.5) * inv_zoom) -
// offsets_input[k] lands in it:
//   0. (cell_mask_kernel, before the pass) the emptiness of every cell of the plane's cell grid is one
//      bit of a column-major bitmask in global memory: a thread owns one column and 32 rows (the column
//      stage of the cell hash computed once) and stores one word; a cell is empty when its first
//      uniform does not exceed its Knuth threshold, and the screen (first_draw_maybe) lists one in 2^8 of
//      the empty ones too.  Every cell is hashed once per plane;
//   1. the CTA copies the bits of its window -- the cells its owned samples can reach -- into shared
//      memory (column-major: word k of window column c holds rows 32k .. 32k + 31);
//   2. the set bits, ranked in column-major order, list the non-empty cells; their grain counts (the
//      Poisson draws of src/pixelwise.rs:77-82) are prefix-summed into a CSR over the list and their
//      grains (centre, radius^2) regenerated into shared memory;
//   3. each thread takes the owned pixels of one offset (or a share of them) and runs the
//      reference's per-sample test: for each cell column i0..i1 of the sample's range
//      (src/pixelwise.rs:55-58), the bits of rows j0..j1 are cut from the mask, and when any is set
//      their grains -- contiguous in the CSR, since cells of one column follow each other in the list
//      -- get the disk test dx*dx + dy*dy <= r*r (src/pixelwise.rs:96-99);
//   4. hit counts go to per-pixel shared counters, then to the output plane (integers, exact in f32).
// The indicator is an OR over the grains of the sample's cells, so the result equals the reference's
// early-exit loop bit for bit.
#pragma once
#include "fg_pixelwise.cuh"

namespace fg {

struct PwSparse {
    static constexpr int kThreads = 256, kCtasPerSm = 3;
    static constexpr int kGrainMax = 2048;   // staged grains
    static constexpr int kListMax = 2048;    // non-empty cells of the window
    static constexpr int kMaskWords = 1280;  // window bitmask, columns an odd number of words apart
    static constexpr int kRowsMax = 256;     // window rows
    static constexpr int kRangeSlots = 4;    // tabulated cell ranges per offset and axis
};

// Mask words per window column in shared memory: the column's words rounded up to an odd count, so
// that lanes reading the same word row of columns a multiple of 8 apart meet on different banks.
__host__ __device__ __forceinline__ int sparse_col_stride(int hw) { return hw | 1; }

// A sample's cell range on one axis, relative to the window [w0, w1] (at most kMaskWords cells): low
// 11 bits the first cell - w0, high 5 bits the last cell - the first; kRangeSlow when the range leaves
// the window or spans more than 32 cells (the per-sample loop decides such samples).
constexpr unsigned kRangeSlow = 0xFFFFu;
__device__ __forceinline__ unsigned sparse_range_code(float g, float rm, float delta, int w0, int w1) {
    const int c0 = f2i_floor(FG_FDIV(FG_FSUB(g, rm), delta));  // src/pixelwise.rs:55-58
    const int c1 = f2i_floor(FG_FDIV(FG_FADD(g, rm), delta));
    if (c0 < w0 || c1 > w1 || c1 < c0 || c1 - c0 > 31) return kRangeSlow;
    return (unsigned)(c0 - w0) | ((unsigned)(c1 - c0) << 11);
}

// The window's cells (steps 1 and 2, and step 3 in the sample-major form).
struct PwSparseWindow {
    uint2 mask2[PwSparse::kMaskWords];           // (word w, the next word of the same column or 0)
    unsigned short wrank[PwSparse::kMaskWords];  // non-empty cells before each mask word (column-major)
    unsigned short list[PwSparse::kListMax];     // non-empty cells: window index i * Hc + j, column-major
    unsigned int gsc[PwSparse::kListMax];        // per listed cell: first grain | grain count << 16
};
struct PwSparseShared {
    float4 grains[PwSparse::kGrainMax];          // centre, r^2, window cell (i - wi0) | (j - wj0) << 16 as bits
    PwSparseWindow w;
    int4 rect[kPwKChunk];                       // owned pixel rectangle per offset: xa, xe, ya, ye
    // cell ranges (sparse_range_code) of the first kRangeSlots columns and rows of each offset's
    // rectangle: entry [slot * n + k]
    unsigned short range_x[PwSparse::kRangeSlots * kPwKChunk], range_y[PwSparse::kRangeSlots * kPwKChunk];
    unsigned int cnt[kPwFootMax];
    int wsum[40];
    int wi0, wi1, wj0, wj1, Wc, Hc, hw, hs;     // the window: cells [wi0, wi1] x [wj0, wj1], hw words per
                                                // column stored hs = sparse_col_stride(hw) words apart
    int fx0, fx1, fy0, fy1, nsamples;           // owned-pixel footprint, owned samples
    int rw_min, rw_max, rh_min, rh_max;         // extremes of the offsets' rectangle widths and heights
    int stop, ngrains;
    float est_grains, est_cells;
};

// The CTA's PwSparseShared: the start of its dynamic shared memory, named through the shared array
// itself, so that the out-of-line functions below address it as shared memory (a reference passed in
// would reach them as a generic address).
__device__ __forceinline__ PwSparseShared &sparse_smem() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return *reinterpret_cast<PwSparseShared *>(smem_raw);
}

// Geometry of the sparse pass: block edge `bs` (input pixels) = ratio x the fat grid's edge, block grid
// origin and width (the fat grid is (a.bx0, a.by0, a.nbx) with a.bsize); and the plane's emptiness
// bitmask: cells [gi0, gi0 + gw) x [gj0, gj0 + 32 ghw), word (c, k) = cellmask[k * gw + c] holding rows
// gj0 + 32k .. + 31 of column gi0 + c (bit r = row gj0 + 32k + r).
struct PwSparseGrid {
    float bs;
    int ratio;
    int sbx0, sby0, nsbx, nsby;
    const unsigned int *cellmask;
    int gi0, gj0, gw, ghw;
};

// The plane's emptiness bitmask (step 0): word (column c, word row k), the lanes of a warp taking neighbouring
// columns of one word row (all 32 lanes; those past the last column write nothing).
// What bounds it: the shifts, xors and multiplies of the row hash and the screen, once per cell.
__device__ __forceinline__ void cell_mask_word(const PixelwiseArgs &a, const PwSparseGrid &g, int c, int k,
                                               unsigned int *cellmask) {
    const int i = g.gi0 + c, jb = g.gj0 + 32 * k, lane = (int)(threadIdx.x & 31);
    const uint64_t colh = cell_col_hash(a.seed, i);
    const CellParam *cells = a.cells + cell_axis_pixel(i, a.delta, a.in_w);
    // the word's 32 rows have the same lambda pixel rows on every lane: lane r converts row r, and the
    // rows where a new one starts cut the word into runs
    const int iy = cell_axis_pixel(jb + lane, a.delta, a.in_h);
    const int above = __shfl_up_sync(0xffffffffu, iy, 1);  // lane 0: its own
    const unsigned starts = __ballot_sync(0xffffffffu, iy != above);
    // The row stage of mix3 is fmix64(rotl64(col + j, 41) + phi).  With base = col + jb, when adding
    // r < 32 carries nothing out of base's low 23 bits, rotl64(base + r, 41) = rotl64(base, 41) + r * 2^41,
    // so the row hash's input is one constant plus r * 2^41 (only its high word changes); a word whose
    // rows would carry (31 in 2^23) takes the row hash as is.
    const uint64_t base = colh + (uint64_t)(int64_t)jb;
    const uint64_t c0 = rotl64(base, 41) + kPhi;
    const bool plain = (base & 0x7FFFFFull) <= 0x7FFFFFull - 31;
    unsigned int word = 0;
    for (int r0 = 0; r0 < 32;) {
        const unsigned later = starts & (r0 < 31 ? ~0u << (r0 + 1) : 0u);
        const int r1 = later ? __ffs(later) - 1 : 32;
        const uint32_t bound = maybe_bound(cells[(long long)__shfl_sync(0xffffffffu, iy, r0) * a.in_w].thresh);
        // the few empty cells that the screen lists are counted exactly by the passes that read the
        // bitmask (sparse_cell_count, cell_count_h)
        if (plain) {
#pragma unroll 4
            for (int r = r0; r < r1; r++)
                word |= (first_draw_maybe(fmix64(c0 + ((uint64_t)r << 41)), bound) ? 1u : 0u) << r;
        } else {
            for (int r = r0; r < r1; r++)
                word |= (first_draw_maybe(cell_row_hash(colh, jb + r), bound) ? 1u : 0u) << r;
        }
        __syncwarp();
        r0 = r1;
    }
    if (c < g.gw) cellmask[(long long)k * g.gw + c] = word;
}

// The reference's per-sample loop for a sample the staged window cannot serve (out of line: rare).
__device__ __noinline__ bool sparse_regen_sample(const PixelwiseArgs &a, float xg, float yg, int i0, int i1, int j0,
                                                 int j1) {
    const UniformF32 U = uniform_f32_new(0.0f, a.delta);
    return eval_regen(a, U, xg, yg, i0, i1, j0, j1);
}

// Grain count of cell (i, j), which the emptiness bitmask lists as non-empty, with the stream left
// after the Poisson draws: cell_count_h with the seeded stream's first output as its first draw (no
// separate first-draw hash).
__device__ __forceinline__ uint32_t sparse_cell_count(const PixelwiseArgs &a, int i, int j, Xoshiro *rng) {
    const CellParam cp = a.cells[cell_pixel(a, i, j)];
    const uint64_t h = cell_row_hash(cell_col_hash(a.seed, i), j);
    Xoshiro r = small_seed(h);
    uint32_t q = 0u;
    bool sure = false;
    if (cp.thresh >= 0) {
        // the first draw (above the threshold for every listed cell but one whose seed words 1, 2, 7 and
        // 8 are all zero, which the bitmask lists to be safe)
        const uint64_t first = r.next();
        if ((long long)(first >> 11) <= cp.thresh) {
            *rng = r;
            return 0u;
        }
        const float e = (float)(uint32_t)(cp.thresh >> 21) * 2.3283064365386963e-10f;
        sure = knuth_count_f32<true>(unit_f32(first), e, r, q);
    }
    if (!sure) {
        const DrawnCount d = cp.thresh >= 0 ? knuth_count_f64(h, cp.exp_lambda) : poisson_f64(h, (float)-cp.exp_lambda);
        r = d.rng;
        q = d.q;
    }
    *rng = r;
    return q;
}

// The fat-grid blocks of sparse block (sbx, sby), appended to the deferred list (list[0] = count).
__device__ __forceinline__ void sparse_defer(const PixelwiseArgs &a, const PwSparseGrid &g, int sbx, int sby,
                                             int nby, int *list) {
    for (int q = 0; q < g.ratio * g.ratio; q++) {
        const int bx = sbx * g.ratio + q % g.ratio, by = sby * g.ratio + q / g.ratio;
        if (bx < a.bx0 || bx >= a.bx0 + a.nbx || by < a.by0 || by >= a.by0 + nby) continue;
        list[1 + atomicAdd(list, 1)] = (by - a.by0) * a.nbx + (bx - a.bx0);
    }
}

// Sample (xg, yg) with cell-range codes rx, ry (neither kRangeSlow): 1 covered, else 0.  For each cell
// column of the range (src/pixelwise.rs:55-58) one 64-bit shared load gives the bits of its rows; the
// grains of the non-empty cells get the disk test (src/pixelwise.rs:96-99).  The columns are scanned
// first, branch-free, into a mask of the ones holding non-empty cells, and only those are visited: a
// warp's lanes then diverge over their few non-empty columns instead of over every column.
__device__ __forceinline__ int sparse_sample_hit(const PwSparseShared &S, float xg, float yg, unsigned rx,
                                                 unsigned ry) {
    const int hs = S.hs;
    const int c0 = (int)(rx & 0x7FFu), ncol = (int)(rx >> 11);
    const int r0 = (int)(ry & 0x7FFu), b0 = r0 & 31;
    const unsigned keep = (2u << (ry >> 11)) - 1u;  // span <= 31: 2u << 31 wraps to 0 and keep is all ones
    const unsigned below = (1u << b0) - 1u;
    const int w0 = c0 * hs + (r0 >> 5);
    unsigned cols = 0u;
    for (int i = 0; i <= ncol; i++) {
        const uint2 m = S.w.mask2[w0 + i * hs];
        cols |= ((__funnelshift_r(m.x, m.y, b0) & keep) != 0u ? 1u : 0u) << i;
    }
    while (cols) {
        const int w = w0 + (__ffs(cols) - 1) * hs;
        cols &= cols - 1u;
        const uint2 m = S.w.mask2[w];
        unsigned bits = __funnelshift_r(m.x, m.y, b0) & keep;
        int rank = S.w.wrank[w] + __popc(m.x & below);
        do {  // the column's non-empty cells of the range, in row order
            bits &= bits - 1u;
            const unsigned sc = S.w.gsc[rank++];
            const int g0 = (int)(sc & 0xFFFFu), ge = g0 + (int)(sc >> 16);
            for (int g = g0; g < ge; g++) {
                const float4 G = S.grains[g];
                const float dx = FG_FSUB(xg, G.x), dy = FG_FSUB(yg, G.y);
                if (FG_FADD(FG_FMUL(dx, dx), FG_FMUL(dy, dy)) <= G.z) return 1;
            }
        } while (bits);
    }
    return 0;
}

// The second pass over a thread's samples: the ones whose range left the window.
__device__ __noinline__ void sparse_slow_sample(const PixelwiseArgs &a, float xg, float yg, int x, int y);

__device__ __forceinline__ void sparse_count_hit(const PixelwiseArgs &a, PwSparseShared &S, int x, int y) {
    const int fw = S.fx1 - S.fx0, fh = S.fy1 - S.fy0;
    if ((long long)fw * fh <= kPwFootMax && x >= S.fx0 && x - S.fx0 < fw && y >= S.fy0 && y - S.fy0 < fh)
        atomicAdd(&S.cnt[(y - S.fy0) * fw + (x - S.fx0)], 1u);
    else
        atomicAdd(&a.out[(long long)y * a.out_w + x], 1.0f);
}

// Step 3.  The offsets are sorted by x, and consecutive threads take consecutive offsets, each walking
// the pixels its offset owns (`parts` threads per offset, taking alternate rows, when N < the CTA
// size): a warp's lanes evaluate samples of about the same pixel whose points lie close together in x,
// so their mask loads fall on neighbouring columns.  Cell ranges come from the table the ownership pass
// filled when every rectangle fits it, else they are computed here.
// One pass over the thread's samples: pass 0 evaluates every sample from the staged window and counts
// the ones whose range leaves it; pass 1 sends exactly those to the per-sample loop (and counts them).
template <int kPass>
__device__ __forceinline__ unsigned sparse_sample_pass(const PixelwiseArgs &a, PwSparseShared &S) {
    using C = PwSparse;
    const int tid = threadIdx.x, nthreads = blockDim.x;
    unsigned slow = 0;
    const bool table = S.rw_max <= C::kRangeSlots && S.rh_max <= C::kRangeSlots;
    const int parts = a.n >= nthreads ? 1 : nthreads / a.n;
    const int wi0 = S.wi0, wi1 = S.wi1, wj0 = S.wj0, wj1 = S.wj1;
    for (int t = tid; t < a.n * parts; t += nthreads) {
        const int k = t % a.n, p = t / a.n;
        const int4 R = S.rect[k];
        const float2 o = a.offs[k];
        for (int y = R.z + p; y < R.w; y += parts) {
            const float yg = xg_of(y, a.inv_zoom, o.y);
            const unsigned ry = table ? S.range_y[(y - R.z) * a.n + k]
                                      : sparse_range_code(yg, a.rm, a.delta, wj0, wj1);
            for (int x = R.x; x < R.y; x++) {
                const float xg = xg_of(x, a.inv_zoom, o.x);
                const unsigned rx = table ? S.range_x[(x - R.x) * a.n + k]
                                          : sparse_range_code(xg, a.rm, a.delta, wi0, wi1);
                const bool out = rx == kRangeSlow || ry == kRangeSlow;
                if (kPass == 0) {
                    if (out) slow++;
                    else if (sparse_sample_hit(S, xg, yg, rx, ry)) sparse_count_hit(a, S, x, y);
                } else if (out) {
                    slow++;
                    sparse_slow_sample(a, xg, yg, x, y);
                }
            }
        }
    }
    return slow;
}

__device__ __noinline__ void sparse_samples(const PixelwiseArgs &a) {
    PwSparseShared &S = sparse_smem();
    if (!(a.rm > 0.0f)) return;  // a grain radius is at most rm: nothing can cover a sample
    const unsigned slow = sparse_sample_pass<0>(a, S);
    if (__syncthreads_or(slow != 0)) {
        if (slow) atomicAdd(&a.diag[0], (unsigned long long)slow);
        sparse_sample_pass<1>(a, S);
    }
}

__device__ __noinline__ void sparse_slow_sample(const PixelwiseArgs &a, float xg, float yg, int x, int y) {
    PwSparseShared &S = sparse_smem();
    const int i0 = f2i_floor(FG_FDIV(FG_FSUB(xg, a.rm), a.delta));
    const int i1 = f2i_floor(FG_FDIV(FG_FADD(xg, a.rm), a.delta));
    const int j0 = f2i_floor(FG_FDIV(FG_FSUB(yg, a.rm), a.delta));
    const int j1 = f2i_floor(FG_FDIV(FG_FADD(yg, a.rm), a.delta));
    if (sparse_regen_sample(a, xg, yg, i0, i1, j0, j1)) sparse_count_hit(a, S, x, y);
}

// Step 2, out of line: the list of non-empty cells (column-major) with the rank before each mask
// word, then their grain counts, CSR prefix and grains.  Returns false (uniformly) when the list or
// the grains overflow their shared-memory buffers.
__device__ __noinline__ bool sparse_stage(const PixelwiseArgs &a) {
    PwSparseShared &S = sparse_smem();
    using C = PwSparse;
    const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
    const int Wc = S.Wc, Hc = S.Hc, hs = S.hs, wi0 = S.wi0, wj0 = S.wj0;
    if (tid == 0) S.ngrains = 0;  // read after the list's barrier
    const int nwords = Wc * hs;
    int nlist;
    {
        const int per = (nwords + nthreads - 1) / nthreads;
        const int b = tid * per, e = min(nwords, b + per);
        int local = 0;
        for (int w = b; w < e; w++) local += __popc(S.w.mask2[w].x);
        int total;
        int run = block_excl_scan(local, S.wsum, &total);
        nlist = total;
        if (total <= C::kListMax) {
            for (int w = b; w < e; w++) {
                S.w.wrank[w] = (unsigned short)run;
                unsigned m = S.w.mask2[w].x;
                const int col = w / hs, row0 = (w - col * hs) * 32;
                while (m) {
                    const int bit = __ffs(m) - 1;
                    m &= m - 1u;
                    S.w.list[run++] = (unsigned short)(col * Hc + row0 + bit);
                }
            }
        }
    }
    __syncthreads();
    if (nlist > C::kListMax) return false;
    // counts and grains in one pass: a warp takes 32 consecutive listed cells at a time, each lane counts
    // its cell's grains (the Poisson draws of src/pixelwise.rs:77-82), the lanes reserve their grains'
    // slots with a warp scan and one shared counter, and each lane regenerates its grains from the
    // stream the Poisson draws left (src/pixelwise.rs:84-95)
    const UniformF32 U = uniform_f32_new(0.0f, a.delta);
    for (int t0 = tid & ~31; t0 < nlist; t0 += nthreads) {  // warp-uniform bounds (the shuffles below)
        const int t = t0 + lane;
        int i = 0, j = 0;
        uint32_t q = 0u;
        Xoshiro rng;
        if (t < nlist) {
            const int c = S.w.list[t];
            i = wi0 + c / Hc;
            j = wj0 + c % Hc;
            q = sparse_cell_count(a, i, j, &rng);
        }
        const float cellw = __uint_as_float((unsigned)(i - wi0) | ((unsigned)(j - wj0) << 16));
        const int qc = (int)min(q, (uint32_t)C::kGrainMax + 1u);
        int incl = qc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        int base = 0;
        if (lane == 31) base = atomicAdd(&S.ngrains, incl);  // lane 31 holds the warp's total
        base = __shfl_sync(0xffffffffu, base, 31);
        const int first = base + incl - qc;
        if (t < nlist) {
            S.w.gsc[t] = (unsigned)(first & 0xFFFF) | ((unsigned)min(qc, 0xFFFF) << 16);
            if (first + qc <= C::kGrainMax) {
                const float sx = FG_FMUL((float)i, a.delta), sy = FG_FMUL((float)j, a.delta);
                for (int k = 0; k < qc; k++) {
                    const float cx = FG_FADD(sx, uniform_f32_from(U, rng.next()));
                    const float cy = FG_FADD(sy, uniform_f32_from(U, rng.next()));
                    float r = radius_draw(a, rng);
                    if (r > a.rm) r = a.rm;
                    const float rr = (r <= 0.0f) ? -1.0f : FG_FMUL(r, r);  // -1 never passes the disk test
                    S.grains[first + k] = make_float4(cx, cy, rr, cellw);
                }
            }
        }
    }
    __syncthreads();
    return S.ngrains <= C::kGrainMax;  // an overflow wrote no grain past the buffer; the block is redone
}

// One block of edge bs at block coordinates (bx, by) (all threads of the CTA; the dynamic shared memory
// holds PwSparseShared): 0 rendered (or nothing to render), 1 left undone (its buffers would overflow:
// nothing written), 2 stopped by cancellation.
__device__ __noinline__ int pixelwise_sparse_block(const PixelwiseArgs &a, const PwSparseGrid &g, float bs, int bx,
                                                   int by) {
    using C = PwSparse;
    PwSparseShared &S = sparse_smem();
    const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
    // the cancellation word, read now and tested after the ownership pass (its latency overlaps it)
    int cancel_seen = 0;
    if (tid == 0 && a.cancel) cancel_seen = *(volatile int *)a.cancel;

    const float X0 = FG_FMUL((float)bx, bs), X1 = FG_FMUL((float)(bx + 1), bs);
    const float Y0 = FG_FMUL((float)by, bs), Y1 = FG_FMUL((float)(by + 1), bs);
    // Every owned sample has xg in [X0, X1) and computes its cell range with these same rounded,
    // monotone operations, so its range lies inside [wi0, wi1] x [wj0, wj1].
    const int wi0 = f2i_floor(FG_FDIV(FG_FSUB(X0, a.rm), a.delta));
    const int wi1 = f2i_floor(FG_FDIV(FG_FADD(X1, a.rm), a.delta));
    const int wj0 = f2i_floor(FG_FDIV(FG_FSUB(Y0, a.rm), a.delta));
    const int wj1 = f2i_floor(FG_FDIV(FG_FADD(Y1, a.rm), a.delta));
    const int Wc = wi1 - wi0 + 1, Hc = wj1 - wj0 + 1;
    const int hw = (Hc + 31) >> 5;  // mask words per window column
    const int hs = sparse_col_stride(hw);
    const bool fits = Wc > 0 && Hc > 0 && Hc <= C::kRowsMax && Wc * hs <= C::kMaskWords &&
                      wi0 >= g.gi0 && wi1 < g.gi0 + g.gw && wj0 >= g.gj0 && wj1 < g.gj0 + 32 * (g.ghw - 1);

    if (tid == 0) {
        S.wi0 = wi0; S.wi1 = wi1; S.wj0 = wj0; S.wj1 = wj1; S.Wc = Wc; S.Hc = Hc; S.hw = hw; S.hs = hs;
        S.est_grains = 0.0f;
        S.est_cells = 0.0f;
        S.fx0 = 0x7fffffff; S.fx1 = -1; S.fy0 = 0x7fffffff; S.fy1 = -1; S.nsamples = 0;
        S.rw_min = 0x7fffffff; S.rw_max = -1; S.rh_min = 0x7fffffff; S.rh_max = -1;
    }
    __syncthreads();
    // ---- expected grains and non-empty cells of the window: lambda integrated over its rectangle (a
    // cell takes the lambda of the pixel containing its origin; edge pixels extend outwards)
    if (fits) {
        const float wx0 = FG_FMUL((float)wi0, a.delta), wx1 = FG_FMUL((float)(wi1 + 1), a.delta);
        const float wy0 = FG_FMUL((float)wj0, a.delta), wy1 = FG_FMUL((float)(wj1 + 1), a.delta);
        const int px0 = (int)floorf(wx0), px1 = (int)floorf(wx1), py0 = (int)floorf(wy0), py1 = (int)floorf(wy1);
        const int nx = px1 - px0 + 1, npx = nx * (py1 - py0 + 1);
        float ge = 0.0f, ce = 0.0f;
        const float inv_cell = 1.0f / (a.delta * a.delta);
        for (int t = tid; t < npx; t += nthreads) {
            const int px = px0 + t % nx, py = py0 + t / nx;
            const float ox = fminf((float)(px + 1), wx1) - fmaxf((float)px, wx0);
            const float oy = fminf((float)(py + 1), wy1) - fmaxf((float)py, wy0);
            if (ox > 0.0f && oy > 0.0f) {
                const int cx = min(max(px, 0), a.in_w - 1), cy = min(max(py, 0), a.in_h - 1);
                const float lam = a.lam[(long long)cy * a.in_w + cx];
                ge += lam * ox * oy;
                ce += (1.0f - __expf(-lam * a.delta * a.delta)) * ox * oy * inv_cell;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ge += __shfl_xor_sync(0xffffffffu, ge, o);
            ce += __shfl_xor_sync(0xffffffffu, ce, o);
        }
        if (lane == 0 && (ge > 0.0f || ce > 0.0f)) {
            atomicAdd(&S.est_grains, ge);
            atomicAdd(&S.est_cells, ce);
        }
    }
    // ---- ownership: rectangles per offset, sample total, pixel footprint, rectangle size extremes
    // (N <= kPwKChunk)
    {
        int lx0 = 0x7fffffff, lx1 = -1, ly0 = 0x7fffffff, ly1 = -1, ns = 0;
        int wmin = 0x7fffffff, wmax = -1, hmin = 0x7fffffff, hmax = -1;
        for (int k = tid; k < a.n; k += nthreads) {
            const float2 o = a.offs[k];
            const int xa = first_at_least(X0, a.out_w, a.inv_zoom, a.zoom, o.x);
            const int xe = first_at_least(X1, a.out_w, a.inv_zoom, a.zoom, o.x);
            const int ya = first_at_least(Y0, a.out_h, a.inv_zoom, a.zoom, o.y);
            const int ye = first_at_least(Y1, a.out_h, a.inv_zoom, a.zoom, o.y);
            S.rect[k] = make_int4(xa, xe, ya, ye);
            // the cell ranges of the rectangle's first columns and rows (pixelwise_sparse_block's table)
            for (int s2 = 0; s2 < min(xe - xa, C::kRangeSlots); s2++) {
                const unsigned c = sparse_range_code(xg_of(xa + s2, a.inv_zoom, o.x), a.rm, a.delta, wi0, wi1);
                S.range_x[s2 * a.n + k] = (unsigned short)c;
            }
            for (int s2 = 0; s2 < min(ye - ya, C::kRangeSlots); s2++) {
                const unsigned c = sparse_range_code(xg_of(ya + s2, a.inv_zoom, o.y), a.rm, a.delta, wj0, wj1);
                S.range_y[s2 * a.n + k] = (unsigned short)c;
            }
            wmin = min(wmin, xe - xa); wmax = max(wmax, xe - xa);
            hmin = min(hmin, ye - ya); hmax = max(hmax, ye - ya);
            if (xe > xa && ye > ya) {
                ns += (xe - xa) * (ye - ya);
                lx0 = min(lx0, xa); lx1 = max(lx1, xe);
                ly0 = min(ly0, ya); ly1 = max(ly1, ye);
            }
        }
        ns = __reduce_add_sync(0xffffffffu, ns);
        lx0 = __reduce_min_sync(0xffffffffu, lx0);
        lx1 = __reduce_max_sync(0xffffffffu, lx1);
        ly0 = __reduce_min_sync(0xffffffffu, ly0);
        ly1 = __reduce_max_sync(0xffffffffu, ly1);
        wmin = __reduce_min_sync(0xffffffffu, wmin);
        wmax = __reduce_max_sync(0xffffffffu, wmax);
        hmin = __reduce_min_sync(0xffffffffu, hmin);
        hmax = __reduce_max_sync(0xffffffffu, hmax);
        if (lane == 0) {
            if (ns > 0) {
                atomicAdd(&S.nsamples, ns);
                atomicMin(&S.fx0, lx0); atomicMax(&S.fx1, lx1);
                atomicMin(&S.fy0, ly0); atomicMax(&S.fy1, ly1);
            }
            if (wmax >= 0) {  // the warp saw offsets
                atomicMin(&S.rw_min, wmin); atomicMax(&S.rw_max, wmax);
                atomicMin(&S.rh_min, hmin); atomicMax(&S.rh_max, hmax);
            }
        }
    }
    if (tid == 0) {
        S.stop = cancel_seen;
        if (cancel_seen) *(volatile int *)(a.cancel + 1) = 1;
    }
    __syncthreads();
    if (S.stop) return 2;
    if (S.nsamples == 0) return 0;
    if (!fits || S.est_grains > 0.75f * (float)C::kGrainMax || S.est_cells > 0.75f * (float)C::kListMax)
        return 1;
    const int fw = S.fx1 - S.fx0, fh = S.fy1 - S.fy0;
    const bool use_cnt = (long long)fw * fh <= kPwFootMax;
    if (use_cnt)
        for (int t = tid; t < fw * fh; t += nthreads) S.cnt[t] = 0u;

    // ---- 1. the window's bits from the plane's bitmask (word k of window column c: rows 32k .. 32k + 31)
    {
        const int rb = wj0 - g.gj0, rw = rb >> 5, rs = rb & 31;
        const unsigned tail = (Hc & 31) ? ((1u << (Hc & 31)) - 1u) : 0xffffffffu;
        for (int idx = tid; idx < Wc * hs; idx += nthreads) {
            const int k = idx / Wc, c = idx - k * Wc;  // consecutive threads: consecutive columns
            unsigned word = 0u;                        // the pad word of an even hw stays empty
            if (k < hw) {
                const int gc = wi0 - g.gi0 + c;
                const unsigned lo = g.cellmask[(long long)(rw + k) * g.gw + gc];
                const unsigned hi = rs ? g.cellmask[(long long)(rw + k + 1) * g.gw + gc] : 0u;
                word = __funnelshift_r(lo, hi, rs);
                if (k == hw - 1) word &= tail;
            }
            S.w.mask2[c * hs + k].x = word;
        }
        __syncthreads();
        for (int w = tid; w < Wc * hs; w += nthreads) {
            const int k = w % hs;
            S.w.mask2[w].y = k + 1 < hw ? S.w.mask2[w + 1].x : 0u;
        }
        __syncthreads();
    }

    // ---- 2. non-empty cells, their counts and grains
    if (!sparse_stage(a)) return 1;

    // ---- 3. the owned samples
    sparse_samples(a);
    __syncthreads();

    // ---- 4. flush the per-pixel counts
    if (use_cnt) {
        for (int t = tid; t < fw * fh; t += nthreads) {
            const unsigned c = S.cnt[t];
            if (c) atomicAdd(&a.out[(long long)(S.fy0 + t / fw) * a.out_w + (S.fx0 + t % fw)], (float)c);
        }
    }
    if (tid == 0) {
        atomicAdd(&a.diag[3], 1ull);
        atomicAdd(&a.diag[4], 1ull);
    }
    return 0;
}

// Sparse block (sbx, sby): whole, or -- when it overflows -- as its fat-grid blocks one after another;
// a fat-grid block that overflows too is appended to the deferred list for the fat pass (each fat-grid
// block is either rendered here or listed, never both).
__device__ __forceinline__ void pixelwise_sparse_root(const PixelwiseArgs &a, const PwSparseGrid &g, int sbx, int sby,
                                                      int nby, int *list) {
    const int st = pixelwise_sparse_block(a, g, g.bs, sbx, sby);
    if (st != 1) return;
    if (g.ratio == 1) {
        if (threadIdx.x == 0) sparse_defer(a, g, sbx, sby, nby, list);
        return;
    }
    for (int q = 0; q < g.ratio * g.ratio; q++) {
        const int bx = sbx * g.ratio + q % g.ratio, by = sby * g.ratio + q / g.ratio;
        if (bx < a.bx0 || bx >= a.bx0 + a.nbx || by < a.by0 || by >= a.by0 + nby) continue;
        __syncthreads();  // the previous block's shared state is no longer read
        const int sq = pixelwise_sparse_block(a, g, a.bsize, bx, by);
        if (sq == 2) return;
        if (sq == 1 && threadIdx.x == 0) list[1 + atomicAdd(list, 1)] = (by - a.by0) * a.nbx + (bx - a.bx0);
    }
}

}  // namespace fg
