// fg_pixelwise_stream.cuh -- the grain-major pass of the pixel-wise coverage estimator (src/pixelwise.rs:11-106),
// for planes whose grains reach less than half an output pixel (plan_stream).
//
// The plane's cells are cut into square tiles, and a tile's grains are generated once, straight from the
// plane's emptiness bitmask (cell_mask_kernel), each lane of a warp drawing the grains of one cell.  A grain
// covers a sample (pixel, offset) when the sample's distance is at most its radius (src/pixelwise.rs:96-99)
// and the sample's cell range holds the grain's cell (src/pixelwise.rs:55-58).  For one offset only one pixel
// can lie within half a pixel of the grain, and the offsets for which one does follow from the phases of both
// (fg_phase.cuh): the grain's phases on the two axes and its radius select two masks of the offsets, whose
// intersection are its few candidates, which the warp tests 32 at a time.  A hit sets the sample's bit in the
// tile's part of the plane -- the pixels that its grains reach through some offset -- in shared memory; at the
// tile's end the words that are not zero join the plane's bits in global memory, and the epilogue counts them.
// Coverage is an OR over the cells, so neither the order nor a bit set twice changes it, and no grain is held,
// nor generated for a neighbouring tile as well.
// Segments of 32 output pixels that hold many grains are left to the per-sample kernel (stream_classify).
//
// What bounds it: the instructions of the grains' draws (seed words, Poisson and position draws, the
// log-normal radius) and of their candidates: 70 ps a grain on the log-normal plane below.  It replaced a form of the
// sparse pass that staged each block's grains in shared memory, generating a window's margin again for every block,
// and the fat pass over the denser blocks: GB300, 1024^2 log-normal 0.025 N 256 sparse + fat 32.6 ms, stream +
// per-sample 9.8; 1080p radius 0.1 N 32 2.49 and 1.00; 256^2 ramp 0.12 N 64 0.30 and 0.15.
#pragma once

#include "fg_phase.cuh"
#include "fg_pixelwise_sparse.cuh"

namespace fg {

struct PwStream {
    // Eight warps share a tile's tables and bits: four take 1024^2 log-normal, N 256 from 14.9 to 16.4 ms, and leave
    // the saturated tiles of small planes to fewer (200^2 ramp radius 0.2, N 200: 0.54 ms against 0.81).
    static constexpr int kThreads = 256;
    static constexpr int kPairs = 256;               // a warp's queue of (grain, entry) candidates
};

struct PwStreamWarp {
    float4 grain[64];  // ring of drawn grains: centre, r^2, cell (column | row << 16, of the tile) as bits
    uint2 cell[64];    // ring of cells to draw: column, row of the plane's bitmask
    unsigned short pairs[PwStream::kPairs];  // lane << 8 | entry
};
template <int NW>
struct PwStreamShared {
    float4 ent[32 * NW];  // the offsets: o.x, o.y, o.x * zoom, o.y * zoom
    unsigned int mask[phase_table_words(NW)];  // [axis][class][bucket][word]
    PwStreamWarp warp[PwStream::kThreads / 32];
    int tile, chunk, unused[2];
    // then the tile's bits: pixel (x, y) of the footprint has words [(y * fw + x) * nw, +nw)
    __device__ __forceinline__ unsigned int *bits() { return reinterpret_cast<unsigned int *>(this + 1); }
};

// tile: edge in cells (a multiple of 32); ntx x nty tiles from cell (gi0, gj0); nw: words of a pixel's bits;
// fp_words: words of a tile's bits at most; sub: parts of a chunk of 32 x 32 cells (one warp's work at a time)
struct PwStreamGrid {
    const unsigned int *cellmask;
    int gi0, gj0, gw, ghw;
    const float4 *ent;          // [n]
    const unsigned int *masks;  // phase_table_words(words of the kernel's variant)
    float eps;        // rounding margin of a grain's phase band, in output pixels
    float near_rm;    // |dx| up to this: the sample's range holds the grain's cell
    float class_scale;  // a band's half-width times this: its radius class
    int tile, ntx, nty, nw, fp_words, sub;
    int direct, cols;  // direct: no tiles, the hits go to the plane's bits; cols: chunks of a word row
    unsigned int *bits;  // [out_h * out_w * nw]
    int *next;           // the next tile
    const unsigned char *dense;  // per segment of 32 output pixels: left to the per-sample pass
    const int *dense_count;
    int segs;                    // segments of an output row
};

// The output pixels that are left to the per-sample pass, in segments of 32 pixels of a row (one warp each):
// a grain costs the stream pass about the same everywhere, while a sample of a dense segment is covered by
// the first cells that are looked at.
__device__ __forceinline__ void stream_classify(const PixelwiseArgs &a, long long seg, int segs, float limit,
                                                unsigned char *dense, int *count, int *list) {
    if (seg >= (long long)segs * a.out_h) return;
    const int lane = threadIdx.x & 31, y = (int)(seg / segs), x0 = 32 * (int)(seg % segs), x = x0 + lane;
    float lam = 0.0f;
    if (x < a.out_w) {
        const int xi = min(a.in_w - 1, max(0, (int)floorf(((float)x + 0.5f) * a.inv_zoom)));
        const int yi = min(a.in_h - 1, max(0, (int)floorf(((float)y + 0.5f) * a.inv_zoom)));
        lam = a.lam[(long long)yi * a.in_w + xi];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lam += __shfl_xor_sync(0xffffffffu, lam, o);
    if (lane != 0) return;
    const bool is = lam > limit * (float)min(32, a.out_w - x0);
    dense[seg] = is ? 1 : 0;
    if (is) list[atomicAdd(count, 1)] = (int)seg;
}

// The pixel coordinate of an offset that grain coordinate p = g * zoom - 0.5 can reach, as a float: p + o * zoom
// rounded to an integer by adding and removing 1.5 * 2^23.
__device__ __forceinline__ float stream_pixel(float p, float oz) {
    constexpr float kRint = 12582912.0f;
    return FG_FSUB(FG_FADD(FG_FADD(p, oz), kRint), kRint);
}

// The candidate (grain at (gx, gy) with r^2 = rr in cell (i, j), entry e): its bit when it is covered.
// (all 32 lanes; src: the lane that holds the grain)
struct StreamGrain {
    float gx, gy, rr;
    int i, j;
};
template <int NW>
__device__ __forceinline__ void stream_test(const PixelwiseArgs &a, const PwStreamGrid &g, PwStreamShared<NW> &S,
                                            unsigned int *bits, const StreamGrain &G, bool live, int src, int e, int fx0,
                                            int fy0, int fw, int fh) {
    const float gx = __shfl_sync(0xffffffffu, G.gx, src), gy = __shfl_sync(0xffffffffu, G.gy, src);
    const float rr = __shfl_sync(0xffffffffu, G.rr, src);
    const float4 O = S.ent[e];
    const float rx = stream_pixel(FG_FSUB(FG_FMUL(gx, a.zoom), 0.5f), O.z);
    const float ry = stream_pixel(FG_FSUB(FG_FMUL(gy, a.zoom), 0.5f), O.w);
    const float xg = FG_FSUB(FG_FMUL(FG_FADD(rx, 0.5f), a.inv_zoom), O.x);
    const float yg = FG_FSUB(FG_FMUL(FG_FADD(ry, 0.5f), a.inv_zoom), O.y);
    const float dx = FG_FSUB(xg, gx), dy = FG_FSUB(yg, gy);
    bool hit = live && FG_FADD(FG_FMUL(dx, dx), FG_FMUL(dy, dy)) <= rr;
    // A sample nearer than rm by some roundings on both axes has the grain's cell in its range; the others
    // compute it.
    const bool edge = hit && fmaxf(fabsf(dx), fabsf(dy)) > g.near_rm;
    if (__any_sync(0xffffffffu, edge)) {
        const int i = __shfl_sync(0xffffffffu, G.i, src), j = __shfl_sync(0xffffffffu, G.j, src);
        if (edge)
            hit = i >= f2i_floor(FG_FDIV(FG_FSUB(xg, a.rm), a.delta)) &&
                  i <= f2i_floor(FG_FDIV(FG_FADD(xg, a.rm), a.delta)) &&
                  j >= f2i_floor(FG_FDIV(FG_FSUB(yg, a.rm), a.delta)) &&
                  j <= f2i_floor(FG_FDIV(FG_FADD(yg, a.rm), a.delta));
    }
    if (!hit) return;
    const int x = (int)rx - fx0, y = (int)ry - fy0;
    if ((unsigned)x < (unsigned)fw && (unsigned)y < (unsigned)fh)  // else outside the plane
        atomicOr(bits + (y * fw + x) * g.nw + (e >> 5), 1u << (e & 31));
}

// The candidates of 32 grains, one per lane (G.rr < 0: none): each lane intersects the two axes' words for its
// grain's phases and radius and counts them, the warp lists its (grain, offset) candidates at the lanes' prefix
// of the counts, as many as the queue holds at a time, and tests them 32 at a time, every lane busy.
template <int NW>
__device__ __forceinline__ void stream_candidates(const PixelwiseArgs &a, const PwStreamGrid &g, PwStreamShared<NW> &S,
                                                  PwStreamWarp &W, unsigned int *bits, const StreamGrain &G, int fx0,
                                                  int fy0, int fw, int fh) {
    const int lane = threadIdx.x & 31;
    unsigned m[NW];
    int cnt = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) m[w] = 0u;
    if (G.rr >= 0.0f) {
        const float w = fmaf(sqrtf(G.rr), a.zoom * 1.0000039f, g.eps);  // the half-width ((1 + 2^-18): sqrt's rounding)
        const int cls = phase_class(w, g.class_scale);
        const int bx = phase_bucket(FG_FSUB(FG_FMUL(G.gx, a.zoom), 0.5f));
        const int by = phase_bucket(FG_FSUB(FG_FMUL(G.gy, a.zoom), 0.5f));
        const unsigned *mx = S.mask + (cls * kPhaseBuckets + bx) * NW;
        const unsigned *my = S.mask + ((kPhaseClasses + cls) * kPhaseBuckets + by) * NW;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            m[w] = mx[w] & my[w];
            cnt += __popc(m[w]);
        }
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int at = incl - cnt;  // the lane's next candidate, of the warp's
    for (int base = 0; base < total; base += PwStream::kPairs) {
        const int end = min(incl, base + PwStream::kPairs);
#pragma unroll
        for (int w = 0; w < NW; w++)
            while (m[w] != 0u && at < end) {
                W.pairs[at++ - base] = (unsigned short)((lane << 8) | (32 * w + __ffs(m[w]) - 1));
                m[w] &= m[w] - 1u;
            }
        __syncwarp();
        const int here = min(total - base, PwStream::kPairs);
        for (int i = 0; i < here; i += 32) {
            const bool live = i + lane < here;
            const unsigned pr = W.pairs[live ? i + lane : 0];
            stream_test(a, g, S, bits, G, live, (int)(pr >> 8), (int)(pr & 0xFFu), fx0, fy0, fw, fh);
        }
        __syncwarp();  // the queue is read before it is written again
    }
}

// Dynamic shared memory: PwStreamShared and fp_words words of bits.
// DIRECT (small planes): the warps take chunks of the whole plane, keep their queues from one to the next and set
// the hits' bits in global memory.  A tile of such a plane holds few grains a warp: 256^2 ramp radius 0.12, N 64,
// where each tile's last steps ran with few lanes, 330 us a call in tiles, 255 us so; 700 x 900, N 100, zoom 1.5
// 2.37 and 2.08 ms.  With many hits a grain the atomics show (200^2 radius 0.2, N 200, 25 hits: 0.52 and 0.58 ms), and
// on large planes too (1080p radius 0.1, N 32: 1.87 and 2.30 ms).
template <int NW, bool DIRECT>
__global__ void __launch_bounds__(PwStream::kThreads)
    pixelwise_stream_kernel(const __grid_constant__ PixelwiseArgs a, const __grid_constant__ PwStreamGrid g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PwStreamShared<NW> &S = *reinterpret_cast<PwStreamShared<NW> *>(smem_raw);
    constexpr int nthreads = PwStream::kThreads;
    const int tid = threadIdx.x, lane = tid & 31;
    PwStreamWarp &W = S.warp[tid >> 5];
    unsigned int *bits = DIRECT ? g.bits : S.bits();
    for (int e = tid; e < a.n; e += nthreads) S.ent[e] = g.ent[e];
    for (int b = tid; b < phase_table_words(NW); b += nthreads) S.mask[b] = g.masks[b];
    const UniformF32 U = uniform_f32_new(0.0f, a.delta);
    const int ntiles = g.ntx * g.nty, chunk_rows = g.tile >> 5;
    const bool any_dense = *g.dense_count != 0;
    CancelPoll poll;  // (DIRECT)
    poll.begin();
    for (;;) {
        __syncthreads();  // the tables; the previous tile's bits are written out
        int tile = 0;
        if (!DIRECT) {
            if (tid == 0) {
                const int t = atomicAdd(g.next, 1);
                S.tile = (t < ntiles && !cancel_requested(a.cancel)) ? t : -1;
                S.chunk = 0;
            }
            __syncthreads();
            tile = S.tile;
            if (tile < 0) return;
        }
        const int tc = (tile % g.ntx) * g.tile, tw = (tile / g.ntx) * chunk_rows;  // first column, first word row
        // the pixels whose samples its grains can reach, with a pixel of slack for the rounding
        const float X0 = (float)(g.gi0 + tc) * a.delta - a.rm, X1 = (float)(g.gi0 + tc + g.tile) * a.delta + a.rm;
        const float Y0 = (float)(g.gj0 + 32 * tw) * a.delta - a.rm, Y1 = (float)(g.gj0 + 32 * tw + g.tile) * a.delta + a.rm;
        const int fx0 = DIRECT ? 0 : max(0, (int)floorf((X0 + a.offx_min) * a.zoom - 0.5f) - 1);
        const int fx1 = DIRECT ? a.out_w - 1 : min(a.out_w - 1, (int)ceilf((X1 + a.offx_max) * a.zoom - 0.5f) + 1);
        const int fy0 = DIRECT ? 0 : max(0, (int)floorf((Y0 + a.offy_min) * a.zoom - 0.5f) - 1);
        const int fy1 = DIRECT ? a.out_h - 1 : min(a.out_h - 1, (int)ceilf((Y1 + a.offy_max) * a.zoom - 0.5f) + 1);
        const int fw = fx1 - fx0 + 1, fh = fy1 - fy0 + 1;
        const int row_words = fw * g.nw, words = row_words * fh;
        if (!DIRECT) {
            if (fw <= 0 || fh <= 0 || (long long)fw * fh * g.nw > g.fp_words) continue;  // (the plan's bound holds)
            for (int w = tid; w < words; w += nthreads) bits[w] = 0u;
            __syncthreads();
        }

        int head = 0, queued = 0, ghead = 0, grains = 0;  // the warp's rings; uniform
        auto cover = [&](int count) {  // the first `count` grains, one per lane
            const float4 v = W.grain[(ghead + (lane < count ? lane : 0)) & 63];
            __syncwarp();
            ghead += count;
            grains -= count;
            StreamGrain G;
            G.gx = v.x;
            G.gy = v.y;
            G.rr = lane < count ? v.z : -1.0f;
            G.i = g.gi0 + tc + (int)(__float_as_uint(v.w) & 0xFFFFu);
            G.j = g.gj0 + 32 * tw + (int)(__float_as_uint(v.w) >> 16);
            stream_candidates<NW>(a, g, S, W, bits, G, fx0, fy0, fw, fh);
        };
        // Each lane draws the grains of one cell, one a step, and takes the next cell from the ring when it has
        // no more: a lane whose cell holds several grains does not leave the others waiting.
        Xoshiro rng = {0, 0, 0, 0};
        uint32_t q = 0u;
        float sx = 0.0f, sy = 0.0f, at = 0.0f;
        bool more = true;  // cells may still come
        auto step = [&]() {
            const unsigned idle = __ballot_sync(0xffffffffu, q == 0u);
            const int take = min(queued, __popc(idle)), rank = __popc(idle & ((1u << lane) - 1u));
            if (q == 0u && rank < take) {
                const uint2 cell = W.cell[(head + rank) & 63];
                const int i = g.gi0 + (int)cell.x, j = g.gj0 + (int)cell.y;
                at = __uint_as_float((cell.x - (unsigned)tc) | ((cell.y - 32u * (unsigned)tw) << 16));
                sx = FG_FMUL((float)i, a.delta);
                sy = FG_FMUL((float)j, a.delta);
                q = sparse_cell_count(a, i, j, &rng);
            }
            head += take;
            queued -= take;
            float4 v = make_float4(0.0f, 0.0f, -1.0f, at);
            if (q != 0u) {
                q--;
                v.x = FG_FADD(sx, uniform_f32_from(U, rng.next()));
                v.y = FG_FADD(sy, uniform_f32_from(U, rng.next()));
                float r = radius_draw(a, rng);
                if (r > a.rm) r = a.rm;
                if (r > 0.0f) v.z = FG_FMUL(r, r);  // a radius <= 0 covers nothing
            }
            const unsigned have = __ballot_sync(0xffffffffu, v.z >= 0.0f);
            if (v.z >= 0.0f) W.grain[(ghead + grains + __popc(have & ((1u << lane) - 1u))) & 63] = v;
            grains += __popc(have);
            __syncwarp();
            if (grains >= 32 || (!more && have == 0u)) cover(min(grains, 32));
        };
        const int rows = 32 / g.sub, across = DIRECT ? g.cols : chunk_rows;
        const int chunks = across * (DIRECT ? g.ghw : chunk_rows) * g.sub;
        int taken = 0, col = 0, k = 0;
        unsigned word = 0u, pending = 0u;
        // Cells into the ring until it holds 32 or there are no more, then a step: one place for each, as the code of
        // a step is what the instruction cache holds.
        for (;;) {
            while (more && queued < 32) {
                if (pending == 0u) {
                    int c = chunks;
                    if (lane == 0 && !(DIRECT && poll.requested(a.cancel))) c = atomicAdd(DIRECT ? g.next : &S.chunk, 1);
                    c = __shfl_sync(0xffffffffu, c, 0);
                    if (c >= chunks) {
                        more = false;
                        break;
                    }
                    taken++;
                    const int part = c % g.sub;
                    c /= g.sub;
                    col = tc + 32 * (c % across) + lane;
                    k = tw + c / across;
                    if (any_dense) {
                        // nothing to do when every pixel whose samples the chunk's grains reach is left to the
                        // per-sample pass
                        const float cx = (float)(g.gi0 + col - lane) * a.delta, cy = (float)(g.gj0 + 32 * k) * a.delta;
                        const float side = 32.0f * a.delta + a.rm;
                        const int px0 = max(0, (int)floorf((cx - a.rm + a.offx_min) * a.zoom - 0.5f) - 1);
                        const int px1 = min(a.out_w - 1, (int)ceilf((cx + side + a.offx_max) * a.zoom - 0.5f) + 1);
                        const int py0 = max(0, (int)floorf((cy - a.rm + a.offy_min) * a.zoom - 0.5f) - 1);
                        const int py1 = min(a.out_h - 1, (int)ceilf((cy + side + a.offy_max) * a.zoom - 0.5f) + 1);
                        bool left = true;
                        if (px0 <= px1)
                            for (int py = py0 + lane; py <= py1 && left; py += 32)
                                for (int sg = px0 >> 5; sg <= px1 >> 5; sg++)
                                    left = left && g.dense[(long long)py * g.segs + sg] != 0;
                        if (__all_sync(0xffffffffu, left)) continue;
                    }
                    word = (col < g.gw && k < g.ghw) ? __ldg(g.cellmask + (long long)k * g.gw + col) : 0u;
                    if (g.sub > 1) word &= (0xffffffffu >> (32 - rows)) << (rows * part);
                    pending = __ballot_sync(0xffffffffu, word != 0u);
                    if (pending == 0u) continue;
                }
                if (word != 0u) {
                    W.cell[(head + queued + __popc(pending & ((1u << lane) - 1u))) & 63] =
                        make_uint2((unsigned)col, (unsigned)(32 * k + __ffs(word) - 1));
                    word &= word - 1u;
                }
                queued += __popc(pending);
                pending = __ballot_sync(0xffffffffu, word != 0u);
                __syncwarp();
            }
            if (queued == 0 && grains == 0 && !__any_sync(0xffffffffu, q != 0u)) break;
            step();
        }
        if (DIRECT) {
            if (lane == 0 && taken) {
                atomicAdd(&a.diag[3], (unsigned long long)taken);
                atomicAdd(&a.diag[5], (unsigned long long)taken);
            }
            return;
        }
        __syncthreads();
        if (tid == 0) {
            atomicAdd(&a.diag[3], 1ull);
            atomicAdd(&a.diag[5], 1ull);
        }
        for (int w = tid; w < words; w += nthreads) {
            const unsigned v = bits[w];
            if (v)
                atomicOr(g.bits + ((long long)(fy0 + w / row_words) * a.out_w + fx0) * g.nw + w % row_words, v);
        }
    }
}

// The segments left to the per-sample pass, their samples in parts of `part` (a divisor of 32): each warp takes the
// next part.
template <bool kTwoStep>
__global__ void __launch_bounds__(kPwRegenThreads)
    pixelwise_dense_kernel(const __grid_constant__ PixelwiseArgs a, unsigned int *bits, int nw, int segs, int part,
                           int *__restrict__ next, const int *__restrict__ count, const int *__restrict__ list) {
    __shared__ RegenQueue queues[kPwRegenThreads / 32];
    const int lane = threadIdx.x & 31, parts = (a.n + part - 1) / part;
    const long long n = (long long)*count * parts;
    const UniformF32 U = uniform_f32_new(0.0f, a.delta);
    unsigned long long done = 0;
    CancelPoll poll;
    poll.begin();
    for (;;) {
        int i = -1;
        if (lane == 0 && !poll.requested(a.cancel)) i = atomicAdd(next, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i < 0 || i >= n) break;
        const int seg = list[i / parts], y = seg / segs, x = 32 * (seg % segs) + lane;
        const int k0 = i % parts * part, k1 = min(a.n, k0 + part);
        const bool valid = x < a.out_w;
        pixelwise_pixel_queue<kTwoStep>(a, U, x, y, valid, k0, k1, queues[threadIdx.x >> 5],
                              valid ? bits + ((long long)y * a.out_w + x) * nw : nullptr);
        done += (unsigned long long)min(32, a.out_w - 32 * (seg % segs)) * (unsigned long long)(k1 - k0);
    }
    if (lane == 0 && done) atomicAdd(&a.diag[0], done);
}

}  // namespace fg
