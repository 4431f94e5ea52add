// fg_grainwise.cuh -- device code of the grain-wise integrator (src/grainwise.rs:12-142), shared by
// the standalone kernel (fg_grainwise.cu) and the batched persistent kernel (fg_batch.cu).
#pragma once
#include <algorithm>

#include "fg_kernels.cuh"
#include "fg_rng.cuh"
#include "fg_color.cuh"

namespace fg {

constexpr int kGwThreads = 512;
constexpr int kGwWarps = kGwThreads / 32;

// The CTA's shared-memory mask covers the output rectangle [rx0, rx0 + rw) x [ry0, ry0 + rh) with the
// `words` mask words of one sample chunk per pixel; bits of other output pixels go straight to the
// global mask.
struct GwTile {
    int rx0, ry0, rw, rh, words, out_w;
    float frx0, fry0, frw, frh;      // the rectangle as floats
    float flast_x, flast_y;          // last output column / row as floats
    unsigned int *gmask;             // the chunk's first word of out_w x out_h x gwords
    int gwords;
    float eps;  // margin of the one-pixel form (gw_splat)
};

// floor / ceil of an f32.  With kSmall (every coordinate within +-2^22) they are one directed-rounding
// add and one exact subtract of 1.5 * 2^23, which stay on the FP32 pipes.
template <bool kSmall>
__device__ __forceinline__ float gw_floor(float v) {
    if (kSmall) return __fsub_rn(__fadd_rd(v, 12582912.0f), 12582912.0f);
    return floorf(v);
}
template <bool kSmall>
__device__ __forceinline__ float gw_ceil(float v) {
    if (kSmall) return __fsub_rn(__fadd_ru(v, 12582912.0f), 12582912.0f);
    return ceilf(v);
}

// bounds(center, radius, limit) (src/grainwise.rs:126-142) as [max(lo, lo_t), min(hi, hi_t)] with
// lo = ceil((c - r) - 0.5), hi = floor((c + r) - 0.5) and [lo_t, hi_t] = [0, limit-1]: the reference
// yields Some iff lo <= hi, lo <= limit-1 and hi >= 0, and then clamps to [0, limit-1], which is
// exactly this interval when it is non-empty.  Coordinates stay below 2^24, so comparing integral
// floats is the reference's i32 comparison.
template <bool kSmall>
__device__ __forceinline__ bool gw_range(float c, float r, float lo_t, float hi_t, float &a, float &b) {
    a = fmaxf(gw_ceil<kSmall>(FG_FSUB(FG_FSUB(c, r), 0.5f)), lo_t);
    b = fminf(gw_floor<kSmall>(FG_FSUB(FG_FADD(c, r), 0.5f)), hi_t);
    return a <= b;
}

// Stage B: the reference's exact bounds() on both axes, then its centre tests and bit sets
// (src/grainwise.rs:69-101) for one (grain, offset) pair: grain (czx, czy, ro) = zoomed centre and
// radius, offset o, sample k of the chunk.  Most pairs have one pixel or none in their bounds, so the loops
// test their end after the body.  Pixels of the tile's rectangle are integers below 2^24, so their index is
// taken in f32.
// A radius below 0.45 (with T.eps, several ulps of the largest coordinate) leaves the nearest pixel alone: any
// other centre is half a pixel away or more.  Where both distances are below the radius by T.eps the bounds
// hold whatever their roundings, and only a pair nearer to its edge computes them.
// 124 x 1024, radius 0.2, N 256 4.51 -> 4.24 ms; 1024^2 -> 2048^2 log-normal 0.05 6.47 -> 6.20 ms.
__device__ __forceinline__ void gw_set(const GwTile &T, unsigned int *mask, float fx, float fy, int k) {
    const float lx = FG_FSUB(fx, T.frx0), ly = FG_FSUB(fy, T.fry0);
    const unsigned bit = 1u << (k & 31);
    if (lx >= 0.0f && lx < T.frw && ly >= 0.0f && ly < T.frh)
        atomicOr(mask + (int)FG_FADD(FG_FMUL(ly, T.frw), lx) * T.words + (k >> 5), bit);
    else
        atomicOr(T.gmask + ((long long)(int)fy * T.out_w + (int)fx) * T.gwords + (k >> 5), bit);
}
template <bool kSmall>
__device__ __forceinline__ void gw_splat(const GwTile &T, unsigned int *mask, float czx, float czy, float ro,
                                         const float2 o, int k) {
    const float tx = FG_FADD(czx, o.x), ty = FG_FADD(czy, o.y);
    float y0, y1, x0, x1;
    if (kSmall && FG_FADD(ro, T.eps) < 0.45f) {
        constexpr float kRint = 12582912.0f;  // 1.5 * 2^23: adding and removing it rounds to an integer
        const float fx = FG_FSUB(FG_FADD(FG_FSUB(tx, 0.5f), kRint), kRint);
        const float fy = FG_FSUB(FG_FADD(FG_FSUB(ty, 0.5f), kRint), kRint);
        const float dx = FG_FSUB(FG_FADD(fx, 0.5f), tx), dy = FG_FSUB(FG_FADD(fy, 0.5f), ty);
        if (!(FG_FADD(FG_FMUL(dx, dx), FG_FMUL(dy, dy)) <= FG_FMUL(ro, ro))) return;
        if (!(fx >= 0.0f && fx <= T.flast_x && fy >= 0.0f && fy <= T.flast_y)) return;
        if (fmaxf(fabsf(dx), fabsf(dy)) > FG_FSUB(ro, T.eps)) {
            if (!(gw_range<kSmall>(ty, ro, 0.0f, T.flast_y, y0, y1) && gw_range<kSmall>(tx, ro, 0.0f, T.flast_x, x0, x1)))
                return;
            if (fx < x0 || fx > x1 || fy < y0 || fy > y1) return;
        }
        gw_set(T, mask, fx, fy, k);
        return;
    }
    const bool in_y = gw_range<kSmall>(ty, ro, 0.0f, T.flast_y, y0, y1);
    const bool in_x = gw_range<kSmall>(tx, ro, 0.0f, T.flast_x, x0, x1);
    if (!(in_x && in_y)) return;
    const float rsq = FG_FMUL(ro, ro);
    for (float fy = y0;;) {
        const float dy = FG_FSUB(FG_FADD(fy, 0.5f), ty);
        const float dysq = FG_FMUL(dy, dy);
        if (dysq <= rsq) {
            for (float fx = x0;;) {
                const float dx = FG_FSUB(FG_FADD(fx, 0.5f), tx);
                if (FG_FADD(FG_FMUL(dx, dx), dysq) <= rsq) gw_set(T, mask, fx, fy, k);
                if (!(fx < x1)) break;
                fx = FG_FADD(fx, 1.0f);
            }
        }
        if (!(fy < y1)) break;
        fy = FG_FADD(fy, 1.0f);
    }
}

// ------------------------------------------------------------------ bitmask candidate filter
// The candidate offsets of a grain are found as a bitmask over the sample index k: the unit interval of
// frac(offset) is cut into 128 buckets, and for each axis a sparse table holds, for every bucket b and
// level L, the OR of the sample masks of buckets b .. b + 2^(L+1) - 1 (cyclic).  The
// cyclic interval [c - h, c + h] of an axis test, rounded out to whole buckets, is the OR of two table
// entries; the AND of the x and y masks is a superset of every pair that can set a bit (a pixel centre
// lies within radius_out of the offset grain centre on both axes), and those pairs go to stage B.
// The masks take kGbMaxWords words at most (256 samples).  More samples are cut into chunks of equal
// width, and a work item renders one chunk of its tile: it draws the grains again (150 to 250 lane-ops
// of the about 1000 a grain costs with its pairs) and keeps the filter, the tables and the tile's
// masks small.  A 311x205 plane at zoom 1.5, N 400, r 0.08: 16.0 ms with one item per tile for all
// samples, listing (grain, offset) pairs from a sorted offset table, 6.4 ms with two chunks of 200 (1.7 ms
// with the rest of this file).
constexpr int kGbBuckets = 128;
constexpr int kGbLevels = 6;     // spans 2 .. 64 buckets (a span of 1 takes 2); 128 or more is the full mask
constexpr int kGbMaxWords = 8;   // samples of a chunk: at most 256

// A warp's pair queue (gw_process): the candidate (grain, sample) pairs of its lanes' grains, taken
// out 32 at a time, and the grains they belong to.  Fewer than 32 pairs stay between steps, so the last
// kGwGrains = 31 + 32 grains pushed (and one) are all that the queue can name.
constexpr int kGwPairs = 256;    // queue entries: grain slot << 8 | sample of the chunk
constexpr int kGwGrains = 64;    // grain slots: zoomed centre and radius
struct GwQueue {
    float gx[kGwGrains], gy[kGwGrains], gr[kGwGrains];
    unsigned short pair[kGwPairs];
};

// Words between consecutive table entries: W rounded up to odd, so that the lanes of a warp reading
// word w of the entries of different buckets b hit different banks ((b * S + w) mod 32 is one-to-one
// in b mod 32 for odd S); with the stride W = 8 they met on 4 banks.
__host__ __device__ inline int gb_entry_stride(int W) { return W | 1; }

// The samples whose frac(offset) lies in the cyclic interval [c - h, c + h] (c in [0, 1)), rounded out
// to whole buckets, written to m (kAnd = false) or ANDed into it (kAnd = true).
template <int MW, bool kAnd>
__device__ __forceinline__ void gb_axis_mask(const unsigned *tab, int W, int S, float c, float h, int n,
                                             unsigned (&m)[MW]) {
    const int blo = __float2int_rd(FG_FMUL(FG_FSUB(c, h), (float)kGbBuckets));
    const int bhi = __float2int_rd(FG_FMUL(FG_FADD(c, h), (float)kGbBuckets));
    const int len = bhi - blo + 1;
    if (h >= 0.5f || len >= kGbBuckets) {
        if (!kAnd) {
#pragma unroll
            for (int w = 0; w < MW; w++) {
                const int rem = n - 32 * w;
                m[w] = rem >= 32 ? 0xFFFFFFFFu : (rem > 0 ? (1u << rem) - 1u : 0u);
            }
        }
        return;
    }
    const int b0 = blo & (kGbBuckets - 1);
    const int L = 30 - __clz(len | 2);  // spans of 2^(L+1) <= len buckets (2 for len = 1)
    const unsigned *e0 = tab + (L * kGbBuckets + b0) * S;
    const unsigned *e1 = tab + (L * kGbBuckets + ((b0 + max(len, 2) - (2 << L)) & (kGbBuckets - 1))) * S;
#pragma unroll
    for (int w = 0; w < MW; w++) {
        const unsigned v = w < W ? (e0[w] | e1[w]) : 0u;
        m[w] = kAnd ? (m[w] & v) : v;
    }
}

// Stage B on queue entries [head, head + 32) of a warp, `n` of them valid.
template <bool kSmall>
__device__ __forceinline__ void gw_process(const GwTile &T, unsigned int *mask, const float2 *offk, const GwQueue &Q,
                                           int head, int n, int lane) {
    if (lane < n) {
        const unsigned e = Q.pair[head + lane];
        const int g = (int)(e >> 8), k = (int)(e & 0xFFu);
        gw_splat<kSmall>(T, mask, Q.gx[g], Q.gy[g], Q.gr[g], offk[k], k);
    }
}

// Chunk `chunk` of the samples over part `part` of `parts` of a tile: every parts-th of its pixels (a heavy
// tile is split over several CTAs, each with its own copy of the tile's masks; OR makes the result the same).  Taken
// in turn, not as ranges, the parts of a tile that is bright on one side cost the same (262 x 1186 blobs, radius 0.047,
// N 113, zoom 0.25: 9.7 ms with ranges, 8.1 so; a plane of few grains a pixel pays for the scattered loads, 256 x 256,
// radius 0.1, N 32 at intensity 0.03 31 -> 36 us).
// Each step of a warp draws one grain per lane.  In a part with enough pixels for the CTA's
// warps a lane has a pixel of its own; in a smaller one g = 2 .. 32 lanes share a pixel, until `fill` lanes have
// one: they hold the same stream, draw its next g grains one after another, and each keeps one (128x96, N 32:
// 0.88 -> 0.39 ms; filling the warps 1.5 or 2 times over instead of once was slower, 6.5 -> 7.0 and 8.0 ms
// on the 1024^2 -> 2048^2 plane, and so was half a filling, 7.1 ms).
// With a constant radius a grain is two draws of the stream, so each lane stands at its own grain and steps over the
// other lanes' without forming their values: half of the repeated draws' instructions, which were a third of all
// on saturated planes (7000 grains a pixel, one pair a grain: 123 x 1024, radius 0.025, N 64 19.4 -> 14.0 ms with the
// above; N 128 23.0 -> 17.1, N 256 27.5 -> 23.2).  A log-normal draw has to be decided to know its length.
// A group whose pixel is done takes the next one once half of the warp's groups wait (the Poisson set-up runs
// for all of them at once), so that pixels of unequal lambda keep the lanes busy.
template <bool kSmall, int MW>
__device__ __forceinline__ void grainwise_tile_bits(const GrainwiseArgs &a, int tile_x, int tile_y,
                                                    unsigned char *smem_raw, int part, int parts, int chunk, int fill) {
    const int k0 = 32 * chunk * a.chunk_words;                 // the chunk's samples: [k0, k0 + n)
    const int n = min(a.n - k0, 32 * a.chunk_words);
    const int W = (n + 31) >> 5;
    float2 *offk = reinterpret_cast<float2 *>(smem_raw);                       // [n] (offx, offy) by k
    const int S = gb_entry_stride(W);
    unsigned *tabx = reinterpret_cast<unsigned *>(offk + ((n + 1) & ~1));     // [levels][buckets][S]
    unsigned *taby = tabx + kGbLevels * kGbBuckets * S;
    unsigned short *bk = reinterpret_cast<unsigned short *>(taby + kGbLevels * kGbBuckets * S);  // [n] buckets
    int *next_px = reinterpret_cast<int *>(bk + ((n + 7) & ~7));               // [4]: the next pixel
    GwQueue *queues = reinterpret_cast<GwQueue *>(next_px + 4);                // [warps]
    unsigned int *mask = reinterpret_cast<unsigned int *>(queues + kGwWarps);
    const int tid = threadIdx.x, lane = tid & 31;
    GwQueue &Q = queues[tid >> 5];

    const int ix0 = tile_x * a.tin_w, iy0 = tile_y * a.tin_h;
    const int ix1 = min(ix0 + a.tin_w, a.in_w), iy1 = min(iy0 + a.tin_h, a.in_h);
    GwTile T;
    T.rx0 = min(a.out_w, (int)floorf((float)ix0 * a.zoom));
    T.ry0 = min(a.out_h, (int)floorf((float)iy0 * a.zoom));
    T.rw = min(a.rmax_w, min(a.out_w, (int)floorf((float)ix1 * a.zoom)) - T.rx0);
    T.rh = min(a.rmax_h, min(a.out_h, (int)floorf((float)iy1 * a.zoom)) - T.ry0);
    T.rw = max(T.rw, 0);
    T.rh = max(T.rh, 0);
    T.frx0 = (float)T.rx0;
    T.fry0 = (float)T.ry0;
    T.frw = (float)T.rw;
    T.frh = (float)T.rh;
    T.words = W;
    T.out_w = a.out_w;
    T.eps = 2.0f * a.frac_eps;  // eight ulps of the largest coordinate and more
    T.flast_x = (float)(a.out_w - 1);
    T.flast_y = (float)(a.out_h - 1);
    T.gmask = a.gmask + chunk * a.chunk_words;
    T.gwords = a.words;
    const int region_words = T.rw * T.rh * W;

    // the chunk's offsets, and each sample's x / y bucket
    for (int k = tid; k < n; k += kGwThreads) {
        const float2 o = a.offs[k0 + k];
        offk[k] = o;
        float fx = FG_FSUB(o.x, floorf(o.x)), fy = FG_FSUB(o.y, floorf(o.y));
        if (!(fx < 1.0f)) fx = 0.0f;  // a tiny negative offset rounds up to 1; cyclically that is 0
        if (!(fy < 1.0f)) fy = 0.0f;
        bk[k] = (unsigned short)((int)FG_FMUL(fx, (float)kGbBuckets) | ((int)FG_FMUL(fy, (float)kGbBuckets) << 8));
    }
    for (int t = tid; t < region_words; t += kGwThreads) mask[t] = 0u;
    const int fw = ix1 - ix0, total = fw * (iy1 - iy0);
    // the part's pixels: of each `parts` of the tile in a row one, where that would be a few of the tile's columns the
    // next one each time
    int gcd = fw, step = parts;
    while (step) {
        const int rest = gcd % step;
        gcd = step;
        step = rest;
    }
    const bool turn = fw < 8 * gcd;
    const int px_end = total / parts + ((turn ? (part + total / parts) % parts : part) < total % parts ? 1 : 0);
    if (tid == 0) *next_px = 0;
    int g = 1;  // lanes per pixel
    while (g < 32 && g * px_end < fill) g *= 2;
    const int sub = lane & (g - 1);
    // level 0: two buckets each
    for (int t = tid; t < kGbBuckets * S; t += kGwThreads) tabx[t] = taby[t] = 0u;
    __syncthreads();
    for (int k = tid; k < n; k += kGwThreads) {
        const int bx = bk[k] & 0xFF, by = bk[k] >> 8, w = k >> 5;
        const unsigned bit = 1u << (k & 31);
        atomicOr(&tabx[bx * S + w], bit);
        atomicOr(&tabx[((bx + kGbBuckets - 1) & (kGbBuckets - 1)) * S + w], bit);
        atomicOr(&taby[by * S + w], bit);
        atomicOr(&taby[((by + kGbBuckets - 1) & (kGbBuckets - 1)) * S + w], bit);
    }
    __syncthreads();
    for (int L = 1; L < kGbLevels; L++) {
        for (int t = tid; t < 2 * kGbBuckets * W; t += kGwThreads) {
            const int axis = t / (kGbBuckets * W), r = t - axis * kGbBuckets * W;
            const int b = r / W, w = r - b * W;
            unsigned *tb = axis ? taby : tabx;
            const int b2 = (b + (1 << L)) & (kGbBuckets - 1);
            tb[(L * kGbBuckets + b) * S + w] = tb[((L - 1) * kGbBuckets + b) * S + w] |
                                               tb[((L - 1) * kGbBuckets + b2) * S + w];
        }
        __syncthreads();
    }

    const UniformF32 U = uniform_f32_new(0.0f, 1.0f);
    const float zoom = a.zoom;
    uint32_t left = 0;  // grains of this group's pixel still to draw
    int px = 0, py = 0;
    Xoshiro rng = {0, 0, 0, 0};
    bool more = true;   // the part may still have pixels (warp-uniform)
    int qn = 0;         // pairs in the warp's queue (below 32 between steps)
    int gn = 0;         // grains pushed so far
    for (;;) {
        const unsigned busy = __ballot_sync(0xffffffffu, left > 0);
        if (more && __popc(busy) <= 16) {
            const unsigned idle = ~busy;
            const int want = __popc(idle) / g;  // groups without a pixel
            int base = 0;
            if (lane == 0) base = atomicAdd(next_px, want);
            base = __shfl_sync(0xffffffffu, base, 0);
            more = base + want < px_end;
            const int pi = base + __popc(idle & ((1u << (lane & ~(g - 1))) - 1u)) / g;
            if (((idle >> lane) & 1u) && pi < px_end) {
                const int ti = pi * parts + (turn ? (part + pi) % parts : part);
                px = ix0 + ti % fw;
                py = iy0 + ti / fw;
                const float lv = a.lam[(long long)py * a.in_w + px];
                if (lv > 0.0f) left = poisson_count(mix3(a.seed, kPixelStream, px, py), lv, rng);
                if (!a.lognorm)  // to the lane's own grain
                    for (int t = 0; t < 2 * sub; t++) rng.next();
            }
            continue;
        }
        if (busy == 0u) break;
        {
            // the group's next g grains, one kept by each lane
            bool have = false;
            float ux = 0.0f, uy = 0.0f;
            RadiusDraw rd = {0ull, -1.0f};
            if (!a.lognorm) {
                have = (uint32_t)sub < left;
                ux = uniform_f32_from(U, rng.next());
                uy = uniform_f32_from(U, rng.next());
                for (int t = 1; t < g; t++) {
                    rng.next();
                    rng.next();
                }
                left = left > (uint32_t)g ? left - (uint32_t)g : 0u;
            } else {
                for (int t = 0; t < g; t++) {
                    if (left > 0) {
                        left--;
                        const float vx = uniform_f32_from(U, rng.next()), vy = uniform_f32_from(U, rng.next());
                        const RadiusDraw vd = lognormal_draw(a.log_mu, a.log_sigma, rng);
                        if (t == sub) {
                            have = true;
                            ux = vx;
                            uy = vy;
                            rd = vd;
                        }
                    }
                }
            }
            // its candidate samples as a bitmask
            unsigned m[MW];
#pragma unroll
            for (int w = 0; w < MW; w++) m[w] = 0u;
            int cnt = 0;
            float gx = 0.0f, gy = 0.0f, gr = 0.0f;  // this lane's grain: zoomed centre, zoomed radius
            if (have) {
                const float cx = FG_FADD((float)px, ux), cy = FG_FADD((float)py, uy);
                float r = a.lognorm ? lognormal_radius(rd, a.log_mu, a.log_sigma) : a.radius_mean;
                if (r > a.rm) r = a.rm;
                if (r > 0.0f) {
                    const float ro = FG_FMUL(r, zoom);
                    if (ro > 0.0f) {
                        const float czx = FG_FMUL(cx, zoom), czy = FG_FMUL(cy, zoom);
                        float cyf = FG_FSUB(0.5f, FG_FSUB(czy, floorf(czy)));  // frac(1/2 - czy)
                        if (cyf < 0.0f) cyf = FG_FADD(cyf, 1.0f);
                        float cxf = FG_FSUB(0.5f, FG_FSUB(czx, floorf(czx)));  // frac(1/2 - czx)
                        if (cxf < 0.0f) cxf = FG_FADD(cxf, 1.0f);
                        gx = czx;
                        gy = czy;
                        gr = ro;
                        const float h = FG_FADD(ro, a.frac_eps);
                        gb_axis_mask<MW, false>(tabx, W, S, cxf, h, n, m);
                        gb_axis_mask<MW, true>(taby, W, S, cyf, h, n, m);
#pragma unroll
                        for (int w = 0; w < MW; w++) cnt += __popc(m[w]);
                    }
                }
            }
            // this step's (grain, sample) pairs go to the warp's queue, each lane's at its prefix of the counts,
            // and leave it 32 at a time (every lane busy), the last few staying for the next step
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int tot = __shfl_sync(0xffffffffu, incl, 31);
            if (tot == 0) continue;
            const unsigned with = __ballot_sync(0xffffffffu, cnt > 0);
            const int slot = (gn + __popc(with & ((1u << lane) - 1u))) & (kGwGrains - 1);
            gn += __popc(with);
            if (cnt > 0) {
                Q.gx[slot] = gx;
                Q.gy[slot] = gy;
                Q.gr[slot] = gr;
            }
            for (int done = 0; done < tot;) {
                // the lanes whose pairs still fit, in lane order
                const unsigned fit = __ballot_sync(0xffffffffu, incl - done <= kGwPairs - qn);
                const int upto = fit ? __shfl_sync(0xffffffffu, incl, 31 - __clz(fit)) : 0;
                if (upto <= done) {
                    // one lane's pairs alone overflow the queue (grains that reach most samples): the lanes
                    // take their own pairs, which are about as many on each.  The queue is emptied too: its
                    // pairs would outlive their grains' slots.
                    gw_process<kSmall>(T, mask, offk, Q, 0, qn, lane);
                    qn = 0;
                    __syncwarp();
                    const bool mine = incl - cnt >= done;
#pragma unroll
                    for (int w = 0; w < MW; w++) {
                        unsigned v = mine ? m[w] : 0u;
                        while (v) {
                            const int k = 32 * w + __ffs(v) - 1;
                            v &= v - 1u;
                            gw_splat<kSmall>(T, mask, gx, gy, gr, offk[k], k);
                        }
                    }
                    break;
                }
                if (cnt > 0 && incl - cnt >= done && incl <= upto) {
                    unsigned short *q = Q.pair + qn + (incl - cnt - done);
#pragma unroll
                    for (int w = 0; w < MW; w++) {
                        unsigned v = m[w];
                        while (v) {
                            *q++ = (unsigned short)((slot << 8) | (32 * w + __ffs(v) - 1));
                            v &= v - 1u;
                        }
                    }
                }
                qn += upto - done;
                done = upto;
                __syncwarp();
                int head = 0;
                for (; head + 32 <= qn; head += 32) gw_process<kSmall>(T, mask, offk, Q, head, 32, lane);
                if (head > 0) {  // the rest moves to the front
                    const unsigned short e = Q.pair[head + lane < qn ? head + lane : head - 1];
                    __syncwarp();
                    if (head + lane < qn) Q.pair[lane] = e;
                    qn -= head;
                    __syncwarp();
                }
            }
        }
    }
    gw_process<kSmall>(T, mask, offk, Q, 0, qn, lane);
    __syncthreads();

    // OR the rectangle's words into the global mask (other CTAs' spills land there too).
    for (int t = tid; t < region_words; t += kGwThreads) {
        const unsigned v = mask[t];
        if (v) {
            const int w = t % W, px = t / W;
            const int lx = px % T.rw, ly = px / T.rw;
            atomicOr(T.gmask + ((long long)(T.ry0 + ly) * a.out_w + (T.rx0 + lx)) * a.words + w, v);
        }
    }
}

// Shared-memory bytes of one grain-wise tile.
inline size_t grainwise_tile_smem_bytes(const GrainwiseArgs &a) {
    const size_t W = (size_t)a.chunk_words, n = std::min<size_t>((size_t)a.n, 32 * W);
    return ((n + 1) & ~(size_t)1) * sizeof(float2) +
           2 * (size_t)kGbLevels * kGbBuckets * gb_entry_stride((int)W) * sizeof(unsigned) +
           ((n + 7) & ~(size_t)7) * sizeof(unsigned short) + 4 * sizeof(int) + kGwWarps * sizeof(GwQueue) +
           (size_t)a.rmax_w * a.rmax_h * W * sizeof(unsigned int);
}

// The most CTAs a tile of `px` pixels is split over: one pixel for each warp.
inline int grainwise_most_parts(int px) { return std::max(1, std::min(px / kGwWarps, 0x7FFF)); }

// How tiles are cut into items: a tile of `cost` lane-ops into parts of at most `target` of them, the cost an item
// has when every CTA slot gets kGwItemsPerSlot.  Without the cut, the saturated spots of a blob
// plane (3 % of the pixels, half of the grains) held the kernel to the end: 1024^2 -> 2048^2, N 128, the
// heaviest tile ran 14.7 ms while the CTAs were done in 6.6 ms on average; finer cuts than two items per slot
// repeat the items' set-up and share pixels among more lanes (3 or 4 per slot: 6.5 -> 7.2, 8.0 ms).  A part has no less
// than kGwItemFloor lane-ops (an item's set-up, about 10 us of a CTA) and a pixel per warp.
// Rounding the parts up makes more items than the slots take in kGwItemsPerSlot turns, and where most of them cost the
// same (a plane that is mostly saturated) the few left over take a whole turn more.  So the target is the smallest of
// kGwStretches times that cost at which the items fit, an item taking the share of its slot that as many of its
// size as fit into the slot leave it: 1024 x 123, radius 0.025, N 256 25.3 -> 21.5 ms.  (Stretched further, up to 1.45,
// fewer and larger parts left slots idle: 153 x 771, radius 0.066, N 233, zoom 2 8.5 -> 10.8.)
constexpr int kGwItemsPerSlot = 2;
constexpr float kGwItemFloor = 2.0e6f;
constexpr float kGwPixelCost = 800.0f;  // a pixel's Poisson set-up, in lane-ops (two grain steps)
constexpr int kGwStretches = 4;
__host__ __device__ inline float gw_stretch(int k) { return k == 0 ? 1.0f : k == 1 ? 1.02f : k == 2 ? 1.05f : 1.09f; }
__host__ __device__ inline int gw_parts(float cost, float target, int most_parts) {
    const float p = fminf(ceilf(cost / target), (float)most_parts);
    return p > 1.0f ? (int)p : 1;
}
// A tile whose pixels hold about the same (many) grains: each lane group's first pixel takes as long as every other's,
// so a part whose groups do not fit the CTA's lanes at once, or leave many of them out, wastes them to its end.  Its
// parts are sized for that (gw_even_parts: about as many, up to twice, by the share of the lanes that work) and its
// groups as large as fit at once.
__host__ __device__ inline bool gw_even(float lam_sum, float lam_max, int px) {
    return lam_sum >= 0.75f * lam_max * (float)px && lam_sum >= 50.0f * (float)px;
}
constexpr int kGwEvenFill = kGwThreads / 2 + 1;  // grainwise_tile_bits' fill: the most lanes that are no more than all
__host__ __device__ inline int gw_even_parts(float cost, float target, int most_parts, int px, bool lognorm) {
    int best = gw_parts(cost, target, most_parts);
    if (best == 1) return 1;
    const int lo = gw_parts(cost, 1.25f * target, most_parts), hi = best * 2 < most_parts ? best * 2 : most_parts;
    float best_score = 0.0f;
    const int first = best;
    for (int k = -1; k <= 5; k++) {  // as cut by cost, and filled by groups of 1 .. 32
        const int parts = k < 0 ? first : (int)((((long long)px << k) + kGwThreads - 1) / kGwThreads);
        if (parts < lo || parts > hi) continue;
        const int n = (px + parts - 1) / parts;
        int g = 1;
        while (g < 32 && 2 * g * n <= kGwThreads) g *= 2;
        const int rounds = (n * g + kGwThreads - 1) / kGwThreads;
        const float repeated = (lognorm ? 0.12f : 0.04f) * (float)(g - 1);  // the draws that g lanes repeat
        const float score = (float)n * (float)g / ((float)rounds * (float)kGwThreads) / (1.0f + repeated);
        if (score > 1.02f * best_score) {
            best_score = score;
            best = parts;
        }
    }
    return best;
}
__host__ __device__ inline float gw_slot_share(float cost, float target, int parts) {
    const float fit = floorf((float)kGwItemsPerSlot * target * (float)parts / fmaxf(cost, 1.0f));
    return (float)parts / fmaxf(fit, 1.0f);
}

// The tile variant for chunks of `words` mask words: the words a grain's candidate mask holds in registers.
__host__ __device__ inline int grainwise_variant(int words) {
    return words <= 1 ? 1 : words <= 2 ? 2 : words <= 4 ? 4 : kGbMaxWords;
}

// One input tile of the grain-wise kernel (all threads of the CTA; `smem_raw` holds its shared memory).
// kVariant: grainwise_variant(a.chunk_words), or -1 to dispatch at run time (the batched kernel).
template <bool kSmall, int kVariant = -1>
__device__ __forceinline__ void grainwise_tile(const GrainwiseArgs &a, int tile_x, int tile_y,
                                               unsigned char *smem_raw, int part, int parts, int chunk,
                                               int fill = kGwThreads) {
    if (kVariant > 0)
        grainwise_tile_bits<kSmall, kVariant < 0 ? 1 : kVariant>(a, tile_x, tile_y, smem_raw, part, parts, chunk, fill);
    else if (kSmall && a.chunk_words <= 2)
        grainwise_tile_bits<kSmall, 2>(a, tile_x, tile_y, smem_raw, part, parts, chunk, fill);
    else grainwise_tile_bits<kSmall, kGbMaxWords>(a, tile_x, tile_y, smem_raw, part, parts, chunk, fill);
}

}  // namespace fg
