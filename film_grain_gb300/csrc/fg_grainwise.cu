// fg_grainwise.cu -- the grain-wise integrator (src/grainwise.rs:12-142) for sm_103a.
//
// The reference walks input pixels, draws Poisson(lambda) grains from each pixel's stream, and for
// every grain and offset k ORs bit k into the 64-bit sample masks of the output pixels whose centres
// fall in the offset disk (AtomicU64::fetch_or), then popcounts the masks.  Here a work item is a tile of
// input pixels, or a part of one, and a chunk of the samples; its CTA keeps the sample masks (ceil(N/32) words per
// pixel) of the output rectangle that the tile maps to in shared memory, draws the tile's grains, rasterises them
// with the reference's exact bounds() and centre test, and ORs the masks into the plane's; bits that fall outside
// the rectangle go to the plane's masks at once (so tiles never exchange grains).  The popcount * (1/N) epilogue is
// optionally fused with the luma colour recombination and u8 packing.
//
// Work organisation:
//   - persistent CTAs pull the items, heaviest tiles first (grainwise_order_kernel);
//   - the lanes of a warp take one grain each a step, of a pixel of their own or of one that a group of lanes shares
//     (fg_grainwise.cuh);
//   - an offset can put a pixel centre inside a grain's disk only if frac(czx + offx) lies within
//     radius_out of 1/2 (and likewise for y).  Each lane turns both tests, widened by a rounding margin
//     and rounded out to 1/128 buckets, into a bitmask over the sample index (two lookups per axis in
//     per-tile sparse OR tables), ANDs them, and the set bits -- about 1.2x the true candidates -- go to the
//     warp's queue, from which 32 pairs at a time get stage B: the reference's exact bounds() and centre tests,
//     one pair per lane.  Above 256 samples a work item takes one chunk of them;
//   - the lognormal radius is evaluated with the double-float exp (exp_f64_to_f32).
// Bits are set with shared-memory atomicOr; OR is idempotent and commutative, so the result does not
// depend on the order.
#include "fg_kernels.cuh"
#include "fg_rng.cuh"
#include "fg_color.cuh"
#include "fg_grainwise.cuh"
#include "fg_internal.h"

#include <algorithm>

namespace fg {

// Persistent form: CTAs pull work items (tile, part of it, sample chunk) through the counter a.work[0] from
// the scheduler's list until it is exhausted.
template <bool kSmall, int kVariant>
__global__ void __launch_bounds__(kGwThreads, 2) grainwise_persistent_kernel(const __grid_constant__ GrainwiseArgs a,
                                                                             int ntx) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item;
    const int nitems = a.work[1] * a.chunks;
    const int2 *items = reinterpret_cast<const int2 *>(a.work + 2);
    for (;;) {
        if (threadIdx.x == 0) {
            const int i = atomicAdd(a.work, 1);  // chunk i % chunks of the (i / chunks)-th listed part
            s_item = (i < nitems && !cancel_requested(a.cancel)) ? i : -1;
        }
        __syncthreads();
        const int i = s_item;
        if (i < 0) break;
        const int2 it = items[i / a.chunks];  // (tile, part | even << 15 | parts << 16)
        grainwise_tile<kSmall, kVariant>(a, it.x % ntx, it.x / ntx, smem_raw, it.y & 0x7FFF, it.y >> 16, i % a.chunks,
                                         (it.y & 0x8000) ? kGwEvenFill : kGwThreads);
        __syncthreads();
    }
}

// Expected lane-ops of each input tile and sample chunk (one warp per tile): its grains (sum of lambda) and
// its pixels' Poisson set-up.
__global__ void grainwise_costs_kernel(const float *__restrict__ lam, int in_w, int in_h, int tin_w, int tin_h, int ntx,
                                       int ntiles, float grain_cost, float *__restrict__ cost) {
    const int tile = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (tile >= ntiles) return;
    const int x0 = (tile % ntx) * tin_w, y0 = (tile / ntx) * tin_h;
    const int w = min(x0 + tin_w, in_w) - x0, n = w * (min(y0 + tin_h, in_h) - y0);
    float sum = 0.0f, most = 0.0f;
    // (clamped: the work list's bound needs finite costs, whatever plane the caller passes)
    for (int i = lane; i < n; i += 32) {
        const float l = fminf(fmaxf(lam[(long long)(y0 + i / w) * in_w + x0 + i % w], 0.0f), 1.0e6f);
        sum += l;
        most = fmaxf(most, l);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    }
    // the cost's last bit: the tile is even
    if (lane == 0)
        cost[tile] = __uint_as_float((__float_as_uint(grain_cost * sum + kGwPixelCost * (float)n) & ~1u) |
                                     (gw_even(sum, most, n) ? 1u : 0u));
}

// The work list: tiles by descending cost (a bitonic sort in shared memory, one CTA, for up to kGwSortMax
// tiles; larger grids keep the natural order), each cut into parts (gw_parts).
// work[1] = items, then int2 (tile, part | even << 15 | parts << 16).
constexpr int kGwSortMax = 4096;
__global__ void __launch_bounds__(1024) grainwise_order_kernel(const __grid_constant__ GrainwiseArgs a,
                                                               const float *__restrict__ cost, int ntx, int ntiles,
                                                               int slots, int most_parts) {
    int *work = a.work;
    const int chunks = a.chunks;
    auto cut = [&](float c, int tile, float target) {
        if (!(__float_as_uint(c) & 1u)) return gw_parts(c, target, most_parts);
        const int w = min(a.tin_w, a.in_w - tile % ntx * a.tin_w), h = min(a.tin_h, a.in_h - tile / ntx * a.tin_h);
        return gw_even_parts(c, target, most_parts, w * h, a.lognorm != 0);
    };
    __shared__ float key[kGwSortMax];
    __shared__ int idx[kGwSortMax];
    __shared__ float wsum[32];
    __shared__ float wshare[kGwStretches][32];
    __shared__ int wcnt[33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool sorted = ntiles <= kGwSortMax;
    float sum = 0.0f;
    for (int i = tid; i < ntiles; i += blockDim.x) sum += cost[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) wsum[warp] = sum;
    if (sorted) {
        int n2 = 2;
        while (n2 < ntiles) n2 <<= 1;
        for (int i = tid; i < n2; i += blockDim.x) {
            key[i] = i < ntiles ? cost[i] : -1.0f;  // costs are >= 0: the padding sorts last
            idx[i] = i;
        }
        __syncthreads();
        for (int k = 2; k <= n2; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = tid; i < n2; i += blockDim.x) {
                    const int ixj = i ^ j;
                    if (ixj > i) {
                        const bool desc = (i & k) == 0;
                        if ((key[i] < key[ixj]) == desc) {
                            const float tk = key[i];
                            key[i] = key[ixj];
                            key[ixj] = tk;
                            const int ti = idx[i];
                            idx[i] = idx[ixj];
                            idx[ixj] = ti;
                        }
                    }
                }
                __syncthreads();
            }
        }
    }
    __syncthreads();
    float total = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) total += wsum[w];
    float target = fmaxf(kGwItemFloor, total * (float)chunks / (float)(slots * kGwItemsPerSlot));
    if (target > kGwItemFloor) {  // (else the items are fewer than the slots' turns)
        float share[kGwStretches];
#pragma unroll
        for (int k = 0; k < kGwStretches; k++) share[k] = 0.0f;
        for (int i = tid; i < ntiles; i += blockDim.x)
#pragma unroll
            for (int k = 0; k < kGwStretches; k++) {
                const float t = target * gw_stretch(k);
                share[k] += gw_slot_share(cost[i], t, cut(cost[i], i, t));
            }
#pragma unroll
        for (int k = 0; k < kGwStretches; k++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) share[k] += __shfl_xor_sync(0xffffffffu, share[k], o);
            if (lane == 0) wshare[k][warp] = share[k];
        }
        __syncthreads();
        int fits = 0;
        for (int k = kGwStretches - 1; k >= 0; k--) {
            float sum_k = 0.0f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) sum_k += wshare[k][w];
            if (sum_k * (float)chunks <= (float)slots) fits = k;
        }
        target *= gw_stretch(fits);
    }
    int2 *items = reinterpret_cast<int2 *>(work + 2);
    int base = 0;  // items of the tiles before this round's
    for (int i0 = 0; i0 < ntiles; i0 += blockDim.x) {
        const int i = i0 + tid;
        int tile = 0, parts = 0, even = 0;
        if (i < ntiles) {
            tile = sorted ? idx[i] : i;
            const float c = sorted ? key[i] : cost[i];
            parts = cut(c, tile, target);
            even = (__float_as_uint(c) & 1u) << 15;
        }
        int incl = parts;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wcnt[warp] = incl;
        __syncthreads();
        int first = base + incl - parts, round = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            if (w < warp) first += wcnt[w];
            round += wcnt[w];
        }
        for (int q = 0; q < parts; q++) items[first + q] = make_int2(tile, q | even | (parts << 16));
        base += round;
        __syncthreads();
    }
    if (tid == 0) {
        work[0] = 0;
        work[1] = base;
    }
}

// popcount * (1/N) of the sample masks (src/grainwise.rs:114-122), fused with the colour output:
// mode 0 values only, 1 luma recombination + u8 (src/color.rs:75-96), 2 u8 pack of three planes
// whose masks are consecutive (src/color.rs:101-113).
__global__ void grainwise_epilogue_kernel(const GrainwiseEpilogueArgs a) {
    const long long n = (long long)a.out_w * a.out_h;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float inv_samples = FG_FDIV(1.0f, (float)(a.n > 0 ? a.n : 1));
    float v[3];
    const int planes = a.mode == 2 ? 3 : 1;
    for (int c = 0; c < planes; c++) {
        const unsigned int *m = a.gmask + ((long long)c * n + i) * a.words;
        unsigned cnt = 0;
        for (int w = 0; w < a.words; w++) cnt += __popc(m[w]);
        v[c] = FG_FMUL((float)cnt, inv_samples);
        if (a.out) a.out[(long long)c * n + i] = v[c];
    }
    if (!a.out_rgb8) return;
    unsigned char *o = a.out_rgb8 + 3 * i;
    if (a.mode == 1) {
        const int ox = (int)(i % a.out_w), oy = (int)(i / a.out_w);
        float cbv, crv;
        if (a.in_w == a.out_w && a.in_h == a.out_h) {
            cbv = a.cb[i];
            crv = a.cr[i];
        } else {
            const float sxs = FG_FDIV((float)a.in_w, (float)a.out_w), sys = FG_FDIV((float)a.in_h, (float)a.out_h);
            const long long src = (long long)nearest_src(oy, sys, a.in_h) * a.in_w + nearest_src(ox, sxs, a.in_w);
            cbv = a.cb[src];
            crv = a.cr[src];
        }
        luma_rgb8(v[0], cbv, crv, o);
    } else if (a.mode == 2) {
        o[0] = to_u8(v[0]);
        o[1] = to_u8(v[1]);
        o[2] = to_u8(v[2]);
    }
}

size_t grainwise_smem_bytes(const GrainwiseArgs &a) { return grainwise_tile_smem_bytes(a); }

// The directed-rounding floor/ceil needs every bounds() argument within +-2^22.
bool grainwise_small_coords(const GrainwiseArgs &a) {
    const float span = (float)max(a.out_w, a.out_h) +
                       fmaxf(fmaxf(-a.offx_min, a.offx_max), fmaxf(-a.offy_min, a.offy_max)) + a.rm * a.zoom + 4.0f;
    return span < 4194304.0f;
}

int grainwise_tile_count(const GrainwiseArgs &a) {
    return ((a.in_w + a.tin_w - 1) / a.tin_w) * ((a.in_h + a.tin_h - 1) / a.tin_h);
}

// The scheduler's area: item counter, items, then the list -- every tile's share above the first is a target's
// worth of lane-ops, so there are at most slots * kGwItemsPerSlot of those (twice as many items, of even tiles) -- and
// the tiles' costs.
static size_t grainwise_list_items(const GrainwiseArgs &a, int sms) {
    return 2 * ((size_t)grainwise_tile_count(a) + (size_t)2 * sms * kGwItemsPerSlot + 1);
}
size_t grainwise_work_ints(const GrainwiseArgs &a, int sms) {
    return 2 + 2 * grainwise_list_items(a, sms) + (size_t)grainwise_tile_count(a);
}

cudaError_t launch_grainwise(const GrainwiseArgs &a, int sms, cudaStream_t s) {
    const size_t smem = grainwise_smem_bytes(a);
    const int ntx = (a.in_w + a.tin_w - 1) / a.tin_w, nty = (a.in_h + a.tin_h - 1) / a.tin_h;
    if (ntx <= 0 || nty <= 0) return cudaSuccess;
    const bool small = grainwise_small_coords(a);
    const int v = grainwise_variant(a.chunk_words);
    // tile scheduler: costs from lambda, heaviest first, persistent CTAs
    const int ntiles = ntx * nty, slots = 2 * sms;
    float *cost = reinterpret_cast<float *>(a.work + 2 + 2 * grainwise_list_items(a, sms));
    grainwise_costs_kernel<<<(ntiles + 7) / 8, 256, 0, s>>>(a.lam, a.in_w, a.in_h, a.tin_w, a.tin_h, ntx, ntiles,
                                                            a.grain_cost, cost);
    grainwise_order_kernel<<<1, 1024, 0, s>>>(a, cost, ntx, ntiles, slots, grainwise_most_parts(a.tin_w * a.tin_h));
    void (*k)(GrainwiseArgs, int);
    if (!small) k = grainwise_persistent_kernel<false, kGbMaxWords>;  // coordinates beyond 2^22: one variant
    else if (v == 1) k = grainwise_persistent_kernel<true, 1>;
    else if (v == 2) k = grainwise_persistent_kernel<true, 2>;
    else if (v == 4) k = grainwise_persistent_kernel<true, 4>;
    else k = grainwise_persistent_kernel<true, kGbMaxWords>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kGwThreads, smem);
    if (e != cudaSuccess) return e;
    k<<<sms * std::max(1, per_sm), kGwThreads, smem, s>>>(a, ntx);
    return cudaGetLastError();
}

cudaError_t launch_grainwise_epilogue(const GrainwiseEpilogueArgs &a, cudaStream_t s) {
    const long long n = (long long)a.out_w * a.out_h;
    if (n <= 0) return cudaSuccess;
    grainwise_epilogue_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace fg
