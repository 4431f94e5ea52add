// fg_sg_wgrad.cu -- the surrogate's weight gradients on the fifth-generation tensor cores.
//
//   dW[co][3 ky + kx][ci] += sum over pixels of g[y][x][co] * in[y + ky - 1][x + kx - 1][ci],  db[co] += sum g
//
// Pixels are the reduction dimension.  Both operands lie in shared memory as in global memory, a pixel's
// channels consecutive (TMA, 64- or 32-byte swizzle), which the tensor cores read MN-major: channels along M
// and N, pixels along K.  An MMA multiplies 16 pixels of 128 columns of one row tile:
//   M = 128: the channels of consecutive gradient rows, kRows of them used (with 32 channels the fourth row's
//            slot is not loaded when kRows = 3; what it holds reaches only its own rows of the result);
//   N      : the channels of the kRows + 2 input rows around them, shifted by kx - 1 pixels (a start address).
// The result's block (gradient row, input row) belongs to tap ky = their distance, and is dropped outside
// 0 .. 2.  Three accumulators (kx) stay in tensor memory over a segment of the CTA's rows; the first one
// has 16 more columns, for a constant slot whose channel 0 is one: their sum of g is the bias gradient.
// A CTA (one per SM, three roles: loader, MMA issuer, four warps that read the accumulators) walks a contiguous range
// of row blocks through two or four stages.  At the end of a segment the accumulators are added, rounded to nearest, to
// sums in shared memory, and those at the end onto dW and db with one atomic per element.
// A segment is short because the accumulators' additions cut the sum's low bits off, so that sums of one sign fall
// behind by half a bit per addition: over a CTA's whole share (148 additions on 256 tiles of 64^2) the gradient was
// 2.0e-6 from 64 bits (one sign; 9.2e-7 with both), further than mma.sync's 1.6e-6 (7.7e-7); now 3.7e-7 (3.0e-7).  The
// CTAs' shares grow with the batch, and so did mma.sync's sums, faster than a quarter of a share: hence at most four
// segments.  The loads run on while the accumulators are read.
//
// Measured on 256 tiles of 64^2, 32 -> 32 channels (134 MB, 20 us at the measured copy rate): mma.sync with
// operands staged channel by channel 267 us; this split 63 us; four stages of 64 columns 50 us; the sums
// without shared-memory atomics 45 us; in four segments the same (flushed L2 51.8 us before and after; the output conv's,
// whose gradient rows share warps, 45.7 -> 51.8).  What is left: the input rows, read 5/3 times, and the steps' copies.
//
// Waits are bounded as in fg_sg_tc.cu; a CTA whose wait ran out adds NaN to dW and db.
#include <algorithm>

#include "../../include/film_grain_gb300.h"
#include "fg_internal.h"
#include "fg_sg_tc.cuh"

namespace fg {

constexpr int kWgThreads = 192;  // loader, MMA issuer, four warps that read the accumulators
constexpr int kWgChain = 48;     // MMAs that add to an accumulator in a row, up to kWgSegments segments
constexpr int kWgSegments = 4;

template <int CG, int CX, int PX>  // channels of a gradient pixel (16 or 32) and of an input pixel in shared
struct WgCfg {                     // memory, columns of a row tile (128, or 64 for images no wider)
    static constexpr int kRows = CX == 32 ? 3 : 4;  // gradient rows per step
    static constexpr int kXRows = kRows + 2;
    static constexpr int kGSlots = 128 / CG;
    static constexpr int kGRow = PX * 2 * CG, kXRow = (PX + 8) * 2 * CX;  // bytes of a row slot
    static constexpr int kX = kGSlots * kGRow;                                  // the input rows, then the ones
    static constexpr int kStage = (kX + (kXRows + 1) * kXRow + 1023) / 1024 * 1024;
    static constexpr int kN = kXRows * CX;
    static constexpr int kStages = PX == 64 ? 4 : 2;
    // the CTA's sums: [tap * CX + ci][33] by co, a ky's 16 words further (so that the two gradient rows of a warp
    // meet on different banks), then db
    static constexpr int kSum = 9 * CX * 33 + 32;
    static constexpr int kSumOff = kStages * kStage;
    static constexpr int kBar = kSumOff + (kSum + 32) * 4;
    static constexpr int kSmem = kBar + 16 * kStages + 48;
    static constexpr uint64_t kSwG = CG == 32 ? 4ull : 6ull, kSwX = CX == 32 ? 4ull : 6ull;
    static_assert(3 * kN + 16 <= 512 && kBar % 16 == 0 && kSmem <= 227 * 1024, "sizes");
};

struct WgArgs {
    float *dw, *db;
    int nb, H, W, tiles_x, cout;
    int g_px, x_px;  // pixels of the loaded boxes
    int seg_steps;   // steps of kWgChain MMAs
};

__device__ int g_sg_wg_timeout;

template <int CG, int CX, int PX>
__global__ void __launch_bounds__(kWgThreads, 1) sg_wgrad_tc_kernel(const __grid_constant__ CUtensorMap tm_g,
                                                                    const __grid_constant__ CUtensorMap tm_x,
                                                                    const __grid_constant__ WgArgs a) {
    using C = WgCfg<CG, CX, PX>;
    constexpr int kStages = C::kStages;
    extern __shared__ __align__(1024) unsigned char wg_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(wg_sm);
    const uint32_t full = sbase + C::kBar, freed = full + 8 * kStages, done = freed + 8 * kStages, acc_full = done + 8,
                   acc_free = acc_full + 8, tmem_slot = acc_free + 8;
    volatile int *s_abort = reinterpret_cast<volatile int *>(wg_sm + C::kBar + 16 * kStages + 32);
    float *sum = reinterpret_cast<float *>(wg_sm + C::kSumOff), *sdb = sum + C::kSum;

    if (tid == 0) {
        for (int i = 0; i < kStages; i++) {
            mbar_init(full + 8 * i, 1);
            mbar_init(freed + 8 * i, 1);
        }
        mbar_init(done, 1);
        mbar_init(acc_full, 1);
        mbar_init(acc_free, 4);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int e = tid; e < C::kSum + 32; e += kWgThreads) sum[e] = 0.0f;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tmem_slot), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // the constant slots: channel 0 of every pixel one, in the input rows' swizzle
    for (int e = tid; e < kStages * C::kXRow / 16; e += kWgThreads) {
        const int st = e / (C::kXRow / 16), b = e - st * (C::kXRow / 16);
        constexpr int kCh = CX / 8;
        const int px = b / kCh, c = b - px * kCh;
        // the 16-byte chunk that holds channels 0 .. 7 of this pixel after the swizzle (address bits 4-5 by 7-8,
        // or 4 by 7)
        const int at = CX == 32 ? (px >> 1) & 3 : (px >> 2) & 1;
        *reinterpret_cast<uint4 *>(wg_sm + st * C::kStage + C::kX + C::kXRows * C::kXRow + b * 16) =
            make_uint4(c == at ? 0x3F80u : 0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(wg_sm + C::kBar + 16 * kStages + 24);

    // the CTA's steps [t0, t1): kRows rows of one column tile each, down the columns of all images
    const int per_col = (a.H + C::kRows - 1) / C::kRows;
    const long long total = (long long)a.nb * a.tiles_x * per_col;
    const long long t0 = total * blockIdx.x / gridDim.x, t1 = total * (blockIdx.x + 1) / gridDim.x;
    const int steps = (int)(t1 - t0);
    const int seg_steps = (steps - 1) / min(kWgSegments, (steps - 1) / a.seg_steps + 1) + 1;  // (nearly) equal segments
    const int segs = (steps - 1) / seg_steps + 1;
    bool ok = true;
    int issued = 0;  // the loader's stages, for the wind-down
    if (warp == 0) {
        if (lane == 0) {
            for (long long t = t0; t < t1; t++) {
                const int i = (int)(t - t0), s = i % kStages;
                if (i >= kStages && !mbar_wait(freed + 8 * s, (uint32_t)((i / kStages + 1) & 1), s_abort)) {
                    *s_abort = 1;
                    break;
                }
                const long long col = t / per_col;
                const int y0 = (int)(t - col * per_col) * C::kRows, img = (int)(col / a.tiles_x),
                          x0 = (int)(col - (long long)img * a.tiles_x) * PX;
                mbar_expect_tx(full + 8 * s, (uint32_t)(C::kRows * a.g_px * 2 * CG + C::kXRows * a.x_px * 2 * CX));
                const uint32_t dst = sbase + (uint32_t)(s * C::kStage);
                auto load = [&](const CUtensorMap *tm, uint32_t to, int x, int y) {
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                        "%3, %4, %5}], [%6];\n" ::"r"(to),
                        "l"(reinterpret_cast<uint64_t>(tm)), "r"(0), "r"(x), "r"(y), "r"(img), "r"(full + 8 * s)
                        : "memory");
                };
                for (int r = 0; r < C::kRows; r++) load(&tm_g, dst + r * C::kGRow, x0, y0 + r);
                for (int r = 0; r < C::kXRows; r++) load(&tm_x, dst + C::kX + r * C::kXRow, x0 - 1, y0 - 1 + r);
                issued = i + 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint64_t g0 = tc_desc(sbase, C::kGRow, 16 * CG) | (C::kSwG << 61);
        const uint64_t x0d = tc_desc(sbase + C::kX, C::kXRow, 16 * CX) | (C::kSwX << 61);
        int seg = 0, in_seg = 0;  // segments before this one, its steps so far
        for (long long t = t0; t < t1; t++, in_seg++) {
            const int i = (int)(t - t0), s = i % kStages;
            if (in_seg == seg_steps) {
                tc_commit(acc_full);
                ok = __all_sync(0xffffffffu, mbar_wait(acc_free, (uint32_t)(seg & 1), s_abort));
                if (!ok) {
                    *s_abort = 1;
                    break;
                }
                seg++;
                in_seg = 0;
            }
            ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, (uint32_t)((i / kStages) & 1), s_abort));
            if (!ok) {
                *s_abort = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const long long col = t / per_col;
            const int x0 = (int)(col % a.tiles_x) * PX;
            const int ksteps = (min(PX, a.W - x0) + 15) / 16;  // the gradient is zero past the image's edge
            const uint64_t gd = g0 + (uint64_t)(s * (C::kStage >> 4)), xd = x0d + (uint64_t)(s * (C::kStage >> 4));
            for (int k = 0; k < ksteps; k++) {
#pragma unroll
                for (int kx = 0; kx < 3; kx++) {
                    const uint32_t d = tmem + (uint32_t)(kx == 0 ? 0 : 16 + kx * C::kN);
                    tc_mma(d, gd + (uint64_t)(k * 2 * CG), xd + (uint64_t)(((16 * k + kx) * 2 * CX) >> 4),
                           tc_idesc((uint32_t)(kx == 0 ? C::kN + 16 : C::kN), true), in_seg > 0 || k > 0);
                }
            }
            tc_commit(freed + 8 * s);
        }
        if (ok) tc_commit(acc_full);
        tc_commit(done);
        __syncwarp();
    } else {
        // the segments' results onto the sums, a quarter of the tensor memory (gradient rows) per warp: plain f32
        // additions to shared memory (an atomic would make of each a compare-and-swap loop), the warps at
        // different kx, or at the bias, at a time
        const int quad = warp & 3, m = quad * 32 + lane, gy = m / CG, co = m % CG, gy0 = quad * 32 / CG,
                  gy1 = (quad * 32 + 31) / CG;
        const bool mine = gy < C::kRows && co < a.cout;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16);
        for (int seg = 0; seg < segs; seg++) {
            int stop = mbar_wait(acc_full, (uint32_t)(seg & 1), s_abort) ? 0 : 1;
            // the four warps go on together or not at all
            asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %0, 0;\n barrier.cta.red.or.pred q, 1, 128, p;\n"
                         " selp.s32 %0, 1, 0, q;\n}\n"
                         : "+r"(stop)
                         :
                         : "memory");
            if (stop) {
                *s_abort = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            // every warp reads something in the last turn; after that the next segment may overwrite
            auto release = [&](int turn) {
                if (turn < 3) return;
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_free);
            };
            for (int turn = 0; turn < 4; turn++) {
                const int kx = (quad + turn) & 3;
                if (gy0 < C::kRows && kx < 3) {
                    // the input rows around the warp's gradient rows, all of them before the first is added
                    constexpr int kXr = 128 / CG > 4 ? 4 : 3;
                    uint32_t v[kXr][CX];
#pragma unroll
                    for (int x = 0; x < kXr; x++)
                        tc_load(v[x], base + (uint32_t)((kx == 0 ? 0 : 16 + kx * C::kN) + min(gy0 + x, C::kXRows - 1) * CX));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    release(turn);
#pragma unroll
                    for (int x = 0; x < kXr; x++) {
                        const int ky = gy0 + x - gy;
                        if (mine && ky >= 0 && ky <= 2) {
                            float *to = sum + (3 * ky + kx) * CX * 33 + 16 * ky + co;
#pragma unroll
                            for (int j = 0; j < CX; j++) to[33 * j] += __uint_as_float(v[x][j]);
                        }
                        __syncwarp();  // two gradient rows of a warp add to the same elements in different steps
                    }
                } else if (gy0 < C::kRows) {
                    uint32_t b;
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n"
                                 : "=r"(b)
                                 : "r"(base + (uint32_t)C::kN));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    release(turn);
                    for (int g = gy0; g <= gy1; g++) {
                        if (mine && gy == g) sdb[co] += __uint_as_float(b);
                        __syncwarp();
                    }
                } else {
                    release(turn);  // a quarter without gradient rows
                }
                asm volatile("barrier.cta.sync 1, 128;\n" ::: "memory");
            }
        }
    }
    // ---- the end: one atomic per element
    __syncthreads();
    ok = *s_abort == 0;
    if (!ok) {
        if (tid == 0) {
            atomicExch(&g_sg_wg_timeout, 1);
            const int none = 0;
            for (int i = max(0, issued - kStages); i < issued; i++)
                (void)mbar_wait(full + 8 * (i % kStages), (uint32_t)((i / kStages) & 1), &none);
            (void)mbar_wait(done, 0, &none);
        }
        __syncthreads();
    }
    {
        const float nan = __int_as_float(0x7fc00000);
        for (int e = tid; e < a.cout * 9 * CX; e += kWgThreads) {
            const int co = e / (9 * CX), r = e - co * (9 * CX);
            atomicAdd(&a.dw[e], ok ? sum[r * 33 + 16 * (r / (3 * CX)) + co] : nan);
        }
        if (tid < a.cout) atomicAdd(&a.db[tid], ok ? sdb[tid] : nan);
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
}

template <int CG, int CX, int PX>
static cudaError_t launch_wg_px(const void *g, int g_cstride, const void *x, int x_cstride, WgArgs a, cudaStream_t s) {
    using C = WgCfg<CG, CX, PX>;
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    a.tiles_x = (a.W + PX - 1) / PX;
    a.g_px = std::min(PX, (a.W + 15) & ~15);          // whole K steps (zero past the image's edge)
    a.x_px = std::min(PX + 8, ((a.W + 15) & ~15) + 8);  // with the halo columns, in whole swizzle periods
    a.seg_steps = kWgChain / (a.g_px / 16);
    CUtensorMap tm[2];
    for (int k = 0; k < 2; k++) {
        const cuuint64_t ch = (cuuint64_t)std::min(k ? CX : CG, k ? x_cstride : g_cstride);
        const cuuint64_t px = 2 * (cuuint64_t)(k ? x_cstride : g_cstride);
        const cuuint64_t dims[4] = {ch, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.nb};
        const cuuint64_t strides[3] = {px, (cuuint64_t)a.W * px, (cuuint64_t)a.H * a.W * px};
        const cuuint32_t box[4] = {(cuuint32_t)(k ? CX : CG), (cuuint32_t)(k ? a.x_px : a.g_px), 1, 1};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        if (encode(&tm[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(k ? x : g), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, (k ? CX : CG) == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sg_wgrad_tc_kernel<CG, CX, PX>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
    if (e != cudaSuccess) return e;
    const long long steps = (long long)a.nb * a.tiles_x * ((a.H + C::kRows - 1) / C::kRows);
    sg_wgrad_tc_kernel<CG, CX, PX><<<(unsigned)std::min<long long>(steps, std::max(1, sms)), kWgThreads, C::kSmem, s>>>(
        tm[0], tm[1], a);
    return cudaGetLastError();
}

// Images up to 64 pixels wide: rows of 64 columns in four stages instead of 128 in two, whose copies' latency
// was most of a step (256 tiles of 64^2, 32 -> 32 channels: 63 -> 50 us).
template <int CG, int CX>
static cudaError_t launch_wg(const void *g, int g_cstride, const void *x, int x_cstride, const WgArgs &a, cudaStream_t s) {
    return a.W <= 64 ? launch_wg_px<CG, CX, 64>(g, g_cstride, x, x_cstride, a, s)
                     : launch_wg_px<CG, CX, 128>(g, g_cstride, x, x_cstride, a, s);
}

// The weight gradient of a conv kind (input, residual, output) on the tensor cores, added onto dw and db.
// Returns cudaErrorNotSupported when the buffers are not 16-byte aligned or the tensor maps cannot be made.
cudaError_t launch_sg_wgrad_tc(int kind, const void *g, int g_cstride, const void *x, int x_cstride, float *dw, float *db,
                               int nb, int H, int W, cudaStream_t s) {
    if ((reinterpret_cast<uintptr_t>(g) & 15u) || (reinterpret_cast<uintptr_t>(x) & 15u) || g_cstride % 8 || x_cstride % 8)
        return cudaErrorNotSupported;
    WgArgs a;
    a.dw = dw;
    a.db = db;
    a.nb = nb; a.H = H; a.W = W;
    a.cout = kind == FG_SG_CONV_OUTPUT ? 8 : 32;
    switch (kind) {
    case FG_SG_CONV_INPUT: return launch_wg<32, 16>(g, g_cstride, x, x_cstride, a, s);
    case FG_SG_CONV_RESIDUAL: return launch_wg<32, 32>(g, g_cstride, x, x_cstride, a, s);
    case FG_SG_CONV_OUTPUT: return launch_wg<16, 32>(g, g_cstride, x, x_cstride, a, s);
    default: return cudaErrorNotSupported;
    }
}

// As sg_conv_tc_timeouts, for the weight gradients.
cudaError_t sg_wgrad_tc_timeouts(int *v) {
    const int z = 0;
    cudaError_t e = cudaMemcpyFromSymbol(v, g_sg_wg_timeout, sizeof *v);
    if (e == cudaSuccess && *v) e = cudaMemcpyToSymbol(g_sg_wg_timeout, &z, sizeof z);
    return e;
}

}  // namespace fg
