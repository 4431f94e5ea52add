// fg_sg_tc.cu -- the surrogate's convs on the fifth-generation tensor cores.
//
// NHWC bf16 activations, weights [cout][tap 9][cin] bf16, f32 accumulation (channels in -> out):
//   input          16 -> 32  out = relu(conv3x3(in) + b)
//   residual       32 -> 32  out = in + relu(conv3x3(in) + b)      (aux, for training: the ReLU output)
//   output         32 -> 1   f32 out = u + conv3x3(in) + b
//   data gradient  32 -> 32  out = res + conv3x3(in)               (masked, a second output: out where the
//                  16 -> 32  out = conv3x3(in)                      layer's ReLU output is positive, else 0)
//
// Taking the 32 -> 32 conv (the others differ in their channel counts):
// An implicit GEMM over row tiles of M = 128 pixels.  An input row y contributes to the output rows y + 1, y
// and y - 1 (taps ky = 0, 1, 2), so the three taps' weights stand side by side as one B operand of
// N = 96 columns, ordered ky = 2, 1, 0, and the accumulators of consecutive output rows stand side by side in
// tensor memory in the same order: one tcgen05.mma adds an input row's share to all three rows.  Per row that
// is 3 kx x 2 k-halves = 6 MMAs (M 128, N 96, K 16) instead of 18 of N 32, and the A operand -- what a
// narrow N makes the shared memory deliver over and over, 4 KB per MMA at 128 B per clock against 16 clocks
// of arithmetic -- is read 6 times instead of 18.  An output row's sum still runs over ky, kx, k in that
// order, so its bits do not change.  The first MMA of a new output row runs apart (it overwrites), and a
// window that wraps around the ring of 8 accumulator rows is issued in two pieces.
//
// A CTA (two per SM) walks a contiguous range of all images' row tiles, column by column, so that every CTA
// has the same number of rows and the two halo rows of a range cost little.  Ten warps: one loads input rows
// by TMA into a ring of 6, one issues the MMAs, two groups of four run the epilogue from tensor memory (warp
// quarter q: pixels 32q .. 32q + 31, one pixel's 32 channels per thread).  Rows lie in shared memory as in
// global memory, 64 bytes per pixel, under the 64-byte swizzle: the tensor cores read them K-major (8-pixel
// groups 512 bytes apart), a tap kx is a start address kx pixels in, and the k-half 32 bytes in; the
// swizzle goes by address bits, so it holds for any start.  Outputs are staged in the same swizzle (eight
// neighbouring threads write eight bank groups) and leave by TMA, which also cuts them at the image's edge;
// written directly, a thread's own 64 bytes would touch each 32-byte sector twice.
//
// Images narrower than a row tile's half share row tiles (tc_narrow): a tile's input is then the rows of two or more
// images with their halo pixels, side by side as TMA lays them, read from wherever the tile begins; the
// epilogue finds each position's pixel and stores it by plain stores, as a warp's pixels lie in several images.
//
// Measured, 32 -> 32 at 3 x 1024^2 pixels (403 MB, 60 us at the measured copy rate): 18 MMAs of N 32 per row
// 128 us; this split with one epilogue group and rows as 16-byte TMA pieces 95 us; two groups 92 us; the MMAs
// issued by a converged warp 78 us; with constant operands inside a run 72 us (call by call 139 -> 76 us).
// 720p, 3 planes, a layer 122 -> 62 us, the input conv 90 -> 45 us, the output conv 106 -> 50 us (both on mma.sync
// before).  What is left: the MMA warp's own instructions (a row's 8.5 MMAs with the overwriting and wrapping
// ones are issued in about 900 of its 1590 cycles) and shared-memory traffic.
//
// Every wait on an mbarrier is bounded; a wait that runs out records the fact in g_sg_tc_timeout, writes NaN
// outputs for the CTA's rows not yet written, waits (bounded) for its own copies and MMAs, frees its tensor
// memory and returns.
#include <algorithm>
#include <type_traits>

#include "../../include/film_grain_gb300.h"
#include "fg_internal.h"
#include "fg_sg_tc.cuh"

namespace fg {

constexpr int kTcPx = 128;          // output pixels of one row tile (the MMA's M)
constexpr int kTcHalo = kTcPx + 2;  // input pixels of one row at most
constexpr int kTcNarrowPx = 208;    // input pixels of a row tile of narrow images at most
constexpr int kTcAcc = 8;           // accumulator rows in tensor memory
constexpr int kTcStageBytes = 2048; // a warp's 32 pixels of 32 channels
constexpr int kTcThreads = 320;     // loader, MMA issuer, two groups of four epilogue warps
__device__ int g_sg_tc_timeout;

enum TcMode { kTcInput, kTcResidual, kTcResidualAux, kTcOutput, kTcDgrad, kTcDgradMasked, kTcLinear, kTcLinearMasked };

// Sizes of a mode.  A row slot holds kTcHalo pixels, rounded up to what the swizzle repeats over (8 pixels), or
// the rows of several narrow images.
template <int MODE, bool NARROW>
struct TcCfg {
    static constexpr int kSlots = NARROW ? 4 : 6;  // input rows in flight
    // barriers: rows full, rows free (MMA), rows free (epilogue), accumulators full, accumulators free, drain
    static constexpr int kBars = 3 * kSlots + 2 * kTcAcc + 1;
    static constexpr bool kRelu = MODE == kTcInput || MODE == kTcResidual || MODE == kTcResidualAux;
    static constexpr bool kRes = MODE == kTcResidual || MODE == kTcResidualAux;       // the addend is the input row
    static constexpr bool kAdd = MODE == kTcDgrad || MODE == kTcDgradMasked;          // another tensor
    static constexpr bool kMask = MODE == kTcDgradMasked || MODE == kTcLinearMasked;
    static constexpr bool kTwo = MODE == kTcResidualAux || kMask;
    static constexpr bool kF32 = MODE == kTcOutput;
    static constexpr int kCin = MODE == kTcInput || MODE == kTcLinear || MODE == kTcLinearMasked ? 16 : 32;
    static constexpr int kHalves = kCin / 16;        // MMAs' K steps per tap
    static constexpr int kChunks = kCin / 8;         // 16-byte channel chunks per pixel
    static constexpr int kPxBytes = 2 * kCin;
    static constexpr int kRowBytes = (NARROW ? kTcNarrowPx : (kTcHalo + 7) / 8 * 8) * kPxBytes;
    static constexpr int kCols = kF32 ? 16 : 32;     // accumulator columns of an output row
    static constexpr int kCout = kF32 ? 8 : 32;      // output channels the weights have
    static constexpr int kWRows = MODE == kTcLinearMasked ? 8 : 32;  // output channels of a masked gradient's layer
    static constexpr int kBlock = 3 * kCols * 16;    // weights of one (kx, chunk): rows ky = 2, 1, 0
    static constexpr uint64_t kSwizzle = kCin == 32 ? 4ull : 6ull;  // 64- or 32-byte swizzle
    static constexpr int kWOff = kSlots * kRowBytes;
    static constexpr int kStageOff = (kWOff + 3 * kChunks * kBlock + 511) / 512 * 512;
    static constexpr int kBarOff = kStageOff + (kF32 ? 0 : 8 * (kTwo ? 2 : 1) * kTcStageBytes);
    static constexpr int kSmem = kBarOff + 8 * kBars + 16 + 128;
    static_assert(2 * (kSmem + 1024) <= 228 * 1024, "two CTAs per SM");
    static constexpr uint32_t kTmemCols = kCols * kTcAcc;
};

struct TcArgs {
    const bf16 *w;
    const float *bias;
    const bf16 *res, *relu;  // data-gradient modes: the addend, and the mask's ReLU output
    const float *u;          // output mode
    float *out_f32;
    bf16 *out, *out2;        // out2: aux, or the masked gradient
    int nb, H, W, tiles_x;
    int box_px;              // pixels of an input row box (even, <= kTcHalo)
    // narrow images: a row tile is `step` positions of the line of all images' rows of pitch W + 2 pixels, from the
    // halo pixel on, loaded as the rows of `images` images; tiles_x counts the tiles of the whole line
    int step, images;
};

// The CTA's rows: [t0, t1) of the nb * tiles_x * H row tiles, column-major, as runs of one column.
struct TcRun {
    int img, x0, y0, rows;  // narrow: img the first image loaded, x0 the tile's first position in its row
};
template <bool NARROW>
__device__ __forceinline__ bool tc_run(const TcArgs &a, long long &t, long long t1, TcRun &r) {
    if (t >= t1) return false;
    const long long col = t / a.H;
    r.y0 = (int)(t - col * a.H);
    r.rows = (int)min((long long)(a.H - r.y0), t1 - t);
    if (NARROW) {
        const long long v = col * a.step;
        r.img = (int)(v / (a.W + 2));
        r.x0 = (int)(v - (long long)r.img * (a.W + 2));
    } else {
        r.img = (int)(col / a.tiles_x);
        r.x0 = (int)(col - (long long)r.img * a.tiles_x) * kTcPx;
    }
    t += r.rows;
    return true;
}

// A thread's pixel (four 16-byte chunks) to its place in the warp's 2 KB stage, in the 64-byte swizzle of
// the input rows: eight neighbouring threads write eight different bank groups.
__device__ __forceinline__ void tc_stage(unsigned char *stage, int lane, const uint4 (&v)[4]) {
    unsigned char *p = stage + lane * 64;
    const int k = (lane >> 1) & 3;
#pragma unroll
    for (int c = 0; c < 4; c++) *reinterpret_cast<uint4 *>(p + ((c ^ k) << 4)) = v[c];
}
__device__ __forceinline__ void tma_store(const CUtensorMap *tm, const void *smem, int x, int y, int img) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];\n" ::"l"(
                     reinterpret_cast<uint64_t>(tm)),
                 "r"(0), "r"(x), "r"(y), "r"(img), "r"(smem_u32(smem))
                 : "memory");
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {  // two f32 additions in one instruction
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;\n"
        : "=l"(d)
        : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&d);
}

template <int MODE, bool NARROW>
__global__ void __launch_bounds__(kTcThreads, 2) sg_conv32_tc_kernel(const __grid_constant__ CUtensorMap tmap,
                                                                     const __grid_constant__ CUtensorMap tmap_out,
                                                                     const __grid_constant__ CUtensorMap tmap_out2,
                                                                     const __grid_constant__ TcArgs a) {
    extern __shared__ __align__(1024) unsigned char tc_sm[];
    using C = TcCfg<MODE, NARROW>;
    constexpr int kTcSlots = C::kSlots, kTcBars = C::kBars;
    constexpr bool kRes = C::kRes, kTwo = C::kTwo;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(tc_sm);
    const uint32_t bars = sbase + C::kBarOff;
    const uint32_t full = bars, free_mma = full + 8 * kTcSlots, free_epi = free_mma + 8 * kTcSlots,
                   acc_full = free_epi + 8 * kTcSlots, acc_free = acc_full + 8 * kTcAcc, drain = acc_free + 8 * kTcAcc;
    volatile int *s_abort = reinterpret_cast<volatile int *>(tc_sm + C::kBarOff + 8 * kTcBars);
    const uint32_t tmem_slot = bars + 8 * kTcBars + 4;
    float *s_bias = reinterpret_cast<float *>(tc_sm + C::kBarOff + 8 * kTcBars + 16);
    if ((C::kRelu && tid < 32) || (C::kF32 && tid == 0)) s_bias[tid] = a.bias[tid];

    if (tid == 0) {
        for (int i = 0; i < kTcSlots; i++) {
            mbar_init(full + 8 * i, 1);
            mbar_init(free_mma + 8 * i, 1);
            mbar_init(free_epi + 8 * i, 4);
        }
        for (int i = 0; i < kTcAcc; i++) {
            mbar_init(acc_full + 8 * i, 1);
            mbar_init(acc_free + 8 * i, 4);
        }
        mbar_init(drain, 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tmem_slot),
                     "r"(C::kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // weights: element (co, tap = 3 ky + kx, ci) to block (kx, ci / 8), row kCols (2 - ky) + co
    for (int e = tid; e < C::kCols * 9 * C::kChunks; e += kTcThreads) {
        const int co = e / (9 * C::kChunks), kc = e - co * (9 * C::kChunks), tap = kc / C::kChunks,
                  c = kc - tap * C::kChunks, ky = tap / 3, kx = tap - 3 * ky;
        if (C::kMask) break;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (co < C::kCout) v = *reinterpret_cast<const uint4 *>(a.w + (co * 9 + tap) * C::kCin + 8 * c);
        *reinterpret_cast<uint4 *>(tc_sm + C::kWOff + (kx * C::kChunks + c) * C::kBlock +
                                   (C::kCols * (2 - ky) + co) * 16) = v;
    }
    // the masked data gradients take the layer's own weights [cout kWRows][9][32]: turned around (tap 8 - tap)
    // and transposed here, 32 lanes reading one row's 32 input channels
    if (C::kMask) {
        for (int e = tid; e < 32 * 9 * C::kChunks; e += kTcThreads) {
            const int n = e & 31, tc = e >> 5, tap = tc / C::kChunks, c = tc - tap * C::kChunks, ky = tap / 3,
                      kx = tap - 3 * ky;
            uint4 v;
            bf16 *b = reinterpret_cast<bf16 *>(&v);
#pragma unroll
            for (int j = 0; j < 8; j++)
                b[j] = 8 * c + j < C::kWRows ? a.w[((8 * c + j) * 9 + 8 - tap) * 32 + n] : __float2bfloat16(0.0f);
            *reinterpret_cast<uint4 *>(tc_sm + C::kWOff + (kx * C::kChunks + c) * C::kBlock + (32 * (2 - ky) + n) * 16) = v;
        }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the weights, for the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tc_sm + C::kBarOff + 8 * kTcBars + 4);

    const long long total = (NARROW ? 1ll : (long long)a.nb) * a.tiles_x * a.H;
    const long long t0 = total * blockIdx.x / gridDim.x, t1 = total * (blockIdx.x + 1) / gridDim.x;
    const uint32_t row_bytes = (uint32_t)(NARROW ? a.images * (a.W + 2) : a.box_px) * C::kPxBytes;
    // Input rows are numbered q = 0, 1, ... over the CTA's runs (a run of R output rows has R + 2), output
    // rows n; row q is in slot q % kTcSlots, row n in accumulator n % kTcAcc.
    long long t = t0;
    TcRun r;
    int issued = 0;  // the loader's rows, for the wind-down

    if (warp == 0) {
        if (lane == 0) {
            int q = 0;
            bool ok = true;
            while (ok && tc_run<NARROW>(a, t, t1, r)) {
                for (int i = 0; i < r.rows + 2; i++, q++) {
                    const int s = q % kTcSlots;
                    if (q >= kTcSlots) {
                        const uint32_t ph = (uint32_t)((q / kTcSlots + 1) & 1);
                        ok = mbar_wait(free_mma + 8 * s, ph, s_abort) &&
                             (!kRes || mbar_wait(free_epi + 8 * s, ph, s_abort));
                        if (!ok) {
                            *s_abort = 1;
                            break;
                        }
                    }
                    mbar_expect_tx(full + 8 * s, row_bytes);
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                        "%3, %4, %5}], [%6];\n" ::"r"(sbase + (uint32_t)(s * C::kRowBytes)),
                        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"(NARROW ? -1 : r.x0 - 1), "r"(r.y0 - 1 + i), "r"(r.img),
                        "r"(full + 8 * s)
                        : "memory");
                    issued = q + 1;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint64_t a0 = tc_desc(sbase, 16, 8 * C::kPxBytes) | (C::kSwizzle << 61);
        const uint64_t b0 = tc_desc(sbase + C::kWOff, C::kBlock, 128);
        int q = 0, n0 = 0;  // n0: output rows of the runs before
        bool ok = true;
        while (ok && tc_run<NARROW>(a, t, t1, r)) {
            for (int i = 0; i < r.rows + 2; i++, q++) {
                const int s = q % kTcSlots;
                // the run's output rows that input row i reaches: o0 .. o1, tap ky = i - o
                const int o0 = max(0, i - 2), o1 = min(r.rows - 1, i);
                const bool fresh = i < r.rows;  // row o1 = i starts with this input row
                if (fresh && n0 + i >= kTcAcc) {
                    const int n = n0 + i;
                    ok = mbar_wait(acc_free + 8 * (n % kTcAcc), (uint32_t)((n / kTcAcc + 1) & 1), s_abort);
                }
                ok = ok && mbar_wait(full + 8 * s, (uint32_t)((q / kTcSlots) & 1), s_abort);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    *s_abort = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t ad = a0 + (uint64_t)(s * (C::kRowBytes >> 4)) +
                                    (NARROW ? (uint64_t)(r.x0 * (C::kPxBytes >> 4)) : 0ull);
                // rows [o, o + cnt) of the window: accumulator columns from kCols ((n0 + o) % kTcAcc), weight
                // rows from kCols (2 - ky)
                const int w0 = (n0 + o0) % kTcAcc, cnt = o1 - o0 + 1, head = min(cnt, kTcAcc - w0);
                const uint64_t bd0 = b0 + (uint64_t)(C::kCols * (2 - (i - o0)));
                const uint32_t d0 = tmem + C::kCols * (uint32_t)w0;
                // Inside a run the window is three rows, the last one fresh: everything but the row slot and
                // the accumulator column is a constant of the loop, for each place of the wrap.
                auto inner = [&](auto head_c) {
                    constexpr int kHead = decltype(head_c)::value;  // rows before the wrap
#pragma unroll
                    for (int kx = 0; kx < 3; kx++)
#pragma unroll
                        for (int j = 0; j < C::kHalves; j++) {
                            const uint64_t av = ad + (uint64_t)((kx * C::kPxBytes + 32 * j) >> 4);
                            const uint64_t bv = b0 + (uint64_t)((kx * C::kChunks + 2 * j) * (C::kBlock >> 4));
                            if (kx == 0 && j == 0) {
                                constexpr int kOld = kHead < 2 ? kHead : 2;
                                tc_mma(d0, av, bv, tc_idesc(C::kCols * kOld), true);
                                if (kOld < 2) tc_mma(tmem, av, bv + C::kCols, tc_idesc(C::kCols), true);
                                tc_mma(kHead == 3 ? d0 + 2 * C::kCols : tmem + (2 - kHead) * C::kCols, av,
                                       bv + 2 * C::kCols, tc_idesc(C::kCols), false);
                            } else {
                                tc_mma(d0, av, bv, tc_idesc(C::kCols * kHead), true);
                                if (kHead < 3)
                                    tc_mma(tmem, av, bv + C::kCols * kHead, tc_idesc(C::kCols * (3 - kHead)), true);
                            }
                        }
                };
                if (fresh && cnt == 3 && head >= 3) inner(std::integral_constant<int, 3>());
                else if (fresh && cnt == 3 && head == 2) inner(std::integral_constant<int, 2>());
                else if (fresh && cnt == 3) inner(std::integral_constant<int, 1>());
                else {
#pragma unroll
                    for (int kx = 0; kx < 3; kx++)
#pragma unroll
                        for (int j = 0; j < C::kHalves; j++) {
                            const uint64_t av = ad + (uint64_t)((kx * C::kPxBytes + 32 * j) >> 4);
                            const uint64_t bv = bd0 + (uint64_t)((kx * C::kChunks + 2 * j) * (C::kBlock >> 4));
                            if (kx == 0 && j == 0 && fresh) {
                                const int old = cnt - 1, h = min(old, head);
                                if (h > 0) tc_mma(d0, av, bv, tc_idesc(C::kCols * h), true);
                                if (old > h)
                                    tc_mma(tmem, av, bv + C::kCols * h, tc_idesc(C::kCols * (old - h)), true);
                                tc_mma(tmem + C::kCols * (uint32_t)((n0 + o1) % kTcAcc), av, bv + C::kCols * old,
                                       tc_idesc(C::kCols), false);
                            } else {
                                tc_mma(d0, av, bv, tc_idesc(C::kCols * head), true);
                                if (cnt > head)
                                    tc_mma(tmem, av, bv + C::kCols * head, tc_idesc(C::kCols * (cnt - head)), true);
                            }
                        }
                }
                tc_commit(free_mma + 8 * s);
                if (i >= 2) tc_commit(acc_full + 8 * ((n0 + i - 2) % kTcAcc));
            }
            n0 += r.rows;
        }
        tc_commit(drain);
        __syncwarp();
    } else {
        // two groups of four warps take the output rows in turn: one row's way through the epilogue is
        // about 2000 cycles of latency, and a group alone left every unit of the SM below 50 % busy
        const int quad = warp & 3;  // the tensor-memory lanes this warp may read
        const int group = (warp - 2) >> 2;
        unsigned char *stage = tc_sm + C::kStageOff + (warp - 2) * ((kTwo ? 2 : 1) * kTcStageBytes);
        const int m = quad * 32 + lane;
        int q = 0, n = 0;
        bool ok = true;
        // a halo row, which has no output, is freed once it has arrived (not before: its slot's previous row
        // may still lack another warp's arrival)
        auto free_halo = [&](int row) {
            if (!kRes || group != 0 || lane != 0 || !ok) return;
            ok = mbar_wait(full + 8 * (row % kTcSlots), (uint32_t)((row / kTcSlots) & 1), s_abort);
            if (ok) mbar_arrive(free_epi + 8 * (row % kTcSlots));
            else *s_abort = 1;
        };
        while (tc_run<NARROW>(a, t, t1, r)) {
            free_halo(q);
            for (int o = 0; o < r.rows; o++, n++) {
                if ((n & 1) != group) continue;
                const int y = r.y0 + o, acc = n % kTcAcc;
                int x = r.x0 + m, img = r.img;
                if (NARROW) {
                    img += x / (a.W + 2);
                    x %= a.W + 2;
                    if (m >= a.step || img >= a.nb) x = a.W;  // no pixel
                }
                const size_t p = ((size_t)img * a.H + y) * a.W + x;
                uint4 rv[4], mv[4];
                float uv = 0.0f;
                if (x < a.W) {
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        if (C::kAdd) rv[c] = *reinterpret_cast<const uint4 *>(a.res + p * 32 + 8 * c);
                        if (C::kMask) mv[c] = __ldg(reinterpret_cast<const uint4 *>(a.relu + p * 32 + 8 * c));
                    }
                    if (C::kF32) uv = a.u[p];
                }
                ok = ok && mbar_wait(acc_full + 8 * acc, (uint32_t)((n / kTcAcc) & 1), s_abort);
                const int qi = q + o + 1, s = qi % kTcSlots;  // the input row at the output's place
                if (kRes) ok = ok && mbar_wait(full + 8 * s, (uint32_t)((qi / kTcSlots) & 1), s_abort);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    *s_abort = 1;
                    if (x < a.W) {  // a failed launch cannot pass for a result
                        const uint4 nan4 = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
                        if (C::kF32) a.out_f32[p] = __int_as_float(0x7fc00000);
#pragma unroll
                        for (int c = 0; c < (C::kF32 ? 0 : 4); c++) {
                            if (a.out) *reinterpret_cast<uint4 *>(a.out + p * 32 + 8 * c) = nan4;
                            if (kTwo) *reinterpret_cast<uint4 *>(a.out2 + p * 32 + 8 * c) = nan4;
                        }
                    }
                    continue;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t tcol = tmem + C::kCols * (uint32_t)acc + ((uint32_t)(quad * 32) << 16);
                uint32_t v[32];
                if (C::kF32) {
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(v[0]) : "r"(tcol));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_free + 8 * acc);
                    if (x < a.W) a.out_f32[p] = uv + __uint_as_float(v[0]) + s_bias[0];
                    continue;
                }
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                    "[%32];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                      "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                      "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(tcol));
                if (kRes) {
                    // chunk c of pixel i lies at chunk c ^ (i / 2 % 4) of its 64 bytes (the swizzle)
                    const int px = (NARROW ? r.x0 : 0) + m + 1;
                    const unsigned char *rp = tc_sm + s * C::kRowBytes + px * 64;
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        rv[c] = *reinterpret_cast<const uint4 *>(rp + ((c ^ ((px >> 1) & 3)) << 4));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                // the stage's previous row has been read
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_free + 8 * acc);
                uint4 ov[4], av[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const __nv_bfloat162 *r2 = reinterpret_cast<const __nv_bfloat162 *>(&rv[c]);
                    const __nv_bfloat162 *m2 = reinterpret_cast<const __nv_bfloat162 *>(&mv[c]);
                    __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&ov[c]);
                    __nv_bfloat162 *a2 = reinterpret_cast<__nv_bfloat162 *>(&av[c]);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int ch = 8 * c + 2 * k;
                        float2 z = make_float2(__uint_as_float(v[ch]), __uint_as_float(v[ch + 1]));
                        if (C::kRelu) {
                            z = add2(z, *reinterpret_cast<const float2 *>(&s_bias[ch]));
                            z = make_float2(fmaxf(z.x, 0.0f), fmaxf(z.y, 0.0f));
                        }
                        if (MODE == kTcResidualAux) a2[k] = __float22bfloat162_rn(z);
                        if (kRes || C::kAdd) z = add2(z, __bfloat1622float2(r2[k]));
                        o2[k] = __float22bfloat162_rn(z);
                        if (C::kMask) {
                            const float2 mf = __bfloat1622float2(m2[k]);
                            a2[k].x = mf.x > 0.0f ? o2[k].x : __float2bfloat16(0.0f);
                            a2[k].y = mf.y > 0.0f ? o2[k].y : __float2bfloat16(0.0f);
                        }
                    }
                }
                if (!C::kMask || a.out) tc_stage(stage, lane, ov);
                if (kTwo) tc_stage(stage + kTcStageBytes, lane, av);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    // Only now: the staged values prove that the warp's reads of the row slot have returned.  An
                    // arrival right behind the loads can pass them, and a halo row outside the image (filled
                    // with zeros at once) then overwrites what they are about to read.
                    if (kRes) mbar_arrive(free_epi + 8 * s);
                    if (!NARROW && x < a.W) {  // the box is cut at the image's edge
                        if (!C::kMask || a.out) tma_store(&tmap_out, stage, x, y, r.img);
                        if (kTwo) tma_store(&tmap_out2, stage + kTcStageBytes, x, y, r.img);
                    }
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
                if (NARROW) {
                    // a warp's 32 positions lie in up to three images: plain stores, four lanes to a pixel
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int px = 8 * k + (lane >> 2), c = lane & 3;
                        const bool has = __shfl_sync(0xffffffffu, x < a.W ? 1 : 0, px) != 0;
                        const size_t at = (size_t)__shfl_sync(0xffffffffu, (unsigned long long)p, px) * 32 + 8 * c;
                        const unsigned char *from = stage + px * 64 + ((c ^ ((px >> 1) & 3)) << 4);
                        if (has) {
                            if (!C::kMask || a.out) *reinterpret_cast<uint4 *>(a.out + at) = *reinterpret_cast<const uint4 *>(from);
                            if (kTwo)
                                *reinterpret_cast<uint4 *>(a.out2 + at) =
                                    *reinterpret_cast<const uint4 *>(from + kTcStageBytes);
                        }
                    }
                    __syncwarp();  // the stage is written again for the next row
                }
            }
            q += r.rows + 2;
            free_halo(q - 1);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
        __syncwarp();
    }
    __syncthreads();
    // the copies and MMAs this CTA issued land before its shared and tensor memory are released (after a
    // normal run they have: every row was waited for)
    if (tid == 0 && *s_abort) {
        atomicExch(&g_sg_tc_timeout, 1);
        const int none = 0;
        for (int q = max(0, issued - kTcSlots); q < issued; q++)
            (void)mbar_wait(full + 8 * (q % kTcSlots), (uint32_t)((q / kTcSlots) & 1), &none);
    }
    if (warp == 1) {
        if (lane == 0) {
            const int none = 0;
            (void)mbar_wait(drain, 0, &none);
        }
        __syncwarp();
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(C::kTmemCols)
                     : "memory");
    }
}

template <int MODE, bool NARROW>
static cudaError_t launch_tc_as(const void *in, int in_cstride, TcArgs a, cudaStream_t s) {
    using C = TcCfg<MODE, NARROW>;
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    CUtensorMap tm[3];  // input rows, and 32-pixel boxes of the outputs
    const void *base[3] = {in, C::kF32 ? in : (a.out ? a.out : a.out2), C::kTwo ? a.out2 : (C::kF32 ? in : a.out)};
    for (int k = 0; k < 3; k++) {
        const cuuint64_t ch = k == 0 || C::kF32 ? C::kCin : 32, px = k == 0 || C::kF32 ? 2 * (cuuint64_t)in_cstride : 64;
        const cuuint64_t dims[4] = {ch, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.nb};
        const cuuint64_t strides[3] = {px, (cuuint64_t)a.W * px, (cuuint64_t)a.H * a.W * px};
        const cuuint32_t box[4] = {(cuuint32_t)ch, k == 0 ? (cuuint32_t)(NARROW ? a.W + 2 : a.box_px) : 32u, 1,
                                   k == 0 && NARROW ? (cuuint32_t)a.images : 1u};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        if (encode(&tm[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base[k]), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, ch == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sg_conv32_tc_kernel<MODE, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
    if (e != cudaSuccess) return e;
    const long long rows = (NARROW ? 1ll : (long long)a.nb) * a.tiles_x * a.H;
    const long long grid = std::min<long long>(rows, 2ll * std::max(1, sms));
    sg_conv32_tc_kernel<MODE, NARROW><<<(unsigned)grid, kTcThreads, C::kSmem, s>>>(tm[0], tm[1], tm[2], a);
    return cudaGetLastError();
}

// Images so narrow that a row would leave half of the 128 accumulator rows empty share their row tiles: the
// rows of all images stand in one line, each with its two halo pixels, and the line is cut every 128
// positions -- or, where that would need more than kTcNarrowPx pixels loaded for a tile, every whole number of
// images.  The halo positions' sums are dropped.
// 256 tiles of 64^2, 32 -> 32 channels with the ReLU output (201 MB, 30 us at the measured copy rate): 51 -> 44 us,
// the masked data gradient (335 MB, 50 us) 65 -> 58, the input conv 32 -> 25; 200 images of 50 x 33, a layer call by
// call: 35 us.
static bool tc_narrow(TcArgs &a) {
    const int pitch = a.W + 2;
    if (a.nb < 2 || pitch > kTcNarrowPx / 3) return false;
    const long long line = (long long)a.nb * pitch;
    a.step = kTcPx;
    int off = 0;  // the last first position of a tile in its image's row: the multiples of gcd(128, pitch)
    for (int t = 0; t < pitch; t++) off = std::max(off, t * kTcPx % pitch);
    a.images = (off + kTcHalo + pitch - 1) / pitch;
    if (a.images * pitch > kTcNarrowPx) {
        a.images = kTcPx / pitch;
        if (a.images < 2) return false;
        a.step = a.images * pitch;
    }
    a.tiles_x = (int)((line + a.step - 1) / a.step);
    return true;
}

template <int MODE>
static cudaError_t launch_tc(const void *in, int in_cstride, TcArgs a, cudaStream_t s) {
    return tc_narrow(a) ? launch_tc_as<MODE, true>(in, in_cstride, a, s) : launch_tc_as<MODE, false>(in, in_cstride, a, s);
}

// A surrogate conv on the tensor cores, by the C-ABI's kinds.  For the residual kind res is the input itself; res
// may be out in the data gradient; out2 (may be null) is the ReLU output (residual) or the gradient masked by
// `relu` (then w are the layer's own weights, else already turned around, and out may be null).  Returns
// cudaErrorNotSupported when the buffers overlap otherwise or are not 16-byte aligned, or the tensor maps cannot be
// made (the caller's mma.sync kernels run instead).
cudaError_t launch_sg_conv_tc(int kind, const void *in, int in_cstride, const void *w, const float *bias, const void *res,
                              const float *u, const void *relu, void *out, void *out2, float *out_f32, int nb, int H,
                              int W, cudaStream_t s) {
    if (nb <= 0 || H <= 0 || W <= 0) return cudaSuccess;
    const void *ptrs[] = {in, w, res, relu, out, out2};
    for (const void *p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) & 15u) return cudaErrorNotSupported;
    if (in == out || (out2 && (in == out2 || out2 == out || out2 == res))) return cudaErrorNotSupported;
    if (kind == FG_SG_CONV_RESIDUAL && (res != in || in_cstride != 32)) return cudaErrorNotSupported;
    TcArgs a;
    a.w = static_cast<const bf16 *>(w);
    a.bias = bias;
    a.res = static_cast<const bf16 *>(res);
    a.relu = static_cast<const bf16 *>(relu);
    a.u = u;
    a.out_f32 = out_f32;
    a.out = static_cast<bf16 *>(out);
    a.out2 = static_cast<bf16 *>(out2);
    a.nb = nb; a.H = H; a.W = W;
    a.tiles_x = (W + kTcPx - 1) / kTcPx;
    a.box_px = std::min(kTcHalo, (W + 9) & ~7);  // W + 2 halo pixels, in whole swizzle periods
    switch (kind) {
    case FG_SG_CONV_INPUT: return launch_tc<kTcInput>(in, in_cstride, a, s);
    case FG_SG_CONV_RESIDUAL:
        return out2 ? launch_tc<kTcResidualAux>(in, in_cstride, a, s) : launch_tc<kTcResidual>(in, in_cstride, a, s);
    case FG_SG_CONV_OUTPUT: return launch_tc<kTcOutput>(in, in_cstride, a, s);
    case FG_SG_CONV_DGRAD_RESIDUAL:
        return out2 ? launch_tc<kTcDgradMasked>(in, in_cstride, a, s) : launch_tc<kTcDgrad>(in, in_cstride, a, s);
    case FG_SG_CONV_DGRAD_OUTPUT:
        return out2 ? launch_tc<kTcLinearMasked>(in, in_cstride, a, s) : launch_tc<kTcLinear>(in, in_cstride, a, s);
    default: return cudaErrorNotSupported;
    }
}

// Whether a tensor-core conv ran out of an mbarrier wait since the last call (and clears the flag).
cudaError_t sg_conv_tc_timeouts(int *v) {
    const int z = 0;
    cudaError_t e = cudaMemcpyFromSymbol(v, g_sg_tc_timeout, sizeof *v);
    if (e == cudaSuccess && *v) e = cudaMemcpyToSymbol(g_sg_tc_timeout, &z, sizeof z);
    return e;
}

}  // namespace fg
