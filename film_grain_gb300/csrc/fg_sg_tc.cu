// fg_sg_tc.cu -- the surrogate's 32 -> 32 convs on the fifth-generation tensor cores.
//
// NHWC bf16 activations with 32 channels, weights [cout 32][tap 9][cin 32] bf16, f32 accumulation:
//   residual       out = in + relu(conv3x3(in) + b)      (aux, for training: the ReLU output)
//   data gradient  out = res + conv3x3(in)               (masked: out where relu > 0, else 0)
//
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
// Measured at 3 x 1024^2 pixels (403 MB, 60 us at the measured copy rate): 18 MMAs of N 32 per row 128 us;
// this split, one epilogue group and rows as 16-byte TMA pieces 95 us; two groups 92 us; the MMAs issued by a
// converged warp 78 us (call by call 139 -> 81 us).  What is left is shared-memory traffic: 8.5 MMAs a row
// with the overwriting and wrapping ones, 7 KB each, and 33 KB of rows in and out against 128 B per clock.
//
// Every wait on an mbarrier is bounded; a wait that runs out records the fact in g_sg_tc_timeout, writes NaN
// outputs for the CTA's rows not yet written, waits (bounded) for its own copies and MMAs, frees its tensor
// memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "fg_internal.h"

namespace fg {

typedef __nv_bfloat16 bf16;

constexpr int kTcPx = 128;          // output pixels of one row tile (the MMA's M)
constexpr int kTcHalo = kTcPx + 2;  // input pixels of one row at most
constexpr int kTcRowBytes = 17 * 512;  // 130 x 64 bytes, to the 512 bytes that the 64-byte swizzle repeats over
constexpr int kTcSlots = 6;         // input rows in flight
constexpr int kTcAcc = 8;           // accumulator rows (32 columns each) in tensor memory
constexpr uint32_t kTcTmemCols = 32 * kTcAcc;
constexpr int kTcWOff = kTcSlots * kTcRowBytes;
constexpr int kTcWBytes = 36 * 32 * 16;
constexpr int kTcStageOff = kTcWOff + kTcWBytes;
constexpr int kTcStageBytes = 2048;              // a warp's 32 pixels
constexpr int kTcThreads = 320;                  // loader, MMA issuer, two groups of four epilogue warps
// barriers: rows full, rows free (MMA), rows free (epilogue), accumulators full, accumulators free, drain
constexpr int kTcBars = 3 * kTcSlots + 2 * kTcAcc + 1;
// SM cycles a wait on an mbarrier may take before it gives up (about a second)
constexpr long long kTcWaitCycles = 2000000000ll;

__device__ int g_sg_tc_timeout;

enum TcMode { kTcResidual = 0, kTcResidualAux = 1, kTcDgrad = 2, kTcDgradMasked = 3 };

__host__ __device__ constexpr int tc_outputs(int mode) { return mode == kTcResidualAux || mode == kTcDgradMasked ? 2 : 1; }
__host__ __device__ constexpr int tc_bar_off(int mode) { return kTcStageOff + 8 * tc_outputs(mode) * kTcStageBytes; }
constexpr int tc_smem(int mode) { return tc_bar_off(mode) + 8 * kTcBars + 16 + 128; }

// Instruction descriptor of tcgen05.mma kind::f16: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9 and
// 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t tc_idesc(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: start address, leading (K-direction core-matrix) byte
// offset, stride (M/N-direction core-matrix) byte offset, each >> 4; descriptor version 1 at bit 46.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded wait for the completion of the phase with the given parity; false when the limit ran out or
// another warp gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int *abort) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (*abort || clock64() - t0 > kTcWaitCycles) return false;
    }
}
// The MMA warp runs as one: every lane holds the same operands and the leader's predicate guards the
// instruction itself.  (Issued by one lane inside a branch, the operands went through vector registers and
// an MMA took about 250 cycles to issue, five times its own time.)
__device__ __forceinline__ void tc_commit(uint32_t bar, bool leader) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
        "r"(leader ? 1u : 0u)
        : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc, bool leader) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u), "r"(leader ? 1u : 0u)
        : "memory");
}

struct TcArgs {
    const bf16 *w;
    const float *bias;       // residual modes
    const bf16 *res, *relu;  // data-gradient modes: the addend, and the mask's ReLU output
    bf16 *out, *out2;        // out2: aux, or the masked gradient
    int nb, H, W, tiles_x;
    int box_px;              // pixels of an input row box (even, <= kTcHalo)
};

// The CTA's rows: [t0, t1) of the nb * tiles_x * H row tiles, column-major, as runs of one column.
struct TcRun {
    int img, x0, y0, rows;
};
__device__ __forceinline__ bool tc_run(const TcArgs &a, long long &t, long long t1, TcRun &r) {
    if (t >= t1) return false;
    const long long col = t / a.H;
    r.y0 = (int)(t - col * a.H);
    r.rows = (int)min((long long)(a.H - r.y0), t1 - t);
    r.img = (int)(col / a.tiles_x);
    r.x0 = (int)(col - (long long)r.img * a.tiles_x) * kTcPx;
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

template <int MODE>
__global__ void __launch_bounds__(kTcThreads, 2) sg_conv32_tc_kernel(const __grid_constant__ CUtensorMap tmap,
                                                                     const __grid_constant__ CUtensorMap tmap_out,
                                                                     const __grid_constant__ CUtensorMap tmap_out2,
                                                                     const __grid_constant__ TcArgs a) {
    extern __shared__ __align__(1024) unsigned char tc_sm[];
    constexpr bool kRes = MODE == kTcResidual || MODE == kTcResidualAux;  // the addend is the input itself
    constexpr bool kTwo = MODE == kTcResidualAux || MODE == kTcDgradMasked;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(tc_sm);
    const uint32_t bars = sbase + tc_bar_off(MODE);
    const uint32_t full = bars, free_mma = full + 8 * kTcSlots, free_epi = free_mma + 8 * kTcSlots,
                   acc_full = free_epi + 8 * kTcSlots, acc_free = acc_full + 8 * kTcAcc, drain = acc_free + 8 * kTcAcc;
    volatile int *s_abort = reinterpret_cast<volatile int *>(tc_sm + tc_bar_off(MODE) + 8 * kTcBars);
    const uint32_t tmem_slot = bars + 8 * kTcBars + 4;
    float *s_bias = reinterpret_cast<float *>(tc_sm + tc_bar_off(MODE) + 8 * kTcBars + 16);
    if (kRes && tid < 32) s_bias[tid] = a.bias[tid];

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
                     "r"(kTcTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // weights: element (co, tap = 3 ky + kx, ci) to block (kx, ci / 8), row 32 (2 - ky) + co
    for (int e = tid; e < 32 * 36; e += kTcThreads) {
        const int co = e / 36, kc = e - co * 36, tap = kc >> 2, c = kc & 3, ky = tap / 3, kx = tap - 3 * ky;
        const uint4 v = *reinterpret_cast<const uint4 *>(a.w + co * 288 + kc * 8);
        *reinterpret_cast<uint4 *>(tc_sm + kTcWOff + ((kx * 4 + c) * 96 + 32 * (2 - ky) + co) * 16) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the weights, for the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tc_sm + tc_bar_off(MODE) + 8 * kTcBars + 4);

    const long long total = (long long)a.nb * a.tiles_x * a.H;
    const long long t0 = total * blockIdx.x / gridDim.x, t1 = total * (blockIdx.x + 1) / gridDim.x;
    const uint32_t row_bytes = (uint32_t)a.box_px * 64;
    // Input rows are numbered q = 0, 1, ... over the CTA's runs (a run of R output rows has R + 2), output
    // rows n; row q is in slot q % kTcSlots, row n in accumulator n % kTcAcc.
    long long t = t0;
    TcRun r;
    int issued = 0;  // the loader's rows, for the wind-down

    if (warp == 0) {
        if (lane == 0) {
            int q = 0;
            bool ok = true;
            while (ok && tc_run(a, t, t1, r)) {
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
                        "%3, %4, %5}], [%6];\n" ::"r"(sbase + (uint32_t)(s * kTcRowBytes)),
                        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"(r.x0 - 1), "r"(r.y0 - 1 + i), "r"(r.img),
                        "r"(full + 8 * s)
                        : "memory");
                    issued = q + 1;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const bool leader = lane == 0;
        const uint64_t a0 = tc_desc(sbase, 16, 512) | (4ull << 61);  // 64-byte swizzle, rows of 64 bytes
        const uint64_t b0 = tc_desc(sbase + kTcWOff, 1536, 128);
        int q = 0, n0 = 0;  // n0: output rows of the runs before
        bool ok = true;
        while (ok && tc_run(a, t, t1, r)) {
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
                const uint64_t ad = a0 + (uint64_t)(s * (kTcRowBytes >> 4));
                // rows [o, o + cnt) of the window: accumulator columns from 32 ((n0 + o) % kTcAcc), weight
                // rows from 32 (2 - ky)
                const int w0 = (n0 + o0) % kTcAcc, cnt = o1 - o0 + 1, head = min(cnt, kTcAcc - w0);
                const uint64_t bd0 = b0 + (uint64_t)(32 * (2 - (i - o0)));
                const uint32_t d0 = tmem + 32u * (uint32_t)w0;
#pragma unroll
                for (int kx = 0; kx < 3; kx++)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const uint64_t av = ad + (uint64_t)(4 * kx + 2 * j);
                        const uint64_t bv = bd0 + (uint64_t)((kx * 4 + 2 * j) * 96);
                        if (kx == 0 && j == 0 && fresh) {
                            const int old = cnt - 1, h = min(old, head);
                            if (h > 0) tc_mma(d0, av, bv, tc_idesc(32u * h), true, leader);
                            if (old > h) tc_mma(tmem, av, bv + 32u * h, tc_idesc(32u * (old - h)), true, leader);
                            tc_mma(tmem + 32u * (uint32_t)((n0 + o1) % kTcAcc), av, bv + 32u * old, tc_idesc(32u), false,
                                   leader);
                        } else {
                            tc_mma(d0, av, bv, tc_idesc(32u * head), true, leader);
                            if (cnt > head) tc_mma(tmem, av, bv + 32u * head, tc_idesc(32u * (cnt - head)), true, leader);
                        }
                    }
                tc_commit(free_mma + 8 * s, leader);
                if (i >= 2) tc_commit(acc_full + 8 * ((n0 + i - 2) % kTcAcc), leader);
            }
            n0 += r.rows;
        }
        tc_commit(drain, leader);
        __syncwarp();
    } else {
        // two groups of four warps take the output rows in turn: one row's way through the epilogue is
        // about 2000 cycles of latency, and a group alone left every unit of the SM below 50 % busy
        const int quad = warp & 3;  // the tensor-memory lanes this warp may read
        const int group = (warp - 2) >> 2;
        unsigned char *stage = tc_sm + kTcStageOff + (warp - 2) * (tc_outputs(MODE) * kTcStageBytes);
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
        while (tc_run(a, t, t1, r)) {
            free_halo(q);
            for (int o = 0; o < r.rows; o++, n++) {
                if ((n & 1) != group) continue;
                const int x = r.x0 + m, y = r.y0 + o, acc = n % kTcAcc;
                const size_t p = ((size_t)r.img * a.H + y) * a.W + x;
                uint4 rv[4], mv[4];
                if (!kRes && x < a.W) {
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        rv[c] = *reinterpret_cast<const uint4 *>(a.res + p * 32 + 8 * c);
                        if (kTwo) mv[c] = __ldg(reinterpret_cast<const uint4 *>(a.relu + p * 32 + 8 * c));
                    }
                }
                ok = ok && mbar_wait(acc_full + 8 * acc, (uint32_t)((n / kTcAcc) & 1), s_abort);
                const int qi = q + o + 1, s = qi % kTcSlots;  // the input row at the output's place
                if (kRes) ok = ok && mbar_wait(full + 8 * s, (uint32_t)((qi / kTcSlots) & 1), s_abort);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    *s_abort = 1;
                    if (x < a.W) {  // a failed launch cannot pass for a result
                        const uint4 nan4 = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            *reinterpret_cast<uint4 *>(a.out + p * 32 + 8 * c) = nan4;
                            if (kTwo) *reinterpret_cast<uint4 *>(a.out2 + p * 32 + 8 * c) = nan4;
                        }
                    }
                    continue;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t v[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                    "[%32];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                      "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                      "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(tmem + 32u * (uint32_t)acc + ((uint32_t)(quad * 32) << 16)));
                if (kRes) {
                    // chunk c of pixel i lies at chunk c ^ (i / 2 % 4) of its 64 bytes (the swizzle)
                    const unsigned char *rp = tc_sm + s * kTcRowBytes + (m + 1) * 64;
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        rv[c] = *reinterpret_cast<const uint4 *>(rp + ((c ^ (((m + 1) >> 1) & 3)) << 4));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                // the stage's previous row has been read
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(acc_free + 8 * acc);
                    if (kRes) mbar_arrive(free_epi + 8 * s);
                }
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
                        if (kRes) {
                            z = add2(z, *reinterpret_cast<const float2 *>(&s_bias[ch]));
                            z = make_float2(fmaxf(z.x, 0.0f), fmaxf(z.y, 0.0f));
                        }
                        if (MODE == kTcResidualAux) a2[k] = __float22bfloat162_rn(z);
                        o2[k] = __float22bfloat162_rn(add2(z, __bfloat1622float2(r2[k])));
                        if (MODE == kTcDgradMasked) {
                            const float2 mf = __bfloat1622float2(m2[k]);
                            a2[k].x = mf.x > 0.0f ? o2[k].x : __float2bfloat16(0.0f);
                            a2[k].y = mf.y > 0.0f ? o2[k].y : __float2bfloat16(0.0f);
                        }
                    }
                }
                tc_stage(stage, lane, ov);
                if (kTwo) tc_stage(stage + kTcStageBytes, lane, av);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (x < a.W) {  // the box is cut at the image's edge
                        tma_store(&tmap_out, stage, x, y, r.img);
                        if (kTwo) tma_store(&tmap_out2, stage + kTcStageBytes, x, y, r.img);
                    }
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTcTmemCols)
                     : "memory");
    }
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

template <int MODE>
static cudaError_t launch_tc(const CUtensorMap (&tm)[3], const TcArgs &a, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sg_conv32_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem(MODE));
    if (e != cudaSuccess) return e;
    const long long rows = (long long)a.nb * a.tiles_x * a.H;
    const long long grid = std::min<long long>(rows, 2ll * std::max(1, sms));
    sg_conv32_tc_kernel<MODE><<<(unsigned)grid, kTcThreads, tc_smem(MODE), s>>>(tm[0], tm[1], tm[2], a);
    return cudaGetLastError();
}

// The 32 -> 32 convs on the tensor cores.  res == null: out = in + relu(conv(in) + bias), out2 (may be null)
// = the ReLU output.  Else out = res + conv(in), out2 (may be null) = out where relu > 0; res may be out.
// 32 channels per pixel, out and out2 distinct from in.  Returns cudaErrorNotSupported when the buffers are
// not 16-byte aligned or the tensor map cannot be made (the caller's mma.sync kernel runs instead).
cudaError_t launch_sg_conv32_tc(const void *in, const void *w, const float *bias, const void *res, const void *relu,
                                void *out, void *out2, int nb, int H, int W, cudaStream_t s) {
    if (nb <= 0 || H <= 0 || W <= 0) return cudaSuccess;
    const void *ptrs[] = {in, w, res, relu, out, out2};
    for (const void *p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) & 15u) return cudaErrorNotSupported;
    if (in == out || in == out2 || (out2 && (out2 == out || out2 == res))) return cudaErrorNotSupported;
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    TcArgs a;
    a.w = static_cast<const bf16 *>(w);
    a.bias = bias;
    a.res = static_cast<const bf16 *>(res);
    a.relu = static_cast<const bf16 *>(relu);
    a.out = static_cast<bf16 *>(out);
    a.out2 = static_cast<bf16 *>(out2);
    a.nb = nb; a.H = H; a.W = W;
    a.tiles_x = (W + kTcPx - 1) / kTcPx;
    a.box_px = std::min(kTcHalo, (W + 3) & ~1);  // W + 2 halo pixels, rounded up to even (128-byte rows)
    CUtensorMap tm[3];  // input rows, and 32-pixel boxes of the outputs
    const void *base[3] = {in, out, out2 ? out2 : out};
    for (int k = 0; k < 3; k++) {
        const cuuint64_t dims[4] = {32, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)nb};
        const cuuint64_t strides[3] = {64, (cuuint64_t)W * 64, (cuuint64_t)H * W * 64};
        const cuuint32_t box[4] = {32, k == 0 ? (cuuint32_t)a.box_px : 32u, 1, 1};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        if (encode(&tm[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base[k]), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    if (!res) return out2 ? launch_tc<kTcResidualAux>(tm, a, s) : launch_tc<kTcResidual>(tm, a, s);
    return out2 ? launch_tc<kTcDgradMasked>(tm, a, s) : launch_tc<kTcDgrad>(tm, a, s);
}

// Whether a tensor-core conv ran out of an mbarrier wait since the last call (and clears the flag).
int sg_conv32_tc_timeouts() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_sg_tc_timeout, sizeof v) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    const int z = 0;
    cudaMemcpyToSymbol(g_sg_tc_timeout, &z, sizeof z);
    return v;
}

}  // namespace fg
