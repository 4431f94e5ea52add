// first_draw_maybe against first_draw_screen, with the library's own header (fg_rng.cuh):
//  1. every hash and threshold that first_draw_screen passes, first_draw_maybe passes (thresholds around each
//     hash's own draw, around the distance of the bound, and at the edges);
//  2. on thresholds of 0.1 .. 0.9 of the range, the cells that first_draw_maybe passes beyond those.
// Prints "checked missed checked extra".
#include <cstdint>
#include <cstdio>

#include "fg_rng.cuh"

using namespace fg;

int main() {
    uint64_t st = 99;
    long long checked = 0, missed = 0, checked2 = 0, extra = 0;
    for (int n = 0; n < 200000; n++) {
        st += kPhi;
        const uint64_t h = fmix64(st);
        const long long v = (long long)(small_first_u64(h) >> 11), step = 1ll << 45;  // 2^24 in the high word
        const long long ts[] = {-5, -1, 0, 1, step - 1, step, step + 1, v - 2 * step, v - step - 1, v - step, v - 1, v,
                                v + 1, v + step, (1ll << 53) - step, (1ll << 53) - 2, (1ll << 53) - 1, 1ll << 53};
        for (long long t : ts) {
            checked++;
            if (first_draw_screen(h, screen_bound(t)) && !first_draw_maybe(h, maybe_bound(t))) missed++;
        }
        for (int p = 1; p < 10; p++) {
            const long long t = (long long)(0.1 * p * (double)(1ll << 53));
            checked2++;
            if (!first_draw_screen(h, screen_bound(t)) && first_draw_maybe(h, maybe_bound(t))) extra++;
        }
    }
    std::printf("%lld %lld %lld %lld\n", checked, missed, checked2, extra);
    return 0;
}
