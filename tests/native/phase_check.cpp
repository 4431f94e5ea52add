// The stream pass's phase masks (fg_phase.cuh) against their definition: an offset of z o counts for a grain at
// v = z g - 0.5 with half-width w when an integer lies within w of v + z o.  Random offsets, grains and half-widths,
// and the edges: fractions next to 0, 1 and the buckets' bounds, half-widths at the classes' bounds and the
// largest.  Prints "checked missed passed counted".
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "fg_phase.cuh"

using namespace fg;

static uint64_t st = 7;
static float uniform() {
    st += kPhi;
    return (float)(fmix64(st) >> 40) * 0x1p-24f;
}

int main() {
    long long checked = 0, missed = 0, passed = 0, counted = 0;
    const int ns[] = {1, 31, 32, 33, 64, 100, 256};
    for (int n : ns) {
        for (int rep = 0; rep < 6; rep++) {
            float oz[256];
            for (int e = 0; e < n; e++) {
                oz[e] = (uniform() - 0.5f) * 8.0f;
                if (e % 11 == 3) oz[e] = rintf(oz[e]);                    // whole
                if (e % 11 == 7) oz[e] = nextafterf(rintf(oz[e]), -9.0f); // next below a whole number
            }
            const float w_max = 0.02f + 0.38f * uniform(), scale = (float)kPhaseClasses / w_max;
            for (int t = 0; t < 400; t++) {
                float v = uniform() * 4000.0f;
                if (t % 5 == 1) v = rintf(v * 64.0f) / 64.0f;
                if (t % 5 == 2) v = nextafterf(rintf(v * 64.0f) / 64.0f, 0.0f);
                if (t % 50 == 3) v = -1e-9f;
                float w = w_max * uniform();
                if (t % 7 == 1) w = w_max;
                if (t % 7 == 2) w = w_max * 0.25f * (float)(1 + t % 4);
                const int b = phase_bucket(v), c = phase_class(w, scale);
                for (int e = 0; e < n; e++) {
                    const double at = (double)v + (double)oz[e];
                    const bool want = std::fabs(at - std::rint(at)) <= (double)w;
                    const bool got = (phase_mask_word(oz, n, b, c, e / 32, w_max) >> (e % 32)) & 1u;
                    checked++;
                    if (want && !got) missed++;
                    passed += got ? 1 : 0;
                    counted += want ? 1 : 0;
                }
            }
        }
    }
    std::printf("%lld %lld %lld %lld\n", checked, missed, passed, counted);
    return 0;
}
