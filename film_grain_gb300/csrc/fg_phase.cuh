// fg_phase.cuh -- which offsets can put a sample within a grain's radius, from the phases of both: the tables of
// the stream pass (fg_pixelwise_stream.cuh), host and device.
//
// With z = zoom, a sample of offset o lies at pixel x when x + 0.5 = z (xg + o); a grain at gx is within r of it
// only if z gx - 0.5 + z o is within r z of the integer x.  So with f the fraction of z gx - 0.5, an offset
// counts when f + z o is within the half-width w = r z + eps of an integer.  A table holds, for each bucket of
// f and each class of w (quarters of the largest), the offsets that count for some f and w in them.
#pragma once

#include <cmath>

#include "fg_rng.cuh"

namespace fg {

constexpr int kPhaseBuckets = 64, kPhaseClasses = 4;
// Words of both axes' tables with nw words an entry: [axis][class][bucket][word].
FG_HDC int phase_table_words(int nw) { return 2 * kPhaseClasses * kPhaseBuckets * nw; }

FG_HD int phase_bucket(float v) {  // v = z gx - 0.5: the fraction is exact, and so is its product with 64
    const int b = (int)((v - floorf(v)) * (float)kPhaseBuckets);
    return b < kPhaseBuckets - 1 ? b : kPhaseBuckets - 1;
}
// class_scale = kPhaseClasses / the largest half-width; class c holds half-widths up to (c + 1) / class_scale
// (the rounding of w * class_scale moves a half-width by 2^-22 of it at most: phase_mask_word's slack)
FG_HD int phase_class(float w, float class_scale) {
    const int c = (int)(w * class_scale);
    return c < kPhaseClasses - 1 ? c : kPhaseClasses - 1;
}
// Word `word` of a table entry: oz[e] is z o of offset e.
FG_HD uint32_t phase_mask_word(const float *oz, int n, int bucket, int cls, int word, float w_max) {
    const float reach = w_max * (float)(cls + 1) / (float)kPhaseClasses + 0.5f / (float)kPhaseBuckets + 2e-6f;
    const float centre = ((float)bucket + 0.5f) / (float)kPhaseBuckets;
    uint32_t m = 0u;
    for (int e = 32 * word; e < n && e < 32 * word + 32; e++) {
        const float o = oz[e], v = centre + (o - floorf(o));
        if (fabsf(v - rintf(v)) <= reach) m |= 1u << (e & 31);
    }
    return m;
}

}  // namespace fg
