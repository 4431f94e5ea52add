// Checks the samplers on the 32-bit pipes (poisson_count, knuth_count_f32, lognormal_radius_f32) against the
// f64 samplers: the same value and the same stream position on every stream tried.  Prints
// "<checked> <mismatches> <f64 decisions>" for the Poisson counts, the cells' Knuth counts and the radii.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
static long g_exact = 0, g_fallbacks = 0;
#define FG_EXACT_HOOK() (++g_exact)
#define FG_EXP_FALLBACK_HOOK() (++g_fallbacks)
#include "fg_rng.cuh"

using namespace fg;

static bool same(const Xoshiro &a, const Xoshiro &b) { return memcmp(&a, &b, sizeof a) == 0; }

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    uint64_t st = 2024;
    auto hash = [&] { st += kPhi; return fmix64(st); };

    // both regimes and their border, the ends of the f32 rejection's range
    const float lambdas[] = {1e-4f, 0.03f, 0.7f, 3.0f, 7.5f, 11.0f, 11.999999f, 12.0f, 12.5f, 13.25f, 17.0f, 24.7f,
                             60.0f, 139.0f, 439.3f, 1405.9f, 7029.5f, 20000.25f, 65535.9f, 65536.0f, 300000.0f};
    long checked = 0, bad = 0, exact = 0;
    for (float lam : lambdas) {
        for (long i = 0; i < n; i++) {
            const uint64_t h = hash();
            Xoshiro want_rng = small_seed(h), rng;
            const uint32_t want = poisson_sample(poisson_new((double)lam), want_rng);
            g_exact = 0;
            const uint32_t got = poisson_count(h, lam, rng);
            if (lam < 65536.0f) exact += g_exact;
            checked++;
            if (got != want || !same(rng, want_rng)) {
                if (bad < 5) std::printf("lambda %g: %u, want %u\n", lam, got, want);
                bad++;
            }
        }
    }
    std::printf("%ld %ld %ld\n", checked, bad, exact);

    checked = bad = exact = 0;
    const double exps[] = {0.9999, 0.9, 0.37, 0.05, 0.0123};
    for (double e : exps) {
        const long long thresh = (long long)(e * 9007199254740992.0);
        for (long i = 0; i < 4 * n; i++) {
            const uint64_t h = hash();
            Xoshiro rng = small_seed(h), want_rng = rng;
            const uint64_t first = rng.next();
            if ((long long)(first >> 11) <= thresh) continue;
            (void)want_rng.next();
            const uint32_t want = poisson_knuth_tail(u53_unit(first >> 11), e, want_rng);
            uint32_t got = 0;
            checked++;
            const float ef = (float)(uint32_t)(thresh >> 21) * 2.3283064365386963e-10f;
            if (!knuth_count_f32<true>(unit_f32(first), ef, rng, got)) exact++;
            else if (got != want || !same(rng, want_rng)) bad++;
        }
    }
    std::printf("%ld %ld %ld\n", checked, bad, exact);

    checked = bad = exact = 0;
    const float laws[][2] = {{-3.1073041f, 0.47238073f}, {-3.7630f, 0.38525f}, {0.0f, 0.2f}, {-0.01f, 1.7f}, {2.0f, 3.9f},
                             {-5.0f, 4.5f}, {-2.3025851f, 0.0f}};
    for (const auto &law : laws) {
        Xoshiro rng = small_seed(hash()), want_rng = rng;
        for (long i = 0; i < 20 * n; i++) {
            const float want = exp_f64_to_f32(normal_sample((double)law[0], (double)law[1], want_rng));
            g_exact = 0;
            const float got = lognormal_radius_f32(law[0], law[1], rng);
            exact += g_exact;
            checked++;
            if (memcmp(&got, &want, 4) != 0 || !same(rng, want_rng)) {
                if (bad < 5) std::printf("law %g %g: %a, want %a\n", law[0], law[1], got, want);
                bad++;
                rng = want_rng;
            }
        }
    }
    std::printf("%ld %ld %ld\n", checked, bad, exact);
    return 0;
}
