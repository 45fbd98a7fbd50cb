// Host check of ffmath.cuh's procedural length scale and level weights (float-float with a
// rounding test) against their double evaluations: every value the test accepts must round
// to the double evaluation's float.  Compiled by test_ffscale.py with -ffp-contract=off.
#include "../gpis_extend_gb300/csrc/ffmath.cuh"

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

static uint64_t g_state = 88172645463325252ull;
static float uniform(float lo, float hi)
{
    g_state ^= g_state << 13;
    g_state ^= g_state >> 7;
    g_state ^= g_state << 17;
    return lo + (hi - lo) * (float)((g_state >> 20) & 0xFFFFFF) * 0x1p-24f;
}

int main(int argc, char **argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 2000000;
    long fallback = 0, bad = 0, total = 0;
    const float sets[5][5] = {{0.11f, 0.09f, 3.0f, 2.0f, 2.0f}, {1.0f, 0.5f, 1.0f, 1.0f, 4.0f},
                              {0.2f, -0.19f, 7.0f, 0.0f, 2.0f}, {0.05f, 0.04f, 0.3f, 11.0f, 1.4f},
                              {3.0f, 2.9f, 40.0f, 40.0f, 2.0f}};
    for (const auto &q : sets)
        for (long i = 0; i < n; ++i) {
            float x = uniform(-q[4], q[4]), z = uniform(-q[4], q[4]), got;
            if (i % 97 == 0) x = 0.0f;
            if (i % 101 == 0) x = 1.57079637f / q[2];
            ++total;
            if (!ffm_length_scale(q[0], q[1], q[2], q[3], x, z, got)) {
                fallback += &q != &sets[4];     // (the last set's angles are out of its range)
                continue;
            }
            const float want = (float)((double)q[0] + (double)q[1] * std::sin((double)q[2] * (double)x) *
                                                          std::cos((double)q[3] * (double)z));
            if (ffm_bits(got) != ffm_bits(want) && bad++ < 5)
                std::printf("scale a=%a b=%a x=%a z=%a: %a against %a\n", q[0], q[1], x, z, got, want);
        }
    for (long i = 0; i < 4 * n; ++i) {
        const float f = i < 64 ? std::ldexp(1.0f, -(int)i) : uniform(0.0f, 1.0f);
        float w0, w1;
        ++total;
        if (!ffm_level_weights(f, w0, w1)) {
            ++fallback;
            continue;
        }
        const double d = std::sqrt(1.0 - 2.0 * f + 2.0 * (double)f * f);
        if ((ffm_bits(w0) != ffm_bits((float)((1.0 - f) / d)) || ffm_bits(w1) != ffm_bits((float)(f / d))) && bad++ < 5)
            std::printf("weights f=%a: %a %a\n", f, w0, w1);
    }
    std::printf("checked %ld, fallbacks %ld (%.2e), mismatches %ld\n", total, fallback, (double)fallback / (double)total, bad);
    return bad == 0 && fallback < total / 500 ? 0 : 1;
}
