// Host checks of ff_exact.cuh (built with -ffp-contract=off): decays over every mantissa
// of a binade, and the voltage of a substep as the neuron kernels decide it.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "ff_exact.cuh"

namespace {
uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
float value(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
struct Draw {
    uint64_t z;
    uint64_t next() {
        uint64_t x = (z += 0x9E3779B97F4A7C15ull);
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        return x ^ (x >> 31);
    }
    float unit() { return (float)(next() >> 40) / 16777216.0f; }
};
}  // namespace

// Mismatches of the decay by c over every float of [2^exponent, 2^(exponent + 1)) and
// its negatives; *taken counts those decided.
extern "C" unsigned long long check_decay(double c, int exponent, unsigned long long* taken) {
    const float c1 = (float)c, c2 = (float)(c - (double)c1);
    unsigned long long bad = 0, ok = 0;
    for (uint32_t m = 0; m < 1u << 24; ++m) {
        const float x = value((m >> 23) << 31 | (uint32_t)(127 + exponent) << 23 | (m & 0x7FFFFFu));
        float got;
        if (!sg::ff::decay(x, c1, c2, got)) continue;
        ++ok;
        bad += bits(got) != bits((float)((double)x * c));
    }
    *taken = ok;
    return bad;
}

// Voltages of substeps: recovery within a relative 2^-spread of the value where the
// derivative's terms cancel, with conductances or (`quiet`) none.  *taken counts those
// decided without the double expressions, *near those of them whose derivative is not known.
extern "C" unsigned long long check_substep(int izhikevich, int quiet, int spread, unsigned long long seed,
                                            unsigned long long n, unsigned long long* taken,
                                            unsigned long long* near) {
    Draw d{seed};
    unsigned long long bad = 0, ok = 0, unknown = 0;
    for (unsigned long long i = 0; i < n; ++i) {
        const float v = -80.0f + 30.0f * d.unit(), current = quiet ? 0.0f : 20.0f * d.unit() - 5.0f;
        const double rest = (0.04 * v * v) + (5 * v) + 140 + current;
        const float u = (float)(rest * (1.0 + std::ldexp((double)d.unit() - 0.5, -spread)));
        const float delta = (float)((0.04 * v * v) + (5 * v) + 140 - u + current);
        float f, g, B, got, want;
        const bool known = sg::ff::iz_delta_v(v, u, current, f, g, B);
        if (known) bad += bits(f) != bits(delta);
        bool decided;
        if (izhikevich) {
            const float ga = quiet ? 0.0f : d.unit(), gb = quiet ? 0.0f : 0.1f * d.unit(), sum = ga + gb;
            const float x = ga * -70, y = gb * -90;
            float d1, d2;
            sg::ff::iz_denominator(sum, d1, d2);
            decided = sg::ff::iz_voltage_of(v, f, g, B, known, x, y, d1, d2, 1.0f / d1, got);
            const float drive = delta + x + y;
            want = (float)(((double)v + 0.1 * (double)drive) / (1.0 + 0.1 * (double)sum));
        } else {
            decided = sg::ff::spnet_voltage_of(v, f, g, B, known, got);
            want = (float)((double)v + (double)delta * 0.1);
        }
        ok += decided;
        unknown += decided && !known;
        bad += decided && bits(got) != bits(want);
    }
    *taken = ok;
    *near = unknown;
    return bad;
}
