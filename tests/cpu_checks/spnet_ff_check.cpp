// Host checks of expressions of ff_exact.cuh (spnet's, products with short
// decimals, voltage steps near rest) against the double expressions they stand for (built with -ffp-contract=off): wherever the
// rounding test accepts, the floats are equal bit for bit.  Operands have random
// signs and mantissas and exponents drawn from [lo, hi), a share of them with
// short mantissas, so that sums land on and near rounding boundaries.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "ff_exact.cuh"

namespace {
struct Draw {
    uint64_t z;
    uint64_t next() {
        uint64_t x = (z += 0x9E3779B97F4A7C15ull);
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        return x ^ (x >> 31);
    }
    float value(int lo, int hi) {
        const uint64_t r = next();
        uint32_t m = (uint32_t)r & 0x7FFFFFu;
        if (r >> 60 < 4) m &= 0x7F0000u;
        if (r >> 60 == 15) return 0.0f;
        const uint32_t e = (uint32_t)(127 + lo + (int)((r >> 24) % (uint64_t)(hi - lo)));
        const uint32_t u = ((uint32_t)(r >> 59 & 1) << 31) | e << 23 | m;
        float f;
        std::memcpy(&f, &u, 4);
        return f;
    }
};
uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
}  // namespace

// Voltage steps of neurons near rest: recovery drawn around the value where the
// derivative's terms cancel, to a relative 2^-spread.
extern "C" unsigned long long check_near(int izhikevich, int spread, unsigned long long seed,
                                         unsigned long long n, unsigned long long* accepted) {
    Draw d{seed};
    unsigned long long bad = 0, ok = 0;
    for (unsigned long long i = 0; i < n; ++i) {
        const float v = -80.0f + 30.0f * (float)(d.next() >> 40) / 16777216.0f;
        const bool quiet = d.next() & 1;
        const float ampa = izhikevich && !quiet ? std::fabs(d.value(-12, 1)) : 0.0f;
        const float ga = izhikevich && !quiet ? std::fabs(d.value(-12, 1)) : 0.0f;
        const float gb = izhikevich && !quiet ? std::fabs(d.value(-12, 1)) : 0.0f;
        const float current = quiet ? 0.0f : d.value(-8, 4);
        const double cancel = (0.04 * v * v) + (5 * v) + 140 + current;
        const float recovery = (float)(cancel * (1.0 + std::ldexp((double)d.value(-1, 1), -spread)));
        const float delta = (float)((0.04 * v * v) + (5 * v) + 140 - recovery + current);
        float f, g, B, got, want;
        sg::ff::iz_delta_v_sum(v, recovery, current, f, g, B);
        bool took;
        if (izhikevich) {
            const float sum = ampa + ga + gb, x = ga * -70, y = gb * -90;
            float d1, d2;
            sg::ff::iz_denominator(sum, d1, d2);
            float at, tail = g, err;
            sg::ff::iz_drive_near(f, x, y, B, at, tail, err);
            took = sg::ff::iz_voltage(v, at, d1, d2, 1.0f / d1, got, tail, err) && got <= 30.0f;
            const float drive = delta + x + y;
            want = (float)(((double)v + 0.1 * (double)drive) / (1.0 + 0.1 * (double)sum));
        } else {
            took = sg::ff::spnet_voltage_near(v, f, g, B, got);
            want = (float)((double)v + (double)delta * 0.1);
        }
        ok += took;
        bad += took && bits(got) != bits(want);
    }
    *accepted = ok;
    return bad;
}

// Products with a short decimal, midpoints decided (product's `ties`): p over the
// bit patterns [begin, end), both signs.
extern "C" unsigned long long check_decimal(double c, unsigned begin, unsigned end, unsigned step,
                                            unsigned long long* accepted) {
    const float c1 = (float)c, c2 = (float)(c - (double)c1);
    unsigned long long bad = 0, ok = 0;
    for (unsigned long long u = begin; u < end; u += step)
        for (unsigned sign = 0; sign < 2; ++sign) {
            const unsigned w = (unsigned)u | sign << 31;
            float p, got;
            std::memcpy(&p, &w, 4);
            if (!sg::ff::product(p, c1, c2, got, true)) continue;
            ++ok;
            bad += bits(got) != bits((float)((double)p * c));
        }
    *accepted = ok;
    return bad;
}

// Single-argument expressions over every `step`-th float: 0-2 decays by 0.9, 0.95
// and 0.933, 3-4 sums with 0.01 and 0.1, 5 the weight derivative without spikes, 6-7
// the short-term "w" of "add" and "sub" without one.
extern "C" unsigned long long check_single(int which, unsigned long long begin, unsigned long long step,
                                           unsigned long long* accepted) {
    unsigned long long bad = 0, ok = 0;
#pragma omp parallel for reduction(+ : bad, ok)
    for (long long i = (long long)begin; i < (1ll << 32); i += (long long)step) {
        const uint32_t u = (uint32_t)i;
        float x, got = 0.0f, want;
        std::memcpy(&x, &u, 4);
        const double d = x;
        bool took;
        if (which < 3) {
            const double c = which == 0 ? 0.9 : (which == 1 ? 0.95 : 0.933);
            const float c1 = (float)c;
            took = sg::ff::decay(x, c1, (float)(c - (double)c1), got);
            want = (float)(d * c);
        } else if (which < 5) {
            const double k = which == 3 ? 0.01 : 0.1;
            const float k1 = (float)k;
            took = sg::ff::add_const(x, k1, (float)(k - (double)k1), got);
            want = (float)(d + k);
        } else if (which == 5) {
            took = sg::ff::weight_decay(x, got);
            want = (float)(d - ((d - 0.000001) * 0.0001));
        } else if (which == 6) {
            took = sg::ff::short_term_w_rest<false>(x, got);
            want = (float)(d + (0.5 - d) / 1000);
        } else {
            took = sg::ff::short_term_w_rest<true>(x, got);
            want = (float)(d + (0.2 - d) / 20);
        }
        ok += took;
        bad += took && bits(got) != bits(want);
    }
    *accepted = ok;
    return bad;
}

// Mismatches; *accepted counts the draws the rounding test took.
extern "C" unsigned long long check_spnet(int which, int lo, int hi, unsigned long long seed,
                                          unsigned long long n, unsigned long long* accepted) {
    Draw d{seed};
    unsigned long long bad = 0, ok = 0;
    for (unsigned long long i = 0; i < n; ++i) {
        const float x = d.value(lo, hi), p = d.value(lo, hi), q = d.value(lo, hi);
        float got, want;
        bool took;
        if (which == 0) {
            took = sg::ff::spnet_voltage(x, p, got);
            want = (float)((double)x + (double)p * 0.1);
        } else {
            took = sg::ff::spnet_dw(x, p, q, got);
            want = (float)(0.9 * (double)x + (double)p - (double)q);
        }
        ok += took;
        bad += took && bits(got) != bits(want);
    }
    *accepted = ok;
    return bad;
}
