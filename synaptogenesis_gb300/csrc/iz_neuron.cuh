// Neuron integration: Izhikevich (src/core/state/impl/izhikevich_attributes.cpp:102-213),
// shared by the per-layer update kernel and the batched instance runner, and spnet
// (spnet_attributes.cpp:96-166).
#pragma once

#include "exact_convert.cuh"
#include "ff_exact.cuh"

namespace sg {

#ifdef __CUDACC__
// The substep's three double expressions evaluated in double, one at a time:
// taken where the float-float evaluation's rounding test fails (rarely; out of
// line so that the other lanes branch around the FP64 instructions).
static __device__ __noinline__ float iz_delta_v_double(float voltage, float recovery,
                                                       float current) {
    const double vd = f2d_exact(voltage);
    double dv = __dmul_rn(mul_df_rn(voltage, 0.04), vd);
    dv = __dadd_rn(dv, f2d_exact(5 * voltage));
    dv = __dadd_rn(dv, 140.0);
    dv = __dsub_rn(dv, f2d_exact(recovery));
    dv = __dadd_rn(dv, f2d_exact(current));
    return d2f_rn(dv);
}

static __device__ __noinline__ float iz_voltage_double(float voltage, float drive, float sum_c) {
    const double den = __dadd_rn(1.0, mul_df_rn(sum_c, 0.1));
    return d2f_rn(__ddiv_rn(__dadd_rn(f2d_exact(voltage), mul_df_rn(drive, 0.1)), den));
}

static __device__ __noinline__ float iz_tau_double(float voltage, float delta_v) {
    return (float)(delta_v / (30.0 - voltage + delta_v) * 0.1);
}

// Up to 10 hybrid-Euler substeps that stop once v >= 30 (NaN -> 30), with the
// conductance-implicit voltage update and the recovery step whose time constant is
// adjusted on the substep that crosses threshold: the reference's operations in its
// types and order (the double literals make the voltage arithmetic double).  Each double
// expression is evaluated in float-float arithmetic (ff_exact.cuh) and its float result
// taken where the rounding test proves it equal to the double evaluation.  The
// derivative's test fails where its terms cancel (near rest, and on the first substep
// after a reset); the voltage is then decided from the unrounded derivative
// (iz_voltage_of).  What is left is evaluated in double.  A substep that changes neither
// voltage nor recovery would be repeated by the rest, which are left out.
__device__ __forceinline__ void iz_integrate_ff(float& voltage, float& recovery, float ampa_c,
                                                float nmda_c, float gabaa_c, float gabab_c,
                                                float mf, float base_current, float a, float b) {
    if (!(voltage < 30.0f)) return;
    const float sum_c = ampa_c + nmda_c + gabaa_c + gabab_c;
    float d1, d2;
    ff::iz_denominator(sum_c, d1, d2);        // 1 + 0.1 * sum_c ~ d1 + d2
    const float rd = 1.0f / d1;
    for (int i = 0; (i < 10) && (voltage < 30.0f); ++i) {
        float current = -ampa_c * voltage;
        float q = ff::div_int<60>(voltage + 80);
        float temp = q * q;
        current -= nmda_c * (temp / (1 + temp)) * voltage;
        current -= gabaa_c * (voltage + 70);
        current -= gabab_c * (voltage + 90);
        current *= 1 + mf;
        current += base_current;
        float delta_v, tail, bound, nv;
        const bool known = ff::iz_delta_v(voltage, recovery, current, delta_v, tail, bound);
        const float x = gabaa_c * -70, y = gabab_c * -90;
        if (!ff::iz_voltage_of(voltage, delta_v, tail, bound, known, x, y, d1, d2, rd, nv)) {
            if (!known) delta_v = iz_delta_v_double(voltage, recovery, current);
            nv = iz_voltage_double(voltage, delta_v + x + y, sum_c);
        }
        const float v0 = voltage, r0 = recovery;
        voltage = (nv != nv) ? 30.0f : nv;
        float adjusted_tau = (float)0.1;
        if (voltage > 30.0f && !ff::iz_adjusted_tau(voltage, delta_v, adjusted_tau))
            adjusted_tau = iz_tau_double(voltage, delta_v);
        recovery += a * adjusted_tau * ((b * voltage) - recovery);
        // at rest: the remaining substeps would repeat this one
        if (voltage == v0 && recovery == r0) break;
    }
}

// spnet's double expressions in double, where a rounding test fails.
static __device__ __noinline__ float spnet_delta_double(float voltage, float recovery, float current) {
    return (0.04 * voltage * voltage) + (5 * voltage) + 140 - recovery + current;
}
static __device__ __noinline__ float spnet_voltage_double(float voltage, float delta_v) {
    return voltage + delta_v * 0.1;
}

// spnet's substeps, likewise.
__device__ __forceinline__ void spnet_integrate_ff(float& voltage, float& recovery, float current,
                                                   float a, float b) {
    for (int i = 0; (i < 10) && (voltage < 30.0f); ++i) {
        float delta_v, tail, bound, nv;
        const bool known = ff::iz_delta_v(voltage, recovery, current, delta_v, tail, bound);
        if (!ff::spnet_voltage_of(voltage, delta_v, tail, bound, known, nv)) {
            if (!known) delta_v = spnet_delta_double(voltage, recovery, current);
            nv = spnet_voltage_double(voltage, delta_v);
        }
        const float v0 = voltage, r0 = recovery;
        voltage = (nv != nv) ? 30.0f : nv;
        float adjusted_tau = (float)0.1;
        if (voltage > 30.0f && !ff::iz_adjusted_tau(voltage, delta_v, adjusted_tau))
            adjusted_tau = iz_tau_double(voltage, delta_v);
        recovery += a * adjusted_tau * ((b * voltage) - recovery);
        if (voltage == v0 && recovery == r0) break;          // at rest
    }
}
#endif

}  // namespace sg
