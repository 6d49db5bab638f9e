// Test-only kernels: what the step kernels rest on without a rounding test (ff_exact.cuh:
// decays, sums and derivatives of one float operand) against the double expressions on
// the GPU's FP64 pipe over every float, and whole neuron updates (iz_neuron.cuh) against
// the expressions written in double.  Built by tests/test_gpu_decided.py with nvcc into a
// temporary shared library.
#include <cuda_runtime.h>

#include <cstdint>

#include "iz_neuron.cuh"

namespace {

struct Result {
    unsigned long long mismatches, checked, taken, first;
};

__device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// Which: 0-2 decays by 0.9, 0.95 and 0.933, 3-5 the products with them that decide
// midpoints (and results in the subnormals), 6-7 sums with 0.01 and 0.1, 8 the weight
// derivative without spikes, 9-10 the short-term "w" of "add" and "sub" without one.
__device__ bool taken(int which, float x, float& got, float& want) {
    const double d = x;
    const double c = which % 3 == 0 ? 0.9 : (which % 3 == 1 ? 0.95 : 0.933);
    const double k = which == 6 ? 0.01 : 0.1;
    const float c1 = (float)c, c2 = (float)(c - (double)c1), k1 = (float)k, k2 = (float)(k - (double)k1);
    if (which < 6) {
        want = __double2float_rn(__dmul_rn(d, c));
        return which < 3 ? sg::ff::decay(x, c1, c2, got) : sg::ff::product(x, c1, c2, got, true);
    }
    if (which < 8) {
        want = __double2float_rn(__dadd_rn(d, k));
        return sg::ff::add_const(x, k1, k2, got);
    }
    if (which == 8) {
        want = __double2float_rn(__dsub_rn(d, __dmul_rn(__dsub_rn(d, 0.000001), 0.0001)));
        return sg::ff::weight_decay(x, got);
    }
    const double U = which == 9 ? 0.5 : 0.2, F = which == 9 ? 1000.0 : 20.0;
    want = __double2float_rn(__dadd_rn(d, __ddiv_rn(__dsub_rn(U, d), F)));
    return which == 9 ? sg::ff::short_term_w_rest<false>(x, got) : sg::ff::short_term_w_rest<true>(x, got);
}

__global__ void k_every_float(int which, Result* r) {
    unsigned long long checked = 0, ok = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < (1ull << 32); i += (unsigned long long)gridDim.x * blockDim.x) {
        float got = 0.0f, want;
        ++checked;
        if (!taken(which, __uint_as_float((uint32_t)i), got, want)) continue;
        ++ok;
        if (!same(got, want)) {
            atomicAdd(&r->mismatches, 1ull);
            atomicMin(&r->first, i);
        }
    }
    atomicAdd(&r->checked, checked);
    atomicAdd(&r->taken, ok);
}

__device__ uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ float unit(uint64_t z) { return (float)((z >> 11) & 0xFFFFFF) * (1.0f / 16777216.0f); }

// izhikevich_attributes.cpp:140-183 and spnet_attributes.cpp:96-140, as written.
__device__ void iz_reference(float& v, float& u, float ampa, float nmda, float ga, float gb, float mf,
                             float base, float a, float b) {
    const float sum_c = ampa + nmda + ga + gb;
    for (int i = 0; i < 10 && v < 30.0; ++i) {
        float current = -ampa * v;
        float q = (v + 80) / 60, t = q * q;
        current -= nmda * (t / (1 + t)) * v;
        current -= ga * (v + 70);
        current -= gb * (v + 90);
        current *= 1 + mf;
        current += base;
        const float dv = (0.04 * v * v) + (5 * v) + 140 - u + current;
        v = (v + 0.1 * (dv + (ga * -70) + (gb * -90))) / (1 + (0.1 * sum_c));
        v = v != v ? 30.0f : v;
        const float tau = v > 30.0 ? dv / (30.0 - v + dv) * 0.1 : 0.1;
        u += a * tau * ((b * v) - u);
    }
}
__device__ void spnet_reference(float& v, float& u, float current, float a, float b) {
    for (int i = 0; i < 10 && v < 30.0; ++i) {
        const float dv = (0.04 * v * v) + (5 * v) + 140 - u + current;
        v += dv * 0.1;
        v = v != v ? 30.0f : v;
        const float tau = v > 30.0 ? dv / (30.0 - v + dv) * 0.1 : 0.1;
        u += a * tau * ((b * v) - u);
    }
}

// Random neurons: at rest to a relative 2^-k or anywhere, quiet or driven, reset or
// about to spike, and what is not finite.
__global__ void k_neurons(bool spnet, unsigned long long n, unsigned long long seed, Result* r) {
    unsigned long long checked = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        uint64_t z = mix(seed * 0x100000001B3ull + i);
        auto next = [&] { return z = mix(z); };
        const uint32_t kind = (uint32_t)(next() >> 58);
        const bool fast = next() & 1, quiet = kind < 24;
        const float a = fast ? 0.1f : 0.02f, b = fast ? 0.2f : 0.25f;
        float v = kind % 4 == 0 ? -65.0f : -90.0f + 125.0f * unit(next());
        const float current = quiet ? 0.0f : (unit(next()) - 0.3f) * exp2f(8.0f * unit(next()));
        float u = -20.0f + 40.0f * unit(next());
        if (kind % 8 < 4) {                       // the derivative's terms cancel
            const double rest = (0.04 * v * v) + (5 * v) + 140 + current;
            u = (float)(rest * (1.0 + ldexp((double)unit(next()) - 0.5, -(int)(next() >> 59))));
        }
        auto conductance = [&] { return quiet || (next() & 1) ? 0.0f : exp2f(-12.0f + 14.0f * unit(next())); };
        float ampa = conductance(), nmda = conductance(), ga = conductance(), gb = conductance();
        if (kind == 63) (next() & 1 ? v : u) = next() & 1 ? __uint_as_float(0x7FC00000u) : -INFINITY;
        if (kind == 62) ga = INFINITY;
        const float mf = next() & 1 ? 0.0f : unit(next());
        float v1 = v, u1 = u, v2 = v, u2 = u;
        if (spnet) {
            sg::spnet_integrate_ff(v1, u1, current, a, b);
            spnet_reference(v2, u2, current, a, b);
        } else {
            sg::iz_integrate_ff(v1, u1, ampa, nmda, ga, gb, mf, current, a, b);
            iz_reference(v2, u2, ampa, nmda, ga, gb, mf, current, a, b);
        }
        ++checked;
        if (!same(v1, v2) || !same(u1, u2)) {
            atomicAdd(&r->mismatches, 1ull);
            atomicMin(&r->first, i);
        }
    }
    atomicAdd(&r->checked, checked);
}

template <class F>
int run(unsigned long long* out, F&& launch) {
    Result h = {0, 0, 0, ~0ull}, *d = nullptr;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 1;
    cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
    launch(d);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    out[0] = h.mismatches;
    out[1] = h.checked;
    out[2] = h.taken;
    out[3] = h.first;
    return e == cudaSuccess ? 0 : 2;
}

}  // namespace

extern "C" {

int check_every_float(int which, unsigned long long* out) {
    return run(out, [&](Result* d) { k_every_float<<<152 * 8, 256>>>(which, d); });
}

int check_neurons(int spnet, unsigned long long n, unsigned long long seed, unsigned long long* out) {
    return run(out, [&](Result* d) { k_neurons<<<152 * 8, 256>>>(spnet != 0, n, seed, d); });
}

}  // extern "C"
