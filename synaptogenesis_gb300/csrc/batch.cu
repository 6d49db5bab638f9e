// Batched Izhikevich instances.
//
// Hundreds of independent networks, each with the plain Izhikevich topology:
// a relay layer (FLOAT output, driven each step by value-with-probability-rate
// input) feeding an Izhikevich layer of the same shape through a wrapping
// convergent "add" connection (field x field, stride 1, offset -field/2), plus
// a recurrent fully connected "sub" connection on the Izhikevich layer with
// per-synapse delays.  Sizes, seeds and parameters differ per instance.
//
// Everything random is a counter-based function of the instance seed
// (counter_rng.h), so the same instance can be built as an ordinary network
// for the layer-by-layer path and its spike raster compared bit for bit.
//
// Per step, ONE persistent kernel advances every instance.  Its work units are
// tiles of (tile_rows x 32*tile_colblocks) destination neurons of one
// instance; CTAs take units from an atomic counter, largest first.  A unit:
//   1. stages the instance's output words of step t-1 in shared memory, and
//      the relay outputs of step t-1 (regenerated from the seed) for the
//      tile's rows plus the kernel halo;
//   2. convergent activation: per destination (one lane), the reference's
//      trace activator over k = 0..K-1 (izhikevich_attributes.cpp:228-352);
//   3. recurrent activation over the destination's non-zero synapses in
//      ascending source order.  A synapse of weight 0 keeps zero traces and
//      adds +0.0 to a non-negative sum, so skipping it is exact;
//   4. the neuron update (izhikevich_attributes.cpp:102-213) and the BIT
//      output shift, written to the other half of a ping-pong word buffer so
//      no unit reads a word another unit of the same step has written.
// Nothing in the kernel waits on another CTA: the last CTA to finish resets
// the unit counter and advances the device step counter, which the next
// launch reads.  Launches are captured in CUDA graphs.
//
// Storage.  Destinations are grouped 32 to a "group" (one image row, 32
// consecutive columns); each warp of a unit owns one group.  The recurrent
// synapses of a group are an ELL block: slot s of lane l holds the lane's
// s-th non-zero synapse {source | delay << 27, weight x short-term factors}
// in fc_in and its {short, long} traces in fc_tr, at (base + s) * 32 + l,
// padded with zero synapses to the group's largest count.  Convergent
// per-synapse data is [group][k][lane].
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/syngen.h"
#include "counter_rng.h"
#include "cuda_check.h"
#include "iz_neuron.cuh"
#include "launch.cuh"
#include "props.h"

namespace sg {
void set_last_error(const char* what);
}

namespace {
using namespace sg;

struct InstDev {
    int rows, cols, n, cblocks;
    int field, K;
    float a, b, c, d;
    float rate, value, gconv, gfc;
    float v0, conv_wmax, conv_factor, fc_wmax, fc_density, fc_factor;
    int fc_delays;        // delays are uniform in [0, fc_delays)
    int pad;
    unsigned long long seed;
    long long neuron_off, group_off;
};

struct Unit {
    int inst, row0, cb0, cost;
};

struct StepArgs {
    const InstDev* inst;
    const Unit* units;
    int n_units;
    int tile_rows, tile_cblocks;
    int words_cap;
    const long long* group_base;
    const int* group_slots;
    const uint2* fc_in;
    float2* fc_tr;
    const float* conv_ew;
    float2* conv_tr;
    float* v;
    float* u;
    uint32_t* words;      // [2][n_neurons]
    long long n_neurons;
    int* ctr;
    int* done;
    long long* step;
};

// Trace decays of the "add" (AMPA, NMDA) and "sub" (GABA-A, GABA-B) activators.
constexpr float kAmpaTau = 0.8f, kNmdaTau = 0.993f, kGabaaTau = 0.833f, kGababTau = 0.993f;
constexpr int kConvUnroll = 8;
constexpr int kMaxThreads = 256;

// Wrapped coordinate for x in [-n, 2n) (the field is checked against the
// layer size at creation); equal to ((x % n) + n) % n there.
__device__ __forceinline__ int wrap1(int x, int n) { return x < 0 ? x + n : (x >= n ? x - n : x); }

__device__ __forceinline__ float relay_value(const InstDev& I, long long t, int j) {
    return rng_uniform(I.seed, RNG_INPUT, (unsigned long long)t * I.n + j) < I.rate ? I.value
                                                                                    : 0.0f;
}

// A unit's source words and the relay values around its rows, by all threads.
__device__ __forceinline__ void stage_unit(const InstDev& I, int row0, int tile_rows, long long t,
                                           const uint32_t* __restrict__ words_in, uint32_t* sm,
                                           float* relay) {
    const int relay_rows = tile_rows + I.field - 1;
#pragma unroll 4
    for (int i = threadIdx.x; i < I.n; i += blockDim.x) sm[i] = words_in[I.neuron_off + i];
    for (int e = threadIdx.x; e < relay_rows * I.cols; e += blockDim.x) {
        int rr = e / I.cols, cc = e - rr * I.cols;
        int fr = wrap1(row0 - I.field / 2 + rr, I.rows);
        relay[e] = t > 0 ? relay_value(I, t - 1, fr * I.cols + cc) : 0.0f;
    }
}

// Neuron update; conductances were cleared by the previous update, so each is 0 +
// this step's sum; the layer's input current is 0.
__device__ __forceinline__ void batch_neuron(const StepArgs& A, const InstDev& I, int local,
                                             float s_sum, float l_sum, float f_sum, float fl_sum,
                                             const uint32_t* sm, uint32_t* words_out) {
    const long long nid = I.neuron_off + local;
    float voltage = A.v[nid], recovery = A.u[nid];
    iz_integrate_ff(voltage, recovery, 0.0f + s_sum, 0.0f + l_sum, 0.0f + f_sum, 0.0f + fl_sum,
                    0.0f, 0.0f, I.a, I.b);
    unsigned int spike = voltage >= 30.0;
    words_out[nid] = (sm[local] >> 1) | (spike << 31);
    A.v[nid] = spike ? I.c : voltage;
    A.u[nid] = recovery + (spike * I.d);
}

// The last CTA to finish sets the unit counter and the step for the next launch.
__device__ __forceinline__ void batch_step_done(const StepArgs& A, long long t) {
    __threadfence();
    if (atomicAdd(A.done, 1) == (int)gridDim.x - 1) {
        *A.ctr = 0;
        *A.done = 0;
        *A.step = t + 1;
        __threadfence();
    }
}

// kFcUnroll slots of a lane are loaded while as many are summed, two CTAs to an SM.
// HBM bounds a batch that fills the GPU, so what counts is bytes in flight: 64
// instances of 16..128 a side take 2.74 ms a step with 8 slots and 2 CTAs (6.0 TB/s
// without padding), 2.97 with 16 and 1, 3.43 with 4 and 3, and took 3.41 with 4 slots
// whose trace stores held back the next loads.  (With few groups:
// k_batch_step_split.)
constexpr int kFcUnroll = 8;

__global__ void __launch_bounds__(kMaxThreads, 2) k_batch_step(StepArgs A) {
    extern __shared__ uint32_t sm[];
    __shared__ int s_unit;
    __shared__ long long s_t;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    wait_for_previous();
    if (tid == 0) s_t = *A.step;
    __syncthreads();
    const long long t = s_t;
    const uint32_t* words_in = A.words + (t & 1) * A.n_neurons;
    uint32_t* words_out = A.words + ((t + 1) & 1) * A.n_neurons;
    float* relay = reinterpret_cast<float*>(sm + A.words_cap);

    for (;;) {
        if (tid == 0) s_unit = atomicAdd(A.ctr, 1);
        __syncthreads();
        const int ui = s_unit;
        if (ui >= A.n_units) break;
        const Unit U = A.units[ui];
        const InstDev I = A.inst[U.inst];
        const int h = I.field / 2;
        const int tile_rows = min(A.tile_rows, I.rows - U.row0);
        stage_unit(I, U.row0, tile_rows, t, words_in, sm, relay);
        __syncthreads();

        const int tr = warp / A.tile_cblocks, tcb = warp - tr * A.tile_cblocks;
        const int gr = U.row0 + tr, gcb = U.cb0 + tcb;
        const int col = gcb * 32 + lane;
        if (tr < tile_rows && gcb < I.cblocks && col < I.cols) {
            const long long g = I.group_off + (long long)gr * I.cblocks + gcb;

            // convergent relay -> Izhikevich, "add": AMPA (short) and NMDA (long)
            float s_sum = 0.0f, l_sum = 0.0f;
            {
                const float* ew = A.conv_ew + g * I.K * 32 + lane;
                float2* ct = A.conv_tr + g * I.K * 32 + lane;
                const float* rrow = relay + tr * I.cols;
                for (int k0 = 0, kc = 0; k0 < I.K; k0 += kConvUnroll) {
                    float spike[kConvUnroll], weight[kConvUnroll];
                    float2 x[kConvUnroll];
#pragma unroll
                    for (int j = 0; j < kConvUnroll; ++j) {
                        if (k0 + j >= I.K) break;
                        spike[j] = rrow[wrap1(col - h + kc, I.cols)];
                        weight[j] = __ldg(ew + (k0 + j) * 32);
                        x[j] = ct[(k0 + j) * 32];
                        if (++kc == I.field) {
                            kc = 0;
                            rrow += I.cols;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kConvUnroll; ++j) {
                        if (k0 + j >= I.K) break;
                        const float st = x[j].x + (spike[j] * weight[j] * I.gconv);
                        s_sum += st;
                        const float lt = x[j].y + (spike[j] * weight[j] * I.gconv);
                        l_sum += lt;
                        ct[(k0 + j) * 32] = make_float2(st * kAmpaTau, lt * kNmdaTau);
                    }
                }
            }

            // recurrent fully connected, "sub": GABA-A (short) and GABA-B
            // (long).  The next kFcUnroll slots are loaded before this lot is
            // summed and stored: the loads are the bound, and the compiler
            // may not move them over the trace stores itself.
            float f_sum = 0.0f, fl_sum = 0.0f;
            {
                const long long base = A.group_base[g];
                const int slots = A.group_slots[g];
                const uint2* in = A.fc_in + base * 32 + lane;
                float2* trp = A.fc_tr + base * 32 + lane;
                const float gf = I.gfc;
                uint2 x[2][kFcUnroll];
                float2 y[2][kFcUnroll];
                auto load = [&](int s, uint2 (&xx)[kFcUnroll], float2 (&yy)[kFcUnroll]) {
#pragma unroll
                    for (int j = 0; j < kFcUnroll; ++j)
                        if (s + j < slots) {
                            xx[j] = __ldg(in + (long long)(s + j) * 32);
                            yy[j] = trp[(long long)(s + j) * 32];
                        }
                };
                auto use = [&](int s, const uint2 (&xx)[kFcUnroll], const float2 (&yy)[kFcUnroll]) {
#pragma unroll
                    for (int j = 0; j < kFcUnroll; ++j) {
                        if (s + j >= slots) break;
                        const uint32_t word = sm[xx[j].x & 0x07FFFFFFu];
                        const float spike = (float)((word << (xx[j].x >> 27)) >> 31);
                        const float weight = __uint_as_float(xx[j].y);
                        const float st = yy[j].x + (spike * weight * gf);
                        f_sum += st;
                        const float lt = yy[j].y + (spike * weight * gf);
                        fl_sum += lt;
                        trp[(long long)(s + j) * 32] = make_float2(st * kGabaaTau, lt * kGababTau);
                    }
                };
                load(0, x[0], y[0]);
                for (int s = 0; s < slots; s += 2 * kFcUnroll) {
                    load(s + kFcUnroll, x[1], y[1]);
                    use(s, x[0], y[0]);
                    load(s + 2 * kFcUnroll, x[0], y[0]);
                    use(s + kFcUnroll, x[1], y[1]);
                }
            }

            batch_neuron(A, I, gr * I.cols + col, s_sum, l_sum, f_sum, fl_sum, sm, words_out);
        }
        __syncthreads();
    }

    if (tid == 0) batch_step_done(A, t);
}

// The same step with a CTA of kParts + 1 warps to a group of 32 destinations: kParts
// take the slots in turn, kPartSlots each a round, store their traces and put them in
// shared memory; the last adds the round's in slot order, a round behind, and updates
// the neurons.  For batches too small to fill the GPU, where a group's own chain
// bounds the step (500 slots of 18 instructions in one warp, 6 cycles each) and then
// its neurons' substeps.  12 instances of 16..48 take 29 us a step with 7 + 1 warps,
// 32 with two groups of 3 + 1 in a CTA, 40 with 15 + 1, and took 41 with a warp a
// group and 8 groups a CTA.  Against the best tile of k_batch_step (us a step): 23 / 27 for
// 512 groups of 32 x 32 instances, 37 / 37 for 768, 54 / 46 for 1024; 72 / 111, 109 / 118
// and 145 / 132 for as many of 64 x 64, 61 / 70 for 768 of 48 x 48; 8.5 / 15.6 for 256
// groups of 16 x 16, 21 / 15 for 640; 249 / 382 for the 512 of one 128 x 128 instance,
// 1657 / 1064 for the 1152 of one 192 x 192, one CTA of which fills an SM.
constexpr int kParts = 7, kPartSlots = 4, kRound = kParts * kPartSlots;
constexpr int kPartAhead = 4;            // rounds whose loads are in flight
constexpr int kSplitThreads = (kParts + 1) * 32;

__global__ void __launch_bounds__(kSplitThreads, 2) k_batch_step_split(StepArgs A) {
    extern __shared__ uint32_t sm[];
    __shared__ float2 tile[2][kRound][32];                 // pre-decay traces of a round
    __shared__ int s_unit;
    __shared__ long long s_t;
    const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
    float* relay = reinterpret_cast<float*>(sm + A.words_cap);

    long long t = -1;
    // the first unit is the CTA's own; what is left is taken in turn
    for (int ui = blockIdx.x; ui < A.n_units;) {
        const Unit U = A.units[ui];
        const InstDev I = A.inst[U.inst];
        const int h = I.field / 2;
        const int col = U.cb0 * 32 + lane;
        const bool on = col < I.cols;
        const long long g = I.group_off + (long long)U.row0 * I.cblocks + U.cb0;
        const int slots = A.group_slots[g];
        const long long base = A.group_base[g];
        const uint2* in = A.fc_in + base * 32 + lane;
        float2* trp = A.fc_tr + base * 32 + lane;
        uint2 x[kPartAhead][kPartSlots];
        float2 y[kPartAhead][kPartSlots];
        auto load_in = [&](int r, uint2 (&xx)[kPartSlots]) {
            const int s = r * kRound + part * kPartSlots;
#pragma unroll
            for (int j = 0; j < kPartSlots; ++j)
                if (on && s + j < slots) xx[j] = __ldg(in + (s + j) * 32);
        };
        auto load_tr = [&](int r, float2 (&yy)[kPartSlots]) {
            const int s = r * kRound + part * kPartSlots;
#pragma unroll
            for (int j = 0; j < kPartSlots; ++j)
                if (on && s + j < slots) yy[j] = trp[(s + j) * 32];
        };
        if (part < kParts) {
#pragma unroll
            for (int q = 0; q < kPartAhead; ++q) load_in(q, x[q]);
        }
        if (t < 0) {
            // the layout and the synapses do not change; the rest is the last step's
            wait_for_previous();
            if (tid == 0) s_t = *A.step;
            __syncthreads();
            t = s_t;
        }
        const uint32_t* words_in = A.words + (t & 1) * A.n_neurons;
        uint32_t* words_out = A.words + ((t + 1) & 1) * A.n_neurons;
        if (part < kParts) {
#pragma unroll
            for (int q = 0; q < kPartAhead; ++q) load_tr(q, y[q]);
        }
        stage_unit(I, U.row0, 1, t, words_in, sm, relay);
        __syncthreads();
        const int fc_rounds = (slots + kRound - 1) / kRound;
        const int conv_rounds = (I.K + kRound - 1) / kRound;
        if (part < kParts) {
            // convergent relay -> Izhikevich, "add": AMPA (short) and NMDA (long)
            const float* ew = A.conv_ew + g * I.K * 32 + lane;
            float2* ct = A.conv_tr + g * I.K * 32 + lane;
            int b = 0;
            for (int r = 0; r < conv_rounds; ++r, b ^= 1) {
                const int k0 = r * kRound + part * kPartSlots;
                float weight[kPartSlots];
                float2 c[kPartSlots];
#pragma unroll
                for (int j = 0; j < kPartSlots; ++j)
                    if (on && k0 + j < I.K) {
                        weight[j] = __ldg(ew + (k0 + j) * 32);
                        c[j] = ct[(k0 + j) * 32];
                    }
#pragma unroll
                for (int j = 0; j < kPartSlots; ++j)
                    if (on && k0 + j < I.K) {
                        const int kr = (k0 + j) / I.field, kc = k0 + j - kr * I.field;
                        const float spike = relay[kr * I.cols + wrap1(col - h + kc, I.cols)];
                        const float st = c[j].x + (spike * weight[j] * I.gconv);
                        const float lt = c[j].y + (spike * weight[j] * I.gconv);
                        tile[b][part * kPartSlots + j][lane] = make_float2(st, lt);
                        ct[(k0 + j) * 32] = make_float2(st * kAmpaTau, lt * kNmdaTau);
                    }
                __syncthreads();
            }
            // recurrent fully connected, "sub": GABA-A (short) and GABA-B (long)
            const float gf = I.gfc;
            for (int r = 0; r < fc_rounds; r += kPartAhead) {
#pragma unroll
                for (int q = 0; q < kPartAhead; ++q) {
                    if (r + q >= fc_rounds) break;
                    const int s = (r + q) * kRound + part * kPartSlots;
#pragma unroll
                    for (int j = 0; j < kPartSlots; ++j)
                        if (on && s + j < slots) {
                            const uint32_t word = sm[x[q][j].x & 0x07FFFFFFu];
                            const float spike = (float)((word << (x[q][j].x >> 27)) >> 31);
                            const float weight = __uint_as_float(x[q][j].y);
                            const float st = y[q][j].x + (spike * weight * gf);
                            const float lt = y[q][j].y + (spike * weight * gf);
                            tile[b][part * kPartSlots + j][lane] = make_float2(st, lt);
                            trp[(s + j) * 32] = make_float2(st * kGabaaTau, lt * kGababTau);
                        }
                    load_in(r + q + kPartAhead, x[q]);
                    load_tr(r + q + kPartAhead, y[q]);
                    __syncthreads();
                    b ^= 1;
                }
            }
        } else {
            float sum[4] = {};
            int b = 0;
            auto add = [&](int n, float& s0, float& s1) {
                __syncthreads();
                float2 v[kRound];
#pragma unroll
                for (int i = 0; i < kRound; ++i) v[i] = tile[b][i][lane];
#pragma unroll
                for (int i = 0; i < kRound; ++i)
                    if (i < n) {
                        s0 += v[i].x;
                        s1 += v[i].y;
                    }
                b ^= 1;
            };
            for (int r = 0; r < conv_rounds; ++r) add(I.K - r * kRound, sum[0], sum[1]);
            for (int r = 0; r < fc_rounds; ++r) add(slots - r * kRound, sum[2], sum[3]);
            if (on)
                batch_neuron(A, I, U.row0 * I.cols + col, sum[0], sum[1], sum[2], sum[3], sm, words_out);
        }
        if ((int)gridDim.x >= A.n_units) break;
        if (tid == 0) s_unit = (int)gridDim.x + atomicAdd(A.ctr, 1);
        __syncthreads();
        ui = s_unit;
    }
    if (tid == 0) batch_step_done(A, t);
}

// Group of warp-global index gw: its instance, image row and column.
struct GroupPos {
    const InstDev* I;
    int gr, col;
};

__device__ __forceinline__ GroupPos group_pos(const InstDev* inst, const int* group_inst,
                                              long long gw, int lane) {
    const InstDev* I = inst + group_inst[gw];
    long long lg = gw - I->group_off;
    GroupPos p;
    p.I = I;
    p.gr = (int)(lg / I->cblocks);
    p.col = (int)(lg - (long long)p.gr * I->cblocks) * 32 + lane;
    return p;
}

// Recurrent weight of (to, from): U(0, fc_wmax) kept with probability
// fc_density, else 0.
__device__ __forceinline__ float fc_weight(const InstDev& I, unsigned long long idx) {
    if (!(rng_uniform(I.seed, RNG_FC_MASK, idx) < I.fc_density)) return 0.0f;
    return rng_uniform(I.seed, RNG_FC_WEIGHT, idx) * I.fc_wmax;
}

// Non-zero recurrent synapses per destination: the group's slot count is the
// largest of its lanes.
__global__ void k_batch_count(const InstDev* inst, const int* group_inst, long long n_groups,
                              int* group_slots, unsigned long long* total) {
    long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (gw >= n_groups) return;
    GroupPos p = group_pos(inst, group_inst, gw, lane);
    const InstDev& I = *p.I;
    int cnt = 0;
    if (p.col < I.cols) {
        unsigned long long row = (unsigned long long)(p.gr * I.cols + p.col) * I.n;
        for (int from = 0; from < I.n; ++from) cnt += fc_weight(I, row + from) != 0.0f;
    }
    int mx = __reduce_max_sync(0xFFFFFFFFu, cnt);
    unsigned long long sum = __reduce_add_sync(0xFFFFFFFFu, (unsigned)cnt);
    if (lane == 0) {
        group_slots[gw] = mx;
        atomicAdd(total, sum);
    }
}

__global__ void k_batch_fill(const InstDev* inst, const int* group_inst, long long n_groups,
                             const long long* group_base, const int* group_slots, uint2* fc_in,
                             float2* fc_tr) {
    long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (gw >= n_groups) return;
    GroupPos p = group_pos(inst, group_inst, gw, lane);
    const InstDev& I = *p.I;
    uint2* in = fc_in + group_base[gw] * 32 + lane;
    float2* tr = fc_tr + group_base[gw] * 32 + lane;
    const int slots = group_slots[gw];
    int k = 0;
    if (p.col < I.cols) {
        unsigned long long row = (unsigned long long)(p.gr * I.cols + p.col) * I.n;
        for (int from = 0; from < I.n; ++from) {
            float w = fc_weight(I, row + from);
            if (w == 0.0f) continue;
            uint32_t delay = rng_below(I.seed, RNG_FC_DELAY, row + from, (uint32_t)I.fc_delays);
            // weight x (short term R x short term w), with R = 1
            float ew = w * (1.0f * I.fc_factor);
            in[(long long)k * 32] = make_uint2((uint32_t)from | (delay << 27), __float_as_uint(ew));
            tr[(long long)k * 32] = make_float2(0.0f, 0.0f);
            ++k;
        }
    }
    for (; k < slots; ++k) {
        in[(long long)k * 32] = make_uint2(0u, 0u);
        tr[(long long)k * 32] = make_float2(0.0f, 0.0f);
    }
}

// Convergent weights U(0, conv_wmax) x (R = 1 x short term w) and zero traces;
// lanes past the row's end hold zeros.
__global__ void k_batch_conv_init(const InstDev* inst, const int* group_inst, long long n_groups,
                                  int K, float* conv_ew, float2* conv_tr) {
    long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (gw >= n_groups) return;
    GroupPos p = group_pos(inst, group_inst, gw, lane);
    const InstDev& I = *p.I;
    for (int k = 0; k < I.K; ++k) {
        float ew = 0.0f;
        if (p.col < I.cols) {
            unsigned long long to = (unsigned long long)(p.gr * I.cols + p.col);
            float w = rng_uniform(I.seed, RNG_CONV_WEIGHT, to * I.K + k) * I.conv_wmax;
            ew = w * (1.0f * I.conv_factor);
        }
        conv_ew[(gw * K + k) * 32 + lane] = ew;
        conv_tr[(gw * K + k) * 32 + lane] = make_float2(0.0f, 0.0f);
    }
}

__global__ void k_batch_neuron_init(const InstDev* inst, int n_inst, float* v, float* u) {
    int i = blockIdx.y;
    if (i >= n_inst) return;
    const InstDev& I = inst[i];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < I.n; j += gridDim.x * blockDim.x) {
        v[I.neuron_off + j] = I.v0;
        u[I.neuron_off + j] = I.b * I.v0;
    }
}

template <class T>
T* dalloc(size_t n, std::vector<void*>& owned) {
    void* p = nullptr;
    SG_CUDA(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
    owned.push_back(p);
    return static_cast<T*>(p);
}

struct TuneResult {
    int tile_rows, tile_cblocks;
    float ms;
};

class Batch {
  public:
    Batch(const SgBatchInstance* spec, int count, int tile_rows, int tile_cblocks) {
        if (!spec || count <= 0) throw SgError("batch: no instances");
        validate(spec, count);
        SG_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
        SG_CUDA(cudaGetDevice(&device_));
        SG_CUDA(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, device_));
        SG_CUDA(cudaDeviceGetAttribute(&smem_optin_, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                       device_));
        layout(spec, count);
        generate();
        // counters, words and neurons start defined before the autotuner's
        // real steps (device allocations are not cleared)
        reset();
        if (tile_rows > 0 && tile_cblocks > 0) {
            set_tile(tile_rows, tile_cblocks);
        } else {
            autotune();
        }
        reset();
    }

    ~Batch() {
        if (graph_) cudaGraphExecDestroy(graph_);
        for (void* p : owned_) cudaFree(p);
        if (stream_) cudaStreamDestroy(stream_);
    }

    void step(long long n) {
        while (n >= kGraphSteps) {
            if (!graph_) capture();
            SG_CUDA(cudaGraphLaunch(graph_, stream_));
            n -= kGraphSteps;
            steps_ += kGraphSteps;
            launches_ += kGraphSteps;
        }
        for (; n > 0; --n) {
            launch();
            ++steps_;
            ++launches_;
        }
    }

    void read(int i, const std::string& key, void* out, long long count) {
        if (i < 0 || i >= (int)inst_.size()) throw SgError("batch: instance out of range");
        const InstDev& I = inst_[i];
        if (count < I.n) throw SgError("batch: output buffer smaller than the layer");
        SG_CUDA(cudaStreamSynchronize(stream_));
        const void* src;
        if (key == "voltage") src = v_ + I.neuron_off;
        else if (key == "recovery") src = u_ + I.neuron_off;
        else if (key == "output") src = words_ + (steps_ & 1) * n_neurons_ + I.neuron_off;
        else throw SgError("batch: unknown key " + key);
        SG_CUDA(cudaMemcpy(out, src, (size_t)I.n * 4, cudaMemcpyDeviceToHost));
    }

    Props* report() const {
        auto* r = new Props();
        r->set("instances", std::to_string(inst_.size()));
        r->set("neurons", std::to_string(n_neurons_));
        r->set("groups", std::to_string(n_groups_));
        r->set("slot rows", std::to_string(slot_rows_));
        r->set("fc synapses", std::to_string(fc_synapses_));
        r->set("fc slots", std::to_string(slot_rows_ * 32));
        r->set("conv synapses", std::to_string(conv_synapses_));
        r->set("device bytes", std::to_string(device_bytes_));
        r->set("step bytes", std::to_string(step_bytes()));
        r->set("tile rows", std::to_string(tile_rows_));
        r->set("tile colblocks", std::to_string(tile_cblocks_));
        r->set("units", std::to_string(units_h_.size()));
        r->set("grid", std::to_string(grid_));
        r->set("threads", std::to_string(threads_));
        r->set("shared bytes", std::to_string(smem_));
        r->set("steps", std::to_string(steps_));
        r->set("kernel launches", std::to_string(launches_));
        r->set("graph steps", std::to_string(kGraphSteps));
        for (const TuneResult& t : tuning_) {
            Props c;
            c.set("tile rows", std::to_string(t.tile_rows));
            c.set("tile colblocks", std::to_string(t.tile_cblocks));
            c.set("ms per step", std::to_string(t.ms));
            r->add_to_child_array("autotune", c);
        }
        return r;
    }

    cudaStream_t stream() const { return stream_; }

  private:
    static constexpr int kGraphSteps = 32;

    static void validate(const SgBatchInstance* s, int count) {
        for (int i = 0; i < count; ++i) {
            const SgBatchInstance& x = s[i];
            std::string who = "batch: instance " + std::to_string(i) + ": ";
            if (x.rows < 1 || x.cols < 1) throw SgError(who + "empty layer");
            if ((long long)x.rows * x.cols > (1 << 24)) throw SgError(who + "layer too large");
            if (x.conv_field < 1 || x.conv_field / 2 >= x.rows || x.conv_field / 2 >= x.cols)
                throw SgError(who + "convergent field must satisfy 1 <= field and field/2 < rows, cols");
            if (x.fc_max_delay < 0 || x.fc_max_delay > 31)
                throw SgError(who + "delays must lie in 0..31");
            if (!(x.input_rate >= 0.0f && x.input_rate <= 1.0f))
                throw SgError(who + "input rate must lie in [0, 1]");
            if (!(x.fc_density >= 0.0f && x.fc_density <= 1.0f))
                throw SgError(who + "density must lie in [0, 1]");
        }
    }

    void layout(const SgBatchInstance* spec, int count) {
        long long noff = 0, goff = 0;
        for (int i = 0; i < count; ++i) {
            const SgBatchInstance& s = spec[i];
            InstDev I{};
            I.rows = s.rows;
            I.cols = s.cols;
            I.n = s.rows * s.cols;
            I.cblocks = (s.cols + 31) / 32;
            I.field = s.conv_field;
            I.K = s.conv_field * s.conv_field;
            I.a = s.a; I.b = s.b; I.c = s.c; I.d = s.d;
            I.rate = s.input_rate;
            I.value = s.input_value;
            I.gconv = s.conv_conductance;
            I.gfc = s.fc_conductance;
            I.v0 = s.v0;
            I.conv_wmax = s.conv_wmax;
            I.conv_factor = s.conv_stp_w;
            I.fc_wmax = s.fc_wmax;
            I.fc_density = s.fc_density;
            I.fc_factor = s.fc_stp_w;
            I.fc_delays = s.fc_max_delay + 1;
            I.seed = s.seed;
            I.neuron_off = noff;
            I.group_off = goff;
            noff += I.n;
            goff += (long long)I.rows * I.cblocks;
            max_n_ = std::max(max_n_, I.n);
            max_cols_ = std::max(max_cols_, I.cols);
            max_field_ = std::max(max_field_, I.field);
            max_cblocks_ = std::max(max_cblocks_, I.cblocks);
            max_rows_ = std::max(max_rows_, I.rows);
            if (i > 0 && I.K != inst_[0].K) throw SgError("batch: every instance needs the same field");
            conv_synapses_ += (long long)I.n * I.K;
            inst_.push_back(I);
        }
        n_neurons_ = noff;
        n_groups_ = goff;
        K_ = inst_[0].K;
        group_inst_h_.resize(n_groups_);
        for (size_t i = 0; i < inst_.size(); ++i)
            for (long long g = 0; g < (long long)inst_[i].rows * inst_[i].cblocks; ++g)
                group_inst_h_[inst_[i].group_off + g] = (int)i;
    }

    void generate() {
        d_inst_ = dalloc<InstDev>(inst_.size(), owned_);
        d_group_inst_ = dalloc<int>(n_groups_, owned_);
        d_group_slots_ = dalloc<int>(n_groups_, owned_);
        d_group_base_ = dalloc<long long>(n_groups_, owned_);
        d_counters_ = dalloc<long long>(4, owned_);
        v_ = dalloc<float>(n_neurons_, owned_);
        u_ = dalloc<float>(n_neurons_, owned_);
        words_ = dalloc<uint32_t>(2 * n_neurons_, owned_);
        conv_ew_ = dalloc<float>(n_groups_ * K_ * 32, owned_);
        conv_tr_ = dalloc<float2>(n_groups_ * K_ * 32, owned_);
        // Every upload goes through stream_ (non-blocking): a plain cudaMemcpy
        // from pageable memory may return before its DMA lands and is not
        // ordered with this stream's kernels.
        SG_CUDA(cudaMemcpyAsync(d_inst_, inst_.data(), inst_.size() * sizeof(InstDev),
                                cudaMemcpyHostToDevice, stream_));
        SG_CUDA(cudaMemcpyAsync(d_group_inst_, group_inst_h_.data(), n_groups_ * sizeof(int),
                                cudaMemcpyHostToDevice, stream_));
        unsigned long long* total = reinterpret_cast<unsigned long long*>(d_counters_ + 3);
        SG_CUDA(cudaMemsetAsync(total, 0, sizeof(unsigned long long), stream_));
        unsigned blocks = blocks_for(n_groups_ * 32, 256);
        k_batch_count<<<blocks, 256, 0, stream_>>>(d_inst_, d_group_inst_, n_groups_,
                                                   d_group_slots_, total);
        SG_LAUNCH_CHECK();
        group_slots_h_.resize(n_groups_);
        SG_CUDA(cudaMemcpyAsync(group_slots_h_.data(), d_group_slots_, n_groups_ * sizeof(int),
                                cudaMemcpyDeviceToHost, stream_));
        unsigned long long nz = 0;
        SG_CUDA(cudaMemcpyAsync(&nz, total, sizeof(nz), cudaMemcpyDeviceToHost, stream_));
        SG_CUDA(cudaStreamSynchronize(stream_));
        fc_synapses_ = (long long)nz;
        std::vector<long long> base(n_groups_);
        long long acc = 0;
        for (long long g = 0; g < n_groups_; ++g) {
            base[g] = acc;
            acc += group_slots_h_[g];
        }
        slot_rows_ = acc;
        SG_CUDA(cudaMemcpyAsync(d_group_base_, base.data(), n_groups_ * sizeof(long long),
                                cudaMemcpyHostToDevice, stream_));
        fc_in_ = dalloc<uint2>(slot_rows_ * 32, owned_);
        fc_tr_ = dalloc<float2>(slot_rows_ * 32, owned_);
        k_batch_fill<<<blocks, 256, 0, stream_>>>(d_inst_, d_group_inst_, n_groups_, d_group_base_,
                                                  d_group_slots_, fc_in_, fc_tr_);
        SG_LAUNCH_CHECK();
        k_batch_conv_init<<<blocks, 256, 0, stream_>>>(d_inst_, d_group_inst_, n_groups_, K_,
                                                       conv_ew_, conv_tr_);
        SG_LAUNCH_CHECK();
        SG_CUDA(cudaStreamSynchronize(stream_));
        device_bytes_ = 0;
        device_bytes_ += inst_.size() * sizeof(InstDev) + n_groups_ * (4 + 4 + 8) + 32;
        device_bytes_ += n_neurons_ * 16;
        device_bytes_ += n_groups_ * K_ * 32 * 12;
        device_bytes_ += slot_rows_ * 32 * 16;
    }

    // Bytes one step must move: recurrent slots (read 16, write 8), convergent
    // synapses (read 12, write 8) and neurons (voltage, recovery read and
    // written, output word read and written).
    long long step_bytes() const {
        return slot_rows_ * 32 * 24 + n_groups_ * K_ * 32 * 20 + n_neurons_ * 24;
    }

    // Trace state, neurons, output words and counters back to their initial
    // values (after autotuning, which runs real steps).
    void reset() {
        SG_CUDA(cudaMemsetAsync(fc_tr_, 0, slot_rows_ * 32 * sizeof(float2), stream_));
        SG_CUDA(cudaMemsetAsync(conv_tr_, 0, n_groups_ * K_ * 32 * sizeof(float2), stream_));
        SG_CUDA(cudaMemsetAsync(words_, 0, 2 * n_neurons_ * sizeof(uint32_t), stream_));
        SG_CUDA(cudaMemsetAsync(d_counters_, 0, 3 * sizeof(long long), stream_));
        dim3 grid(std::max(1, std::min(64, (max_n_ + 255) / 256)), (unsigned)inst_.size());
        k_batch_neuron_init<<<grid, 256, 0, stream_>>>(d_inst_, (int)inst_.size(), v_, u_);
        SG_LAUNCH_CHECK();
        SG_CUDA(cudaStreamSynchronize(stream_));
        steps_ = 0;
        launches_ = 0;
    }

    // The units of every instance, unit_rows_ x unit_cblocks_ groups each.
    void make_units() {
        units_h_.clear();
        for (size_t i = 0; i < inst_.size(); ++i) {
            const InstDev& I = inst_[i];
            for (int r0 = 0; r0 < I.rows; r0 += unit_rows_)
                for (int c0 = 0; c0 < I.cblocks; c0 += unit_cblocks_) {
                    long long cost = 0;
                    for (int r = r0; r < std::min(I.rows, r0 + unit_rows_); ++r)
                        for (int c = c0; c < std::min(I.cblocks, c0 + unit_cblocks_); ++c)
                            cost += group_slots_h_[I.group_off + (long long)r * I.cblocks + c] + I.K;
                    cost += I.n / 32 + 1;
                    units_h_.push_back(Unit{(int)i, r0, c0, (int)std::min<long long>(cost, 1 << 30)});
                }
        }
    }

    // The most dynamic shared memory that `kernel` can be launched with.  The limit is
    // the function's, shared by every batch of the process: always the largest, or a
    // smaller batch would lower it for a larger one.
    size_t allow_shared(void (*kernel)(StepArgs)) {
        cudaFuncAttributes fa;
        SG_CUDA(cudaFuncGetAttributes(&fa, kernel));
        const int most = smem_optin_ - (int)fa.sharedSizeBytes;
        SG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        return (size_t)most;
    }
    // CTAs of k_batch_step_split that the GPU holds, 0 if one does not fit.
    long long split_places(size_t smem) {
        if (smem > allow_shared(k_batch_step_split)) return 0;
        int per_sm = 0;
        SG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_step_split,
                                                              kSplitThreads, smem));
        return (long long)per_sm * num_sms_;
    }

    void set_tile(int tile_rows, int tile_cblocks) {
        if (tile_rows < 1 || tile_cblocks < 1 || tile_rows * tile_cblocks * 32 > kMaxThreads)
            throw SgError("batch: tile must have 1..8 warps");
        tile_rows_ = tile_rows;
        tile_cblocks_ = tile_cblocks;
        words_cap_ = (max_n_ + 3) / 4 * 4;
        unit_rows_ = tile_rows;
        unit_cblocks_ = tile_cblocks;
        make_units();
        auto shared = [&](int rows) {
            return (size_t)(words_cap_ + (rows + max_field_ - 1) * max_cols_) * 4;
        };
        if ((int)shared(tile_rows) > smem_optin_)
            throw SgError("batch: instance too large for shared memory");
        // several warps to a group, whatever the tile, up to three groups for each CTA that
        // the GPU holds (two to an SM, fewer beside large instances), two where a group's
        // slots are so few that a CTA's start outweighs them: k_batch_step_split
        const int rounds = slot_rows_ >= 128 * n_groups_ ? 3 : 2;
        const bool split = n_groups_ <= rounds * split_places(shared(1));
        if (split) {
            unit_rows_ = unit_cblocks_ = 1;
            make_units();
        }
        threads_ = split ? kSplitThreads : tile_rows * tile_cblocks * 32;
        smem_ = shared(unit_rows_);
        std::stable_sort(units_h_.begin(), units_h_.end(),
                         [](const Unit& a, const Unit& b) { return a.cost > b.cost; });
        if (!d_units_ || units_h_.size() > units_cap_) {
            units_cap_ = std::max(units_h_.size(), (size_t)(n_groups_ + 1));
            d_units_ = dalloc<Unit>(units_cap_, owned_);
        }
        SG_CUDA(cudaMemcpyAsync(d_units_, units_h_.data(), units_h_.size() * sizeof(Unit),
                                cudaMemcpyHostToDevice, stream_));
        kernel_ = split ? k_batch_step_split : k_batch_step;
        allow_shared(kernel_);
        int per_sm = 0;
        SG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_, threads_, smem_));
        if (per_sm < 1) throw SgError("batch: step kernel does not fit on an SM");
        grid_ = (int)std::min<long long>((long long)units_h_.size(), (long long)per_sm * num_sms_);
        if (graph_) {
            cudaGraphExecDestroy(graph_);
            graph_ = nullptr;
        }
    }

    StepArgs args() const {
        StepArgs a;
        a.inst = d_inst_;
        a.units = d_units_;
        a.n_units = (int)units_h_.size();
        a.tile_rows = unit_rows_;
        a.tile_cblocks = unit_cblocks_;
        a.words_cap = words_cap_;
        a.group_base = d_group_base_;
        a.group_slots = d_group_slots_;
        a.fc_in = fc_in_;
        a.fc_tr = fc_tr_;
        a.conv_ew = conv_ew_;
        a.conv_tr = conv_tr_;
        a.v = v_;
        a.u = u_;
        a.words = words_;
        a.n_neurons = n_neurons_;
        a.ctr = reinterpret_cast<int*>(d_counters_);
        a.done = reinterpret_cast<int*>(d_counters_ + 1);
        a.step = d_counters_ + 2;
        return a;
    }

    void launch() {
        launch_dependent(kernel_, grid_, threads_, smem_, stream_, args());
    }

    void capture() {
        cudaGraph_t g;
        SG_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
        for (int i = 0; i < kGraphSteps; ++i) launch();
        SG_CUDA(cudaStreamEndCapture(stream_, &g));
        cudaError_t e = cudaGraphInstantiate(&graph_, g, 0);
        cudaGraphDestroy(g);
        SG_CUDA(e);
    }

    // Tile shapes with 4 or 8 warps, each timed over a few real steps; the
    // fastest is kept.  The state is reset afterwards.
    void autotune() {
        std::vector<std::pair<int, int>> cands;
        for (int warps : {8, 4})
            for (int tc = 1; tc <= warps; tc *= 2) {
                int tr = warps / tc;
                if (tc > max_cblocks_ && tc > 1) continue;
                if (tr > max_rows_ && tr > 1) continue;
                cands.push_back({tr, tc});
            }
        cudaEvent_t e0, e1;
        SG_CUDA(cudaEventCreate(&e0));
        SG_CUDA(cudaEventCreate(&e1));
        float best = 1e30f;
        std::pair<int, int> pick = cands.front();
        for (auto& c : cands) {
            set_tile(c.first, c.second);
            launch();
            SG_CUDA(cudaEventRecord(e0, stream_));
            const int reps = 3;
            for (int i = 0; i < reps; ++i) launch();
            SG_CUDA(cudaEventRecord(e1, stream_));
            SG_CUDA(cudaEventSynchronize(e1));
            float ms = 0.0f;
            SG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            ms /= reps;
            tuning_.push_back(TuneResult{c.first, c.second, ms});
            if (ms < best) {
                best = ms;
                pick = c;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        set_tile(pick.first, pick.second);
    }

    std::vector<InstDev> inst_;
    std::vector<int> group_inst_h_, group_slots_h_;
    std::vector<Unit> units_h_;
    std::vector<TuneResult> tuning_;
    std::vector<void*> owned_;
    int unit_rows_ = 1, unit_cblocks_ = 1;
    long long n_neurons_ = 0, n_groups_ = 0, slot_rows_ = 0, fc_synapses_ = 0;
    long long conv_synapses_ = 0, device_bytes_ = 0, steps_ = 0, launches_ = 0;
    int max_n_ = 0, max_cols_ = 0, max_rows_ = 0, max_field_ = 0, max_cblocks_ = 0, K_ = 0;
    int tile_rows_ = 0, tile_cblocks_ = 0, threads_ = 0, grid_ = 0, words_cap_ = 0;
    size_t smem_ = 0, units_cap_ = 0;
    void (*kernel_)(StepArgs) = nullptr;
    int device_ = 0, num_sms_ = 0, smem_optin_ = 0;
    cudaStream_t stream_ = nullptr;
    cudaGraphExec_t graph_ = nullptr;
    InstDev* d_inst_ = nullptr;
    int* d_group_inst_ = nullptr;
    int* d_group_slots_ = nullptr;
    long long* d_group_base_ = nullptr;
    long long* d_counters_ = nullptr;   // unit counter, done counter, step, synapse total
    Unit* d_units_ = nullptr;
    float *v_ = nullptr, *u_ = nullptr;
    uint32_t* words_ = nullptr;
    float* conv_ew_ = nullptr;
    float2* conv_tr_ = nullptr;
    uint2* fc_in_ = nullptr;
    float2* fc_tr_ = nullptr;
};

}  // namespace

extern "C" {

SG_BATCH sg_batch_create(const SgBatchInstance* instances, int count, int tile_rows,
                         int tile_colblocks) {
    try {
        return new Batch(instances, count, tile_rows, tile_colblocks);
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    } catch (...) {
        sg::set_last_error("unknown error");
    }
    return nullptr;
}

int sg_batch_step(SG_BATCH b, long long steps) {
    if (!b || steps < 0) return SG_BATCH_EINVAL;
    try {
        static_cast<Batch*>(b)->step(steps);
        return 0;
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return SG_BATCH_ECUDA;
}

int sg_batch_read(SG_BATCH b, int instance, const char* key, void* out, long long count) {
    if (!b || !key || !out) return SG_BATCH_EINVAL;
    try {
        static_cast<Batch*>(b)->read(instance, key, out, count);
        return 0;
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return SG_BATCH_EINVAL;
}

PROPS sg_batch_report(SG_BATCH b) {
    if (!b) return nullptr;
    try {
        return static_cast<Batch*>(b)->report();
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return nullptr;
}

void* sg_batch_stream(SG_BATCH b) { return b ? (void*)static_cast<Batch*>(b)->stream() : nullptr; }

int sg_batch_synchronize(SG_BATCH b) {
    if (!b) return SG_BATCH_EINVAL;
    return cudaStreamSynchronize(static_cast<Batch*>(b)->stream()) == cudaSuccess ? 0
                                                                                  : SG_BATCH_ECUDA;
}

void sg_batch_destroy(SG_BATCH b) {
    try {
        delete static_cast<Batch*>(b);
    } catch (...) {
    }
}

}  // extern "C"
