// Differentiable leaky-integrator rate network: forward cycle and its
// hand-written adjoint (backpropagation through time with checkpoints).
//
// The reference has no differentiable model; its rate_encoding layer
// (src/core/state/impl/rate_encoding_attributes.cpp:14-34) maps input to a
// rate with no memory.  This model gives each neuron a leaky membrane:
//
//   layers l = 0..L-1 of rows x cols neurons (N), batch element b
//   I_0[t]  = x[t]                                     (input sequence)
//   I_l[t]  = sum_k W_l[i][k] * r_{l-1}[t-1][src(i,k)]  (l >= 1, convergent)
//   d_l[t]  = -v_l[t-1] + I_l[t]
//   v_l[t]  = v_l[t-1] + a_l * d_l[t],   a_l = dt / tau_l
//   r_l[t]  = sigmoid(v_l[t]),           v_l[0] = 0
//   y[t]    = R r_{L-1}[t]                             (readout, O outputs)
//   loss    = sum_{t,b,o} (y[t][b][o] - target[b][o])^2 / (T B O)
//
// Convergent connections follow the reference's arborized geometry
// (src/core/engine/kernel/synapse_kernel.h:384-421) with stride 1, spacing 1,
// offset -field/2 and no wrap: out-of-range sources are skipped; weights are
// in the CPU layout [destination][k], k = kernel row * field + kernel column.
// Synchronous update as in the reference's cycle: every layer at t reads the
// rates of t-1.
//
// Adjoint (lambda_l[t] = dloss/dv_l[t]):
//   g_{L-1}[t] = R^T gy[t],  gy[t] = grad_loss * 2 (y[t] - target) / (T B O)
//   g_l[t]     = sum over (j, k) with src(j,k) = i of W_{l+1}[j][k] a_{l+1} lambda_{l+1}[t+1][j]
//   lambda_l[t] = r (1 - r) g_l[t] + (1 - a_l) lambda_l[t+1],  lambda[T+1] = 0
//   dW_l[j][k] = a_l sum_{t,b} lambda_l[t][j] r_{l-1}[t-1][src(j,k)]
//   dR[o][i]   = sum_{t,b} gy[t][o] r_{L-1}[t][i]
//   dtau_l     = -(dt / tau_l^2) sum_{t,b,i} lambda_l[t][i] d_l[t][i]
//   dx[t]      = a_0 lambda_0[t]
// The forward pass stores v every few steps (at least `checkpoint` apart); the
// backward pass recomputes each segment's states from its checkpoint
// (bit-identical: the same kernels on the same inputs), then runs the adjoint
// back through it.  Every sum has a fixed order, and every gradient accumulator
// takes one timestep's sum at a time, so results are deterministic and do not
// depend on the checkpoint stride.
//
// A layer reads only the layer below, one step earlier, and its own state is
// pointwise in time, so a stretch of steps is run layer by layer and not step
// by step: one launch takes a layer through every step of a segment, all of its
// stencils independent but for the pointwise recurrence, which stays in
// registers.  The adjoint runs the same way from the last layer down.  Before, a
// tile's layers ran step by step in one CTA with a barrier per step, recomputing
// halos, and the adjoint took a launch per step: forward and adjoint of 3 x 64x64
// layers, field 5, batch 64, 100 steps took 4.55 ms; 1.83 ms like this (4 x 30x45,
// batch 5, 37 steps: 0.56 and 0.34 ms).
//
// Layout on the device: the convergent weights are transposed once per call
// into the workspace as [layer][k][neuron], so that consecutive threads
// (consecutive neurons) read consecutive weights.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/syngen.h"
#include "cuda_check.h"
#include "launch.cuh"

namespace sg {
void set_last_error(const char* what);
}

namespace {
using namespace sg;

constexpr int kMaxOutputs = 16;
constexpr int kMaxField = 9;
constexpr int kTauBlocks = 64;
constexpr int kBlock = 256;

struct Dims {
    int L, rows, cols, N, field, K, O, B, T, k, nseg, chunk;
    float dt;
    long long BN, S;   // B * N, L * B * N
    long long G;       // gradient elements: (L - 1) * N * K weights, then O * N of the readout
};

// The rate network is checked against an FP64 restatement (not a bit-exact
// reference), so it uses the fast exponential, whose error of up to 2 + 1.173 |v|
// units in the last place is the sigmoid's where exp(-v) outweighs the 1, and
// explicit fused multiply-adds in its sums; the reciprocal is correctly rounded, into
// the subnormals (5 % of a training step over one Newton step from the approximate
// one).  Every kernel is deterministic, so the backward pass recomputes the forward
// states bit for bit.
__device__ __forceinline__ float sigmoid(float v) { return __frcp_rn(1.0f + __expf(-v)); }

// wt[l][k][i] = w[l][i][k]
__global__ void k_rate_transpose(Dims D, const float* __restrict__ w, float* __restrict__ wt) {
    wait_for_previous();
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)(D.L - 1) * D.N * D.K) return;
    const long long per = (long long)D.N * D.K;
    const int l = (int)(idx / per);
    const int rem = (int)(idx - l * per);
    const int k = rem / D.N, i = rem - k * D.N;
    wt[idx] = w[l * per + (long long)i * D.K + k];
}

// ---------------------------------------------------------------------------
// Stencil tiles.  A CTA of kTileWarps warps owns a tile of 32 columns; a thread
// owns PY neurons of one column in consecutive rows, so that the PY + F - 1
// window rows it reads serve F x F terms of every one of them: (PY + F - 1) F
// shared-memory reads for PY F F multiply-adds (0.6 per term at 5 x 5 and
// PY = 2, where a neuron a thread needs 1).  Instruction issue is what bounds
// these kernels, at half to 0.7 of its rate for want of warps: at 5 x 5, two rows (72
// registers, 7 CTAs an SM) took 13.9 us a 10-step launch where four (151, 3 CTAs)
// took 20.1, though four issue fewer instructions (15.8 us with two rows since each
// kernel row is summed by itself and the sigmoid's reciprocal is correctly rounded).
// Everything else in the loop over items (batch element, timestep) is kept short:
// offsets within a layer are 32-bit and worked out once, added to
// bases that are the same for the whole CTA; windows (tile plus halo) come in
// with cp.async, 16 bytes at a time where the layer's rows allow it (V = 4),
// kTileDepth - 1 items ahead, and the part of a window outside the layer (a
// skipped source adds w * 0) is zeroed once and never copied.
// ---------------------------------------------------------------------------
constexpr int kTileWarps = 4;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kTileDepth = 4;

constexpr int tile_py(int field) { return field <= 3 ? 8 : (field <= 7 ? 2 : 1); }

// CTAs an SM should hold of the forward kernel: up to 50 weights fit in 72
// registers, and seven CTAs are one wave of 1024 (3 x 64x64, batch 64, with one chain a
// stencil: 13.9 us a 10-step launch against 14.9 with five).
constexpr int tile_ctas(int field, int py) { return field * field * py <= 50 ? 7 : 1; }

template <int F, int PY, int V>
struct Tile {
    static constexpr int H = F / 2, TY = PY * kTileWarps, WY = TY + 2 * H;
    // columns left of the tile in a window row: whole pieces of V
    static constexpr int LEFT = (H + V - 1) / V * V, WX = 32 + 2 * LEFT;
    static constexpr int COUNT = WY * WX, PIECES = COUNT / V;
    static constexpr int PER = (PIECES + kTileThreads - 1) / kTileThreads;
    int y0, x0, lane, row;                   // the tile; this thread's column, first row in it
    unsigned off[PER];                       // pieces this thread copies,
    unsigned copies;                         // those that lie in the layer,
    unsigned rows_ok;                        // rows of this thread that do,
    unsigned own[PY];                        // and its neurons (0 for the others)

    __device__ Tile(const Dims& D, float (*win)[COUNT]) {
        const int tiles_x = (D.cols + 31) / 32;
        y0 = blockIdx.x / tiles_x * TY;
        x0 = blockIdx.x % tiles_x * 32;
        lane = threadIdx.x & 31;
        row = (threadIdx.x >> 5) * PY;
        rows_ok = copies = 0;
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            const bool in = x0 + lane < D.cols && y0 + row + q < D.rows;
            if (in) rows_ok |= 1u << q;
            own[q] = in ? (unsigned)((y0 + row + q) * D.cols + x0 + lane) : 0u;
        }
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int n = threadIdx.x + e * kTileThreads;
            const int r = y0 - H + n / (WX / V), c = x0 - LEFT + n % (WX / V) * V;
            const bool in = n < PIECES && r >= 0 && r < D.rows && c >= 0 && c < D.cols;
            if (in) copies |= 1u << e;
            off[e] = in ? (unsigned)(r * D.cols + c) : 0u;
            if (n < PIECES && !in)
                for (int s = 0; s < kTileDepth; ++s)
#pragma unroll
                    for (int j = 0; j < V; ++j) win[s][n * V + j] = 0.0f;
        }
    }
    __device__ bool ok(int q) const { return rows_ok >> q & 1u; }
    // one commit group per call, also past the last item (!more)
    __device__ void fetch(float* win, const float* plane, bool more) const {
        if (more) {
#pragma unroll
            for (int e = 0; e < PER; ++e)
                if (copies >> e & 1u) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(
                        win + (threadIdx.x + e * kTileThreads) * V);
                    if (V == 4)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                                     "l"(plane + off[e]) : "memory");
                    else
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst),
                                     "l"(plane + off[e]) : "memory");
                }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // the oldest item's window has landed for every thread, and every thread
    // has read the window before it
    __device__ void wait() const {
        asm volatile("cp.async.wait_group %0;" ::"n"(kTileDepth - 2) : "memory");
        __syncthreads();
    }
    // this thread's corner of a window: the source of its row 0, kernel (0, 0)
    __device__ const float* corner(const float* win) const {
        return win + row * WX + lane + LEFT - H;
    }
};

// The sum of a kernel row's terms.  A stencil adds its rows' sums in order: 2 F
// roundings in a chain and not F x F (over 7 networks and 60 seeds the input's gradient
// errs by 2.275e-7 with row sums and by 2.297e-7 with one chain, which is 3 % faster).
template <int F>
__device__ __forceinline__ float row_sum(const float* w, const float* x) {
    float sum = 0.0f;
#pragma unroll
    for (int kc = 0; kc < F; ++kc) sum = __fmaf_rn(w[kc], x[kc], sum);
    return sum;
}

// One layer l >= 1 through nt steps (c + 1 .. c + nt) for a group of batch
// elements: grid (tiles, batch groups).  src: the rates of layer l - 1 at steps
// c .. c + nt - 1, `src_t` floats apart; r: this layer's rates at c .. c + nt.
struct LayerArgs {
    const float* src;
    long long src_t;
    float* r;
    long long r_t;
    float* d;                // drives of steps c + 1 .. c + nt, S apart, or null
    const float* v0;         // [B][N] at step c, or null (zero)
    float* v1;               // at step c + nt, or null
    float* ckpt;             // checkpoints of this layer, S apart, or null
    int c, nt, bg;
};

template <int F, int PY, int V>
__global__ void __launch_bounds__(kTileThreads, tile_ctas(F, PY)) k_rate_layer(Dims D, int l, LayerArgs A,
                                                             const float* __restrict__ wt,
                                                             const float* __restrict__ tau) {
    using W = Tile<F, PY, V>;
    __shared__ __align__(16) float win[kTileDepth][W::COUNT];
    const W tile(D, win);
    const float a = D.dt / __ldg(tau + l);
    // weights of neurons outside the layer are neuron 0's; nothing they give is stored
    float wk[PY][F * F];
    const float* wl = wt + (long long)(l - 1) * F * F * D.N;
#pragma unroll
    for (int k = 0; k < F * F; ++k, wl += D.N)
#pragma unroll
        for (int q = 0; q < PY; ++q) wk[q][k] = __ldg(wl + tile.own[q]);
    wait_for_previous();
    const int b0 = blockIdx.y * A.bg, b1 = min(D.B, b0 + A.bg);
    const float* src = A.src + (long long)b0 * D.N;          // the next item to fetch
    int pb = b0, pt = 0, slot = 0;
    auto fetch = [&](int into) {
        tile.fetch(win[into], src, pb < b1);
        src += A.src_t;
        if (++pt == A.nt) {
            pt = 0;
            ++pb;
            src += D.N - A.nt * A.src_t;
        }
    };
#pragma unroll
    for (int s = 0; s < kTileDepth - 1; ++s) fetch(s);
    for (int b = b0; b < b1; ++b) {
        const float* v0 = A.v0 ? A.v0 + (long long)b * D.N : nullptr;
        float* r = A.r + (long long)b * D.N;
        float* dd = A.d ? A.d + (long long)b * D.N : nullptr;
        float v[PY];
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            v[q] = v0 ? v0[tile.own[q]] : 0.0f;
            if (tile.ok(q)) r[tile.own[q]] = sigmoid(v[q]);
        }
        int mark = D.k - A.c % D.k;                          // steps to the next checkpoint
        for (int tt = 1; tt <= A.nt; ++tt) {
            tile.wait();
            fetch((slot + kTileDepth - 1) % kTileDepth);
            const float* x = tile.corner(win[slot]);
            slot = (slot + 1) % kTileDepth;
            float I[PY];
#pragma unroll
            for (int q = 0; q < PY; ++q) I[q] = 0.0f;
#pragma unroll
            for (int wr = 0; wr < PY + F - 1; ++wr) {
                float xr[F];
#pragma unroll
                for (int kc = 0; kc < F; ++kc) xr[kc] = x[wr * W::WX + kc];
#pragma unroll
                for (int q = 0; q < PY; ++q) {
                    const int kr = wr - q;
                    if (kr < 0 || kr >= F) continue;
                    I[q] += row_sum<F>(&wk[q][kr * F], xr);
                }
            }
            r += A.r_t;
#pragma unroll
            for (int q = 0; q < PY; ++q) {
                I[q] -= v[q];
                v[q] = v[q] + a * I[q];
                if (tile.ok(q)) r[tile.own[q]] = sigmoid(v[q]);
            }
            if (dd) {
#pragma unroll
                for (int q = 0; q < PY; ++q)
                    if (tile.ok(q)) dd[tile.own[q]] = I[q];
                dd += D.S;
            }
            if (--mark == 0) {
                mark = D.k;
                const int t = A.c + tt;
                if (A.ckpt && t < D.T)
#pragma unroll
                    for (int q = 0; q < PY; ++q)
                        if (tile.ok(q))
                            A.ckpt[t / D.k * D.S + (long long)b * D.N + tile.own[q]] = v[q];
            }
        }
        if (A.v1)
#pragma unroll
            for (int q = 0; q < PY; ++q)
                if (tile.ok(q)) A.v1[(long long)b * D.N + tile.own[q]] = v[q];
    }
}

// Layer 0, driven by x alone: a thread per (batch element, neuron).
constexpr int kAhead = 10;                   // timesteps whose loads are in flight

__global__ void __launch_bounds__(kBlock) k_rate_input(Dims D, LayerArgs A,
                                                       const float* __restrict__ x,
                                                       const float* __restrict__ tau) {
    const long long i = (long long)blockIdx.x * kBlock + threadIdx.x;
    wait_for_previous();
    if (i >= D.BN) return;
    const float a = D.dt / __ldg(tau);
    float v = A.v0 ? A.v0[i] : 0.0f;
    A.r[i] = sigmoid(v);
    const float* xt = x + (long long)A.c * D.BN + i;
    for (int t0 = 0; t0 < A.nt; t0 += kAhead) {
        float in[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            in[u] = t0 + u < A.nt ? __ldg(xt + (t0 + u) * D.BN) : 0.0f;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int tt = t0 + u + 1, t = A.c + tt;
            if (tt > A.nt) break;
            const float d = in[u] - v;
            v = v + a * d;
            A.r[tt * A.r_t + i] = sigmoid(v);
            if (A.d) A.d[(tt - 1) * D.S + i] = d;
            if (A.ckpt && t % D.k == 0 && t < D.T) A.ckpt[t / D.k * D.S + i] = v;
        }
    }
    if (A.v1) A.v1[i] = v;
}

// y[t][b][o] = sum_i R[o][i] r[t][b][i] and the squared error of (t, b), for
// rows (t, b) of a chunk.  A CTA takes kReadRows rows, so that a readout weight
// read from L2 serves all of them, and its warps a slice of the neurons each (V
// consecutive ones to a lane).  A lane sums its neurons in order, a butterfly
// adds the lanes, and the warps are added in order.
constexpr int kReadRows = 8;

// Sums c[] over the warp: of C = 2 * HALF sums a lane keeps half, exchanging the
// other half with the lane M away, and so on down to the neighbour.
template <int HALF, int M = 16, int C>
__device__ __forceinline__ void butterfly(float (&c)[C], int lane) {
    if constexpr (M >= 1) {
        const bool up = lane & M;
#pragma unroll
        for (int e = 0; e < HALF; ++e) {
            const float send = up ? c[e] : c[e + HALF];
            const float keep = up ? c[e + HALF] : c[e];
            c[e] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, M);
        }
        butterfly<HALF / 2, M / 2>(c, lane);
    }
}

template <int V>
__device__ __forceinline__ void load_row(const float* p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        v[0] = *p;
    }
}

template <int V>
__global__ void __launch_bounds__(kBlock, 1) k_rate_readout(Dims D, int c, int nt,
                                                            const float* __restrict__ r,
                                                            long long r_t,
                                                            const float* __restrict__ wo,
                                                            const float* __restrict__ target,
                                                            float* __restrict__ y,
                                                            float* __restrict__ loss_tb) {
    constexpr int C = kReadRows * kMaxOutputs, STEP = 32 * V;
    __shared__ float red[kBlock / 32][C];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long rows = (long long)nt * D.B, row0 = (long long)blockIdx.x * kReadRows;
    const float* src[kReadRows];
#pragma unroll
    for (int j = 0; j < kReadRows; ++j) {
        const long long row = min(row0 + j, rows - 1);
        src[j] = r + (row / D.B + 1) * r_t + row % D.B * D.N;
    }
    float acc[C];
#pragma unroll
    for (int e = 0; e < C; ++e) acc[e] = 0.0f;
    wait_for_previous();
    const int steps = (D.N + STEP - 1) / STEP, per = (steps + kBlock / 32 - 1) / (kBlock / 32);
    const int k1 = min(D.N, (warp + 1) * per * STEP);
    for (int k = warp * per * STEP + lane * V; k < k1; k += STEP) {
        float rv[kReadRows][V];
#pragma unroll
        for (int j = 0; j < kReadRows; ++j) load_row<V>(src[j] + k, rv[j]);
#pragma unroll
        for (int o = 0; o < kMaxOutputs; ++o) {
            if (o >= D.O) break;
            float wv[V];
#pragma unroll
            for (int q = 0; q < V; ++q) wv[q] = __ldg(wo + (long long)o * D.N + k + q);
#pragma unroll
            for (int j = 0; j < kReadRows; ++j)
#pragma unroll
                for (int q = 0; q < V; ++q)
                    acc[j * kMaxOutputs + o] = __fmaf_rn(wv[q], rv[j][q], acc[j * kMaxOutputs + o]);
        }
    }
    butterfly<C / 2>(acc, lane);                             // sums C / 32 * lane and on
#pragma unroll
    for (int e = 0; e < C / 32; ++e) red[warp][lane * (C / 32) + e] = acc[e];
    __syncthreads();
    if (threadIdx.x >= C) return;
    const int j = threadIdx.x / kMaxOutputs, o = threadIdx.x % kMaxOutputs;
    const long long tb = (long long)c * D.B + row0 + j;
    float err = 0.0f;
    if (row0 + j < rows && o < D.O) {
        float sum = 0.0f;
#pragma unroll
        for (int q = 0; q < kBlock / 32; ++q) sum += red[q][threadIdx.x];
        y[tb * D.O + o] = sum;
        err = sum - target[tb % D.B * D.O + o];
        err *= err;
    }
#pragma unroll
    for (int m = kMaxOutputs / 2; m >= 1; m /= 2) err += __shfl_xor_sync(0xFFFFFFFFu, err, m);
    if (o == 0 && row0 + j < rows) loss_tb[tb] = err;
}

// loss = sum over (t, b) of the squared errors / (T B O): 256 strided
// partial sums reduced in a fixed tree.
__global__ void __launch_bounds__(256) k_rate_loss(Dims D, const float* __restrict__ loss_tb,
                                                   float* __restrict__ loss) {
    wait_for_previous();
    __shared__ float sm[256];
    const int tid = threadIdx.x;
    float s = 0.0f;
    for (long long j = tid; j < (long long)D.T * D.B; j += 256) s += loss_tb[j];
    sm[tid] = s;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (tid < k) sm[tid] += sm[tid + k];
        __syncthreads();
    }
    if (tid == 0) *loss = sm[0] / (float)((long long)D.T * D.B * D.O);
}

// gy[t][b][o] = gscale * (y - target), for every step.
__global__ void k_rate_gy(Dims D, float gscale, const float* __restrict__ y,
                          const float* __restrict__ target, float* __restrict__ gy) {
    wait_for_previous();
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)D.T * D.B * D.O) return;
    const long long bo = e % ((long long)D.B * D.O);
    gy[e] = gscale * (y[e] - target[bo]);
}

// ---------------------------------------------------------------------------
// Adjoint of one layer through a segment's steps, last first.  What the layer
// below and the weight gradients read is P_l[t] = a_l lambda_l[t], so that is
// what is stored (P[tt - 1] for step c + tt; for layer 0 it is dx).  lambda
// itself and the sum of lambda d over time stay in registers and cross segments
// in `lam` and `lamd` ([B][N] of this layer).
// ---------------------------------------------------------------------------
struct AdjointArgs {
    const float* r;          // this layer's rates at c .. c + nt, S apart
    const float* d;          // its drives, S apart
    const float* next;       // P_{l+1} of steps c + 1 .. c + nt, S apart
    const float* next_carry; // P_{l+1} of step c + nt + 1
    bool first;              // nothing is carried yet: the carries are zero (next_carry is)
    float* P;                // P_l, P_t apart, or null
    long long P_t;
    float* carry;            // P_l of step c + 1 again, for the segment before, or null
    float *lam, *lamd;
    int nt, bg;
};

struct AdjointNeuron {
    float lam, lamd;
    __device__ float step(float r, float d, float g, float a) {
        lam = r * (1.0f - r) * g + (1.0f - a) * lam;
        lamd = __fmaf_rn(lam, d, lamd);
        return a * lam;
    }
};

// Neuron i of layer l feeds destinations j = i + h - (kr, kc) of layer l + 1:
// the thread keeps those weights, zero where j lies outside the layer.
template <int F, int PY, int V>
__global__ void __launch_bounds__(kTileThreads, tile_ctas(F, PY) > 1 ? 6 : 1) k_rate_adjoint(Dims D, int l, AdjointArgs A,
                                                               const float* __restrict__ wt,
                                                               const float* __restrict__ tau) {
    using W = Tile<F, PY, V>;
    constexpr int H = W::H;
    __shared__ __align__(16) float win[kTileDepth][W::COUNT];
    const W tile(D, win);
    const float a = D.dt / __ldg(tau + l);
    float wk[PY][F * F];
    const float* wl = wt + (long long)l * F * F * D.N;
#pragma unroll
    for (int k = 0; k < F * F; ++k, wl += D.N) {
        const int jc = tile.x0 + tile.lane + H - k % F;
        const bool col = jc >= 0 && jc < D.cols;
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            const int jr = tile.y0 + tile.row + q + H - k / F;
            wk[q][k] = 0.0f;
            if (col && jr >= 0 && jr < D.rows) wk[q][k] = __ldg(wl + (unsigned)(jr * D.cols + jc));
        }
    }
    wait_for_previous();
    const int b0 = blockIdx.y * A.bg, b1 = min(D.B, b0 + A.bg);
    int pb = b0, pt = A.nt, slot = 0;                        // the next item to fetch
    auto fetch = [&](int into) {
        const float* src = (pt == A.nt ? A.next_carry : A.next + pt * D.S) + (long long)pb * D.N;
        tile.fetch(win[into], src, pb < b1);
        if (--pt == 0) { pt = A.nt; ++pb; }
    };
#pragma unroll
    for (int s = 0; s < kTileDepth - 1; ++s) fetch(s);
    for (int b = b0; b < b1; ++b) {
        const long long bn = (long long)b * D.N;
        const float *r = A.r + A.nt * D.S + bn, *dd = A.d + (A.nt - 1) * D.S + bn;
        float* P = A.P ? A.P + (A.nt - 1) * A.P_t + bn : nullptr;
        AdjointNeuron n[PY];
        float p[PY];
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            n[q].lam = A.first ? 0.0f : (A.lam + bn)[tile.own[q]];
            n[q].lamd = A.first ? 0.0f : (A.lamd + bn)[tile.own[q]];
        }
        float rn[PY], dn[PY];                                // the next step's, loaded ahead
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            rn[q] = r[tile.own[q]];
            dn[q] = dd[tile.own[q]];
        }
        for (int tt = A.nt; tt >= 1; --tt) {
            float rv[PY], dv[PY];
            if (tt > 1) {
                r -= D.S;
                dd -= D.S;
            }
#pragma unroll
            for (int q = 0; q < PY; ++q) {
                rv[q] = rn[q];
                dv[q] = dn[q];
                rn[q] = r[tile.own[q]];
                dn[q] = dd[tile.own[q]];
            }
            tile.wait();
            fetch((slot + kTileDepth - 1) % kTileDepth);
            const float* x = tile.corner(win[slot]);
            slot = (slot + 1) % kTileDepth;
            float g[PY];
#pragma unroll
            for (int q = 0; q < PY; ++q) g[q] = 0.0f;
            // window rows from the last, so that kernel rows come in order
#pragma unroll
            for (int wr = PY + F - 2; wr >= 0; --wr) {
                float xr[F];
#pragma unroll
                for (int kc = 0; kc < F; ++kc) xr[kc] = x[wr * W::WX + 2 * H - kc];
#pragma unroll
                for (int q = 0; q < PY; ++q) {
                    const int kr = q + 2 * H - wr;
                    if (kr < 0 || kr >= F) continue;
                    g[q] += row_sum<F>(&wk[q][kr * F], xr);
                }
            }
#pragma unroll
            for (int q = 0; q < PY; ++q) p[q] = n[q].step(rv[q], dv[q], g[q], a);
            if (P) {
#pragma unroll
                for (int q = 0; q < PY; ++q)
                    if (tile.ok(q)) P[tile.own[q]] = p[q];
                P -= A.P_t;
            }
        }
#pragma unroll
        for (int q = 0; q < PY; ++q) {
            if (!tile.ok(q)) continue;
            (A.lam + bn)[tile.own[q]] = n[q].lam;
            (A.lamd + bn)[tile.own[q]] = n[q].lamd;
            if (A.carry) (A.carry + bn)[tile.own[q]] = p[q];
        }
    }
}

// The last layer, driven by the readout: grid (blocks of neurons, batch).
// dloss/dy of kTopSteps steps at a time is kept in shared memory.
constexpr int kTopSteps = 32;

__global__ void __launch_bounds__(kBlock) k_rate_adjoint_top(Dims D, AdjointArgs A,
                                                             const float* __restrict__ wo,
                                                             const float* __restrict__ gy,
                                                             const float* __restrict__ tau) {
    __shared__ __align__(16) float gs[kTopSteps][kMaxOutputs];
    const int i = blockIdx.x * kBlock + threadIdx.x, b = blockIdx.y;
    const bool ok = i < D.N;
    const unsigned own = ok ? i : 0;
    const long long bn = (long long)b * D.N;
    const float a = D.dt / __ldg(tau + D.L - 1);
    float wov[kMaxOutputs];
#pragma unroll
    for (int o = 0; o < kMaxOutputs; ++o) wov[o] = o < D.O ? __ldg(wo + (long long)o * D.N + own) : 0.0f;
    wait_for_previous();
    AdjointNeuron n{A.first ? 0.0f : (A.lam + bn)[own], A.first ? 0.0f : (A.lamd + bn)[own]};
    const float *r = A.r + A.nt * D.S + bn, *d = A.d + (A.nt - 1) * D.S + bn;
    float* P = A.P ? A.P + (A.nt - 1) * A.P_t + bn : nullptr;
    float p = 0.0f;
    for (int t1 = A.nt; t1 >= 1; t1 -= kTopSteps) {
        const int steps = min(kTopSteps, t1);
        float rv[kAhead], dv[kAhead];
        auto load = [&](int u0) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (u0 + u < steps) {
                    rv[u] = r[own];
                    dv[u] = d[own];
                    r -= D.S;
                    d -= D.S;
                }
        };
        load(0);                                             // in flight while gs is staged
        __syncthreads();
        for (int e = threadIdx.x; e < steps * kMaxOutputs; e += kBlock) {
            const int u = e / kMaxOutputs, o = e % kMaxOutputs;
            gs[u][o] = o < D.O ? __ldg(gy + ((long long)(t1 - u - 1) * D.B + b) * D.O + o) : 0.0f;
        }
        __syncthreads();
        for (int u0 = 0; u0 < steps; u0 += kAhead) {
            if (u0 > 0) load(u0);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (u0 + u >= steps) break;
                float g = 0.0f;
#pragma unroll
                for (int o = 0; o < kMaxOutputs; ++o)
                    if (o < D.O) g = __fmaf_rn(wov[o], gs[u0 + u][o], g);
                p = n.step(rv[u], dv[u], g, a);
                if (P) {
                    if (ok) P[own] = p;
                    P -= A.P_t;
                }
            }
        }
    }
    if (!ok) return;
    (A.lam + bn)[own] = n.lam;
    (A.lamd + bn)[own] = n.lamd;
    if (A.carry) (A.carry + bn)[own] = p;
}

// dW of one timestep: grid (tiles, layers >= 1, timesteps of the segment).  A
// thread holds the F x F sums over the batch, in batch order, of its PY neurons'
// P_l[t] times the source rates of t - 1 in their windows.  The step's totals go
// to part[tt][l-1][k][j], and k_rate_dw_acc adds the steps latest first: a fixed
// order that does not depend on where the segments start.
template <int F, int PY, int V>
__global__ void __launch_bounds__(kTileThreads) k_rate_dw(Dims D, const float* __restrict__ seg_P,
                                                          const float* __restrict__ seg_r,
                                                          float* __restrict__ part) {
    using W = Tile<F, PY, V>;
    __shared__ __align__(16) float win[kTileDepth][W::COUNT];
    __shared__ float own[kTileDepth][PY][kTileThreads];      // each thread its own P
    const W tile(D, win);
    const int l = 1 + blockIdx.y, tt = blockIdx.z;
    const float* P = seg_P + tt * D.S + l * D.BN;
    const float* r = seg_r + tt * D.S + (l - 1) * D.BN;
    wait_for_previous();
    float acc[PY][F * F];
#pragma unroll
    for (int q = 0; q < PY; ++q)
#pragma unroll
        for (int k = 0; k < F * F; ++k) acc[q][k] = 0.0f;
    auto fetch = [&](int into, bool more) {
        if (more)
#pragma unroll
            for (int q = 0; q < PY; ++q)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(&own[into][q][threadIdx.x])),
                             "l"(P + tile.own[q]) : "memory");
        tile.fetch(win[into], r, more);
        P += D.N;
        r += D.N;
    };
#pragma unroll
    for (int s = 0; s < kTileDepth - 1; ++s) fetch(s, s < D.B);
    for (int b = 0, slot = 0; b < D.B; ++b) {
        tile.wait();
        fetch((slot + kTileDepth - 1) % kTileDepth, b + kTileDepth - 1 < D.B);
        float p[PY];
#pragma unroll
        for (int q = 0; q < PY; ++q) p[q] = own[slot][q][threadIdx.x];
        const float* x = tile.corner(win[slot]);
        slot = (slot + 1) % kTileDepth;
#pragma unroll
        for (int wr = 0; wr < PY + F - 1; ++wr) {
            float xr[F];
#pragma unroll
            for (int kc = 0; kc < F; ++kc) xr[kc] = x[wr * W::WX + kc];
#pragma unroll
            for (int q = 0; q < PY; ++q) {
                const int kr = wr - q;
                if (kr < 0 || kr >= F) continue;
#pragma unroll
                for (int kc = 0; kc < F; ++kc)
                    acc[q][kr * F + kc] = __fmaf_rn(p[q], xr[kc], acc[q][kr * F + kc]);
            }
        }
    }
    float* out = part + tt * D.G + (long long)(l - 1) * F * F * D.N;
#pragma unroll
    for (int q = 0; q < PY; ++q)
#pragma unroll
        for (int k = 0; k < F * F; ++k)
            if (tile.ok(q)) out[(long long)k * D.N + tile.own[q]] = acc[q][k];
}

// acc[e] += part[tt][e] for the segment's steps, latest first (the first segment
// starts from zero): weight gradients [l-1][k][i], then dR [o][i].
__global__ void k_rate_acc(Dims D, int nt, bool first, const float* __restrict__ part,
                           float* __restrict__ acc) {
    wait_for_previous();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= D.G) return;
    float s = first ? 0.0f : acc[e];
    for (int t1 = nt - 1; t1 >= 0; t1 -= kAhead) {
        float v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = t1 - u >= 0 ? part[(t1 - u) * D.G + e] : 0.0f;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (t1 - u >= 0) s += v[u];
    }
    acc[e] = s;
}

// The finished sums: dw[l][i][k] = acc[l][k][i], and dR.
__global__ void k_rate_out(Dims D, const float* __restrict__ acc, float* __restrict__ dw,
                           float* __restrict__ dwo) {
    wait_for_previous();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per = (long long)D.N * D.K, weights = (D.L - 1) * per;
    if (idx >= D.G) return;
    if (idx >= weights) {
        dwo[idx - weights] = acc[idx];
        return;
    }
    const int l = (int)(idx / per), rem = (int)(idx - l * per), i = rem / D.K, k = rem - i * D.K;
    dw[idx] = acc[l * per + (long long)k * D.N + i];
}

// dR, the same scheme: grid (blocks of neurons, timesteps).  A thread sums V
// consecutive neurons for every output over the batch in order, kUnroll elements'
// rates in flight; the step's dloss/dy is staged kReadoutBatch elements at a time.
// The step's total goes to part[tt][o][i], and k_rate_acc adds the steps latest
// first.
constexpr int kUnroll = 16;
constexpr int kReadoutBatch = 64;
constexpr int kReadoutThreads = 64;

template <int V>
__global__ void __launch_bounds__(kReadoutThreads) k_rate_dwo(Dims D, const float* __restrict__ gy,
                                                             const float* __restrict__ seg_r,
                                                             float* __restrict__ part) {
    __shared__ __align__(16) float gs[kReadoutBatch][kMaxOutputs];
    const int i = (blockIdx.x * kReadoutThreads + threadIdx.x) * V, tt = blockIdx.y;
    const bool ok = i < D.N;
    const float* r = seg_r + (tt + 1) * D.S + (D.L - 1) * D.BN + (ok ? i : 0);
    const float* gt = gy + (long long)tt * D.B * D.O;
    float st[kMaxOutputs][V];
#pragma unroll
    for (int o = 0; o < kMaxOutputs; ++o)
#pragma unroll
        for (int q = 0; q < V; ++q) st[o][q] = 0.0f;
    wait_for_previous();
    for (int b0 = 0; b0 < D.B; b0 += kReadoutBatch) {
        const int nb = min(kReadoutBatch, D.B - b0);
        __syncthreads();
        for (int e = threadIdx.x; e < nb * kMaxOutputs; e += kReadoutThreads) {
            const int b = e / kMaxOutputs, o = e % kMaxOutputs;
            gs[b][o] = o < D.O ? __ldg(gt + (long long)(b0 + b) * D.O + o) : 0.0f;
        }
        __syncthreads();
        for (int b = 0; b < nb; b += kUnroll) {
            float rv[kUnroll][V];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (b + u < nb) load_row<V>(r + (long long)(b0 + b + u) * D.N, rv[u]);
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                if (b + u >= nb) break;
#pragma unroll
                for (int o = 0; o < kMaxOutputs; ++o)
                    if (o < D.O)
#pragma unroll
                        for (int q = 0; q < V; ++q)
                            st[o][q] = __fmaf_rn(gs[b + u][o], rv[u][q], st[o][q]);
            }
        }
    }
    if (!ok) return;
#pragma unroll
    for (int o = 0; o < kMaxOutputs; ++o)
        if (o < D.O)
#pragma unroll
            for (int q = 0; q < V; ++q) part[tt * D.G + (long long)o * D.N + i + q] = st[o][q];
}

// Per layer, sum of lamd over batch and neurons: grid (kTauBlocks, L), each
// block a fixed strided slice reduced in a fixed tree.  The parts of one sign and the
// other cancel, and float additions of what is left err by more than everything before
// them: with all of them in float dtau erred by 2.02e-7 against 64 bits (7 networks, 100
// seeds), with the last 64 in double by 1.76e-7, with all in double by 1.71e-7 (1.74e-7
// where every timestep was added up by itself), for 1 us of a pass.
__global__ void __launch_bounds__(256) k_rate_dtau_partial(Dims D, const float* __restrict__ lamd,
                                                           float* __restrict__ part) {
    wait_for_previous();
    __shared__ double sm[256];
    const int l = blockIdx.y, tid = threadIdx.x;
    const float* from = lamd + l * D.BN;
    double acc = 0.0;
    for (long long e = (long long)blockIdx.x * 256 + tid; e < D.BN; e += (long long)gridDim.x * 256)
        acc += from[e];
    sm[tid] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (tid < s) sm[tid] += sm[tid + s];
        __syncthreads();
    }
    if (tid == 0) part[(long long)l * kTauBlocks + blockIdx.x] = (float)sm[0];
}

// dtau_l = -(dt / tau_l^2) * sum of the layer's partials, in double.
__global__ void __launch_bounds__(256) k_rate_dtau_final(Dims D, const float* __restrict__ tau,
                                                         const float* __restrict__ part,
                                                         float* __restrict__ dtau) {
    wait_for_previous();
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= D.L) return;
    double s[4] = {};                                        // (chains of slow additions)
    for (int q = 0; q < kTauBlocks; q += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += part[(long long)l * kTauBlocks + q + u];
    const float tv = __ldg(tau + l);
    dtau[l] = (float)((s[0] + s[1]) + (s[2] + s[3])) * (-D.dt / (tv * tv));
}

// A segment's state of up to this many bytes stays in L2 and costs less than
// the launches of shorter segments: small networks are not cut up more finely.
constexpr long long kSegmentBytes = 64ll << 20;
constexpr long long kChunkBytes = 64ll << 20;

// States ([L][B][N]) of the segment buffers: lambda, sum of lambda d and two
// carries, then rates [k+1], drives [k] and adjoints [k].  The forward pass keeps
// two layers' chunks there.
long long carry_states(const Dims& D) { return std::max(D.k + 1, 4); }
long long chunk_states(const Dims& D) { return carry_states(D) + 3ll * D.k + 1; }

Dims make_dims(const SgRateShape& s) {
    if (s.layers < 1 || s.rows < 1 || s.cols < 1 || s.batch < 1 || s.steps < 1 ||
        s.checkpoint < 1)
        throw SgError("rate network: sizes must be positive");
    if (s.outputs < 1 || s.outputs > kMaxOutputs)
        throw SgError("rate network: outputs must lie in 1..16");
    if (s.field < 1 || s.field % 2 == 0 || s.field > kMaxField)
        throw SgError("rate network: field must be odd and at most 9");
    if (!(s.dt > 0.0f)) throw SgError("rate network: dt must be positive");
    if ((long long)s.layers * s.batch > 65535) throw SgError("rate network: layers x batch too large");
    if (std::min(s.checkpoint, s.steps) > 65535)
        throw SgError("rate network: at most 65535 steps between checkpoints");
    Dims D;
    D.L = s.layers;
    D.rows = s.rows;
    D.cols = s.cols;
    D.N = s.rows * s.cols;
    D.field = s.field;
    D.K = s.field * s.field;
    D.O = s.outputs;
    D.B = s.batch;
    D.T = s.steps;
    D.dt = s.dt;
    D.BN = (long long)D.B * D.N;
    D.S = D.L * D.BN;
    // per step: rates, drives, adjoints and the weight gradients' totals
    D.G = (long long)(D.L - 1) * D.N * D.K + (long long)D.O * D.N;
    const long long step_bytes = 4 * (3 * D.S + D.G);
    D.k = (int)std::max<long long>(std::min(s.checkpoint, D.T),
                                   std::min<long long>({kSegmentBytes / step_bytes, D.T, 65535}));
    D.nseg = (D.T + D.k - 1) / D.k;
    // forward: two layers' rates of a chunk of steps at a time, within the
    // segment buffers of the backward pass and (mostly) L2; chunks alike
    const long long fit = std::min(chunk_states(D) * D.L / 2, kChunkBytes / (8 * D.BN)) - 1;
    const long long most = std::max<long long>(1, std::min<long long>(fit, D.T));
    D.chunk = (int)((D.T + (D.T + most - 1) / most - 1) / ((D.T + most - 1) / most));
    return D;
}

// Workspace layout (floats): checkpoints [nseg][S]; v at a chunk's end [S]; the
// segment buffers (chunk_states); outputs y [T][B][O], squared errors [T][B],
// dloss/dy [T][B][O], tau partials, transposed weights, the gradients [G], and
// their per-step totals of one segment [k][G].
struct Work {
    float *ckpt, *v, *chunk, *lam, *lamd, *carry[2], *seg_r, *seg_d, *seg_P, *y, *loss_tb, *gy,
        *tau_part, *wt, *grad, *grad_part;
    long long floats;
    bool aligned;            // on 16 bytes (every array then is)
};

Work carve(const Dims& D, void* base) {
    Work w{};
    float* p = static_cast<float*>(base);
    auto take = [&](long long n) {
        float* q = p;
        n = (n + 63) / 64 * 64;       // 256-byte aligned pieces
        if (p) p += n;
        w.floats += n;
        return q;
    };
    const long long weights = (long long)(D.L - 1) * D.K * D.N;
    w.ckpt = take((long long)D.nseg * D.S);
    w.v = take(D.S);
    w.chunk = take(chunk_states(D) * D.S);
    if (w.chunk) {
        w.lam = w.chunk;
        w.lamd = w.lam + D.S;
        w.carry[0] = w.lamd + D.S;
        w.carry[1] = w.carry[0] + D.S;
        w.seg_r = w.chunk + carry_states(D) * D.S;
        w.seg_d = w.seg_r + (long long)(D.k + 1) * D.S;
        w.seg_P = w.seg_d + (long long)D.k * D.S;
    }
    w.y = take((long long)D.T * D.B * D.O);
    w.loss_tb = take((long long)D.T * D.B);
    w.gy = take((long long)D.T * D.B * D.O);
    w.tau_part = take((long long)D.L * kTauBlocks);
    w.wt = take(weights);
    w.grad = take(D.G);
    w.grad_part = take(D.k * D.G);
    w.aligned = reinterpret_cast<uintptr_t>(base) % 16 == 0;
    return w;
}

unsigned grid_of(long long n) { return (unsigned)((n + 255) / 256); }

// Every launch of a pass is a programmatic dependent of the one before it, but for
// k_rate_dw with few CTAs (below).
template <class... P, class... A>
void launch(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t st, A... args) {
    launch_dependent(kernel, grid, dim3((unsigned)threads), 0, st, args...);
}

// CTAs of k_rate_dw are small and run long, a whole batch each.  Launched while the
// adjoint's last wave ends they crowd onto the SMs that are free first, up to a dozen to
// one, and the others stay empty: up to 8 CTAs to an SM wait for the launch before
// (3 x 64x16, field 3, batch 256: 0.71 ms a training step, 1.28 as dependents; 6 x 16x16,
// batch 256: 0.79 and 1.30; 2 x 256x256, batch 4, 9 CTAs to an SM: 0.44 and 0.43).
bool crowds(const dim3& grid) { return (long long)grid.x * grid.y * grid.z <= 8 * num_sms(); }

void transpose_weights(const Dims& D, const float* w, const Work& W, cudaStream_t st) {
    if (D.L < 2) return;
    launch(k_rate_transpose, dim3(grid_of((long long)(D.L - 1) * D.N * D.K)), 256, st, D, w, W.wt);
}

// Rows a thread takes: the full tile_py rows where that leaves a CTA for every
// SM, one (most CTAs) in smaller problems, whose items wait on each other's
// latency.
unsigned tiles(const Dims& D, int py) {
    const int ty = py * kTileWarps;
    return (unsigned)(((D.rows + ty - 1) / ty) * ((D.cols + 31) / 32));
}
bool wide(const Dims& D, long long per_tile) { return tiles(D, tile_py(D.field)) * per_tile >= num_sms(); }

// Pieces of 4 floats need rows that start on 16 bytes.
#define SG_RATE_TILE_V(D_, WIDE, VV, CALL)                                                 \
    switch ((D_).field * 2 + ((WIDE) ? 1 : 0)) {                                           \
        case 2: { constexpr int F = 1, PY = 1, V = VV; CALL; } break;                      \
        case 3: { constexpr int F = 1, PY = tile_py(1), V = VV; CALL; } break;             \
        case 6: { constexpr int F = 3, PY = 1, V = VV; CALL; } break;                      \
        case 7: { constexpr int F = 3, PY = tile_py(3), V = VV; CALL; } break;             \
        case 10: { constexpr int F = 5, PY = 1, V = VV; CALL; } break;                     \
        case 11: { constexpr int F = 5, PY = tile_py(5), V = VV; CALL; } break;            \
        case 14: { constexpr int F = 7, PY = 1, V = VV; CALL; } break;                     \
        case 15: { constexpr int F = 7, PY = tile_py(7), V = VV; CALL; } break;            \
        default: { constexpr int F = 9, PY = 1, V = VV; CALL; } break;                     \
    }
#define SG_RATE_TILE(D_, W_, WIDE, CALL)                                                   \
    if ((D_).cols % 4 == 0 && (W_).aligned) { SG_RATE_TILE_V(D_, WIDE, 4, CALL) }                          \
    else { SG_RATE_TILE_V(D_, WIDE, 1, CALL) }

// Batch elements a CTA takes one after the other: all of them share its weights,
// but a CTA for each of the 5 or more that an SM can hold comes first (3 x 64x64,
// batch 64: 2.11 ms a training step with two elements to a CTA, 1.85 with one then).
int batch_group(const Dims& D, unsigned ntiles) {
    return (int)std::max<long long>(1, (long long)ntiles * D.B / (5 * num_sms()));
}

// Layer l through the steps c + 1 .. c + nt.
void layer_steps(const Dims& D, int l, LayerArgs A, const float* x, const Work& W, const float* tau,
                 cudaStream_t st) {
    if (l == 0) {
        launch(k_rate_input, dim3(grid_of(D.BN)), kBlock, st, D, A, x, tau);
    } else {
        SG_RATE_TILE(D, W, wide(D, D.B), ({
            const unsigned nt = tiles(D, PY);
            A.bg = batch_group(D, nt);
            const dim3 grid(nt, (unsigned)((D.B + A.bg - 1) / A.bg));
            launch(k_rate_layer<F, PY, V>, grid, kTileThreads, st, D, l, A, W.wt, tau);
        }));
    }
}

void forward(const Dims& D, const float* x, const float* w, const float* wo, const float* tau,
             const float* target, float* y_out, float* loss, void* ws, cudaStream_t st) {
    Work W = carve(D, ws);
    transpose_weights(D, w, W, st);
    float* buf[2] = {W.chunk, W.chunk + (D.chunk + 1) * D.BN};
    for (int c = 0; c < D.T; c += D.chunk) {
        const int nt = std::min(D.chunk, D.T - c);
        for (int l = 0; l < D.L; ++l) {
            LayerArgs A{};
            A.src = buf[(l + 1) & 1];
            A.r = buf[l & 1];
            A.src_t = A.r_t = D.BN;
            A.v0 = c > 0 ? W.v + l * D.BN : nullptr;
            A.v1 = W.v + l * D.BN;
            A.ckpt = W.ckpt + l * D.BN;
            A.c = c;
            A.nt = nt;
            layer_steps(D, l, A, x, W, tau, st);
        }
        const long long rows = (long long)nt * D.B;
        launch(W.aligned && D.N % 4 == 0 ? k_rate_readout<4> : k_rate_readout<1>,
               dim3((unsigned)((rows + kReadRows - 1) / kReadRows)), kBlock, st, D, c, nt,
               buf[(D.L - 1) & 1], D.BN, wo, target, W.y, W.loss_tb);
    }
    launch(k_rate_loss, dim3(1), 256, st, D, W.loss_tb, loss);
    if (y_out)
        SG_CUDA(cudaMemcpyAsync(y_out, W.y, (size_t)D.T * D.B * D.O * sizeof(float),
                                cudaMemcpyDeviceToDevice, st));
}

void backward(const Dims& D, const float* x, const float* w, const float* wo, const float* tau,
              const float* target, float grad_loss, void* ws, float* dw, float* dwo,
              float* dtau, float* dx, cudaStream_t st) {
    Work W = carve(D, ws);
    transpose_weights(D, w, W, st);
    const float gscale = grad_loss * 2.0f / (float)((long long)D.T * D.B * D.O);
    launch(k_rate_gy, dim3(grid_of((long long)D.T * D.B * D.O)), 256, st, D, gscale, W.y, target, W.gy);
    const long long weights = (long long)(D.L - 1) * D.N * D.K;
    // nothing follows the last step
    if (D.L > 1) SG_CUDA(cudaMemsetAsync(W.carry[D.nseg & 1], 0, D.S * sizeof(float), st));
    for (int seg = D.nseg - 1; seg >= 0; --seg) {
        const int c = seg * D.k, nt = std::min(D.k, D.T - c);
        const bool first = seg == D.nseg - 1;
        for (int l = 0; l < D.L; ++l) {
            LayerArgs A{};
            A.src = l > 0 ? W.seg_r + (l - 1) * D.BN : nullptr;
            A.r = W.seg_r + l * D.BN;
            A.src_t = A.r_t = D.S;
            A.d = W.seg_d + l * D.BN;
            A.v0 = seg > 0 ? W.ckpt + (long long)seg * D.S + l * D.BN : nullptr;
            A.c = c;
            A.nt = nt;
            layer_steps(D, l, A, x, W, tau, st);
        }
        for (int l = D.L - 1; l >= 0; --l) {
            AdjointArgs A{};
            A.r = W.seg_r + l * D.BN;
            A.d = W.seg_d + l * D.BN;
            A.next = W.seg_P + (l + 1) * D.BN;
            A.next_carry = W.carry[(seg + 1) & 1] + (l + 1) * D.BN;
            // layer 0's P is dx, and nothing else reads it
            A.P = l > 0 ? W.seg_P + l * D.BN : (dx ? dx + (long long)c * D.BN : nullptr);
            A.P_t = l > 0 ? D.S : D.BN;
            A.carry = l > 0 ? W.carry[seg & 1] + l * D.BN : nullptr;
            A.first = first;
            A.lam = W.lam + l * D.BN;
            A.lamd = W.lamd + l * D.BN;
            A.nt = nt;
            if (l == D.L - 1) {
                const dim3 grid((unsigned)((D.N + kBlock - 1) / kBlock), (unsigned)D.B);
                launch(k_rate_adjoint_top, grid, kBlock, st, D, A, wo, W.gy + (long long)c * D.B * D.O, tau);
            } else {
                SG_RATE_TILE(D, W, wide(D, D.B), ({
                    const unsigned n = tiles(D, PY);
                    A.bg = batch_group(D, n);
                    const dim3 grid(n, (unsigned)((D.B + A.bg - 1) / A.bg));
                    launch(k_rate_adjoint<F, PY, V>, grid, kTileThreads, st, D, l, A, W.wt, tau);
                }));
            }
        }
        if (D.L > 1) {
            SG_RATE_TILE(D, W, wide(D, (long long)(D.L - 1) * nt), ({
                const dim3 grid(tiles(D, PY), (unsigned)(D.L - 1), (unsigned)nt);
                if (crowds(grid)) {
                    k_rate_dw<F, PY, V><<<grid, kTileThreads, 0, st>>>(D, W.seg_P, W.seg_r, W.grad_part);
                    SG_LAUNCH_CHECK();
                } else {
                    launch(k_rate_dw<F, PY, V>, grid, kTileThreads, st, D, W.seg_P, W.seg_r, W.grad_part);
                }
            }));
        }
        const int dwo_v = W.aligned && D.N % 4 == 0 ? 4 : 1, per = kReadoutThreads * dwo_v;
        launch(dwo_v == 4 ? k_rate_dwo<4> : k_rate_dwo<1>,
               dim3((unsigned)((D.N + per - 1) / per), (unsigned)nt), kReadoutThreads, st, D,
               W.gy + (long long)c * D.B * D.O, W.seg_r, W.grad_part + weights);
        launch(k_rate_acc, dim3(grid_of(D.G)), 256, st, D, nt, first, W.grad_part, W.grad);
    }
    launch(k_rate_out, dim3(grid_of(D.G)), 256, st, D, W.grad, dw, dwo);
    launch(k_rate_dtau_partial, dim3(kTauBlocks, D.L), 256, st, D, W.lamd, W.tau_part);
    launch(k_rate_dtau_final, dim3((unsigned)((D.L + 255) / 256)), 256, st, D, tau, W.tau_part, dtau);
}

}  // namespace

extern "C" {

long long sg_rate_workspace_bytes(const SgRateShape* shape) {
    if (!shape) return SG_RATE_EINVAL;
    try {
        return carve(make_dims(*shape), nullptr).floats * (long long)sizeof(float);
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return SG_RATE_EINVAL;
}

int sg_rate_forward(const SgRateShape* shape, const float* x, const float* weights,
                    const float* readout, const float* tau, const float* target, float* y,
                    float* loss, void* workspace, void* stream) {
    if (!shape || !x || !readout || !tau || !target || !loss || !workspace) return SG_RATE_EINVAL;
    try {
        Dims D = make_dims(*shape);
        if (D.L > 1 && !weights) return SG_RATE_EINVAL;
        forward(D, x, weights, readout, tau, target, y, loss, workspace,
                static_cast<cudaStream_t>(stream));
        return 0;
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return SG_RATE_ECUDA;
}

int sg_rate_backward(const SgRateShape* shape, const float* x, const float* weights,
                     const float* readout, const float* tau, const float* target,
                     float grad_loss, void* workspace, float* d_weights, float* d_readout,
                     float* d_tau, float* d_x, void* stream) {
    if (!shape || !x || !readout || !tau || !target || !workspace || !d_readout || !d_tau)
        return SG_RATE_EINVAL;
    try {
        Dims D = make_dims(*shape);
        if (D.L > 1 && (!weights || !d_weights)) return SG_RATE_EINVAL;
        backward(D, x, weights, readout, tau, target, grad_loss, workspace, d_weights, d_readout,
                 d_tau, d_x, static_cast<cudaStream_t>(stream));
        return 0;
    } catch (const std::exception& e) {
        sg::set_last_error(e.what());
    }
    return SG_RATE_ECUDA;
}

}  // extern "C"
