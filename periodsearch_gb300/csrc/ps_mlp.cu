// ps_mlp.cu -- training and inference kernels of the learned early-stop
// predictor: a 10-64-64-1 multilayer perceptron with GELU activations in
// FP32.  It maps the first K iterations of an LM fit (the screening depth:
// accepted chi^2 ratios and lambda every K/4 iterations, Ndata, period) to
// log(final rms / rms after those iterations).  Parameters live in one float array (layout kMlp* in
// ps_engine.h): input mean/std, W1[64][10], b1, W2[64][64], b2, W3[64], b3,
// target mean/std.  Standardisation constants are computed on the host;
// training updates W1..b3 with Adam on mean squared error.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <numeric>
#include <random>
#include <vector>

#include "ps_engine.h"

namespace psg {

namespace {

__device__ inline float erf1(float x) { return 1.f + erff(x * 0.70710678118654752f); }
// The derivative, with t = 1 + erf(x / sqrt 2) at hand from the forward pass.
__device__ inline float gelu_grad(float x, float t)
{
    return 0.5f * t + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// One Adam step of a parameter p with moments m, v and gradient gi.
__device__ inline void adam_update(float &p, float &m, float &v, float gi, float lr, float b1, float b2, float eps,
                                   float c1, float c2)
{
    const float mi = fmaf(1.f - b1, gi, __fmul_rn(b1, m));
    const float vi = fmaf(__fmul_rn(1.f - b2, gi), gi, __fmul_rn(b2, v));
    m = mi;
    v = vi;
    p -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Training runs in one kernel per epoch, on one thread-block cluster: the
// mini-batch steps depend on each other, and a step of 512 samples is 15
// MFLOP, so what counts is the number of launches, copies and passes through
// memory between them (twelve launches and a copy per step took 261 us).
//
// A step has two halves, each ended by a cluster barrier:
//   * samples: a CTA takes tiles of 32 samples through forward and backward
//     pass in shared memory and leaves what the gradients need (h1, h2, dz1,
//     dz2, the standardised inputs, d loss / d out) in global memory (L2);
//   * parameters: every parameter belongs to one thread of the cluster, which
//     sums its gradient over the batch in sample order and applies Adam to
//     its registers' copy (value and both moments stay there for the epoch).
//     The batch's values lie with the samples along the rows and come through
//     shared memory in chunks (cp.async by the warps without parameters, three
//     ahead), so that a chain takes four samples of a factor per load; a
//     thread's two parameters share one factor; the biases' other factor is a row of ones, so all parameters
//     run the same code.  The other warps fetch the next step's samples.
// Every sum runs in the order of the sample or unit index, one chain per
// value, whatever the number of CTAs.
// Measured (20000 samples, batch 512, 6 epochs = 234 steps): 61.4 -> 4.1 ms;
// of a step's 32 kcycles the samples' half takes 11, the gradient chains 14,
// the weights' reload 4, the barriers 3.
constexpr int kNt = 512;          // threads
constexpr int kTile = 32;         // samples of a tile
constexpr int kPitch = 68;        // activations: rows of 64, 16-byte aligned
constexpr int kWPitch = 65;       // W2 in shared memory: rows and columns conflict-free
constexpr int kXPitch = 12;

// What the gradients of a batch need, in global memory: rows of pitch Bp (the
// batch rounded up to a chunk; zero beyond the batch) with the samples along
// them: h1, the inputs, dz1, dz2, h2, d loss / d out.
constexpr int kChunk = 64;        // samples of a staged chunk
constexpr int kStages = 4;        // chunks in flight or in use
constexpr int kRowX = kHidden, kRowDz1 = kRowX + kFeat, kRowDz2 = kRowDz1 + kHidden, kRowH2 = kRowDz2 + kHidden,
              kRowDout = kRowH2 + kHidden, kRows = kRowDout + 1;
struct Acts {
    float *rows;      // [kRows][Bp]
    int Bp;
    float *loss;      // [B]
};
constexpr size_t batch_pitch(int B) { return (static_cast<size_t>(B) + kChunk - 1) / kChunk * kChunk; }

// The staged rows of a CTA that owns ROWS units of either layer: h1 and the
// inputs whole, the others for its units.
template <int ROWS>
constexpr int kStagedRows = kRowDz1 + 3 * ROWS + 1;
constexpr int kSPitch = kChunk + 4;   // 16-byte rows on different banks

struct SmemMlp {
    float W1[kHidden * kFeat], b1[kHidden], W2[kHidden * kWPitch], b2[kHidden], W3[kHidden], b3[4];
    float xs[kTile * kXPitch], ys[kTile], dout[kTile];
    float h1[kTile * kPitch], h2[kTile * kPitch], dz1[kTile * kPitch], dz2[kTile * kPitch];
    float ones[kSPitch];
    float stage[kStages * kStagedRows<8> * kSPitch];
};

__device__ inline void load_weights(SmemMlp &s, const float *P)
{
    for (int e = threadIdx.x; e < kHidden * kFeat; e += kNt) s.W1[e] = P[kMlpW1 + e];
    for (int e = threadIdx.x; e < kHidden * kHidden; e += kNt)
        s.W2[(e >> 6) * kWPitch + (e & 63)] = P[kMlpW2 + e];
    if (threadIdx.x < kHidden) {
        s.b1[threadIdx.x] = P[kMlpB1 + threadIdx.x];
        s.b2[threadIdx.x] = P[kMlpB2 + threadIdx.x];
        s.W3[threadIdx.x] = P[kMlpW3 + threadIdx.x];
    }
    if (threadIdx.x == 0) s.b3[0] = P[kMlpB3];
}

// Standardised inputs of the tile's nb samples from sample b0 on (and
// targets), rows idx[b0 ..] of x where idx is given; by threads t0 .. kNt - 1.
__device__ inline void load_tile(SmemMlp &s, const float *x, const float *y, const int *idx, const float *P, int b0,
                                 int nb, int t0)
{
    const int t = static_cast<int>(threadIdx.x) - t0;
    if (t < 0) return;
    for (int e = t; e < nb * kFeat; e += kNt - t0) {
        const int b = e / kFeat, i = e - b * kFeat;
        const int r = idx ? idx[b0 + b] : b0 + b;
        s.xs[b * kXPitch + i] = (x[static_cast<size_t>(r) * kFeat + i] - P[kMlpMu + i]) / P[kMlpSd + i];
    }
    if (y && t < nb) {
        const int r = idx ? idx[b0 + t] : b0 + t;
        s.ys[t] = (y[r] - P[kMlpYMu]) / P[kMlpYSd];
    }
}

// Pre-activations and 1 + erf of the thread's four values of both layers.
struct Pre {
    float z1[4], t1[4], z2[4], t2[4];
};

// h1, h2 of the tile (a barrier before and after).  Thread: unit lane + 32
// (warp & 1), samples (warp >> 1) + 8 r.
__device__ inline void forward_tile(SmemMlp &s, Pre &k)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u = lane + 32 * (warp & 1), b = warp >> 1;
    __syncthreads();
    {
        float acc[4];
#pragma unroll
        for (int r = 0; r < 4; r++) acc[r] = s.b1[u];
#pragma unroll
        for (int i = 0; i < kFeat; i++) {
            const float w = s.W1[u * kFeat + i];
#pragma unroll
            for (int r = 0; r < 4; r++) acc[r] = fmaf(w, s.xs[(b + 8 * r) * kXPitch + i], acc[r]);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            k.z1[r] = acc[r];
            k.t1[r] = erf1(acc[r]);
            s.h1[(b + 8 * r) * kPitch + u] = 0.5f * acc[r] * k.t1[r];
        }
    }
    __syncthreads();
    {
        float acc[4];
#pragma unroll
        for (int r = 0; r < 4; r++) acc[r] = s.b2[u];
#pragma unroll 4
        for (int i = 0; i < kHidden; i += 4) {
            float w[4];
#pragma unroll
            for (int q = 0; q < 4; q++) w[q] = s.W2[u * kWPitch + i + q];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float4 h = *reinterpret_cast<const float4 *>(s.h1 + (b + 8 * r) * kPitch + i);
                acc[r] = fmaf(w[0], h.x, acc[r]);
                acc[r] = fmaf(w[1], h.y, acc[r]);
                acc[r] = fmaf(w[2], h.z, acc[r]);
                acc[r] = fmaf(w[3], h.w, acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            k.z2[r] = acc[r];
            k.t2[r] = erf1(acc[r]);
            s.h2[(b + 8 * r) * kPitch + u] = 0.5f * acc[r] * k.t2[r];
        }
    }
    __syncthreads();
}

// b3 + W3 . h2 of sample b of the tile.
__device__ inline float output_of(const SmemMlp &s, int b)
{
    float acc = s.b3[0];
#pragma unroll 8
    for (int j = 0; j < kHidden; j++) acc = fmaf(s.W3[j], s.h2[b * kPitch + j], acc);
    return acc;
}

// Outputs (standardised) of n samples.
__global__ void __launch_bounds__(kNt) predict_kernel(const float *x, const float *P, int n, float *out)
{
    extern __shared__ __align__(16) char smem[];
    SmemMlp &s = *reinterpret_cast<SmemMlp *>(smem);
    load_weights(s, P);
    for (int b0 = blockIdx.x * kTile; b0 < n; b0 += gridDim.x * kTile) {
        const int nb = min(kTile, n - b0);
        __syncthreads();
        load_tile(s, x, nullptr, nullptr, P, b0, nb, 0);
        Pre pre;
        forward_tile(s, pre);
        if (threadIdx.x < nb) out[b0 + threadIdx.x] = output_of(s, threadIdx.x);
    }
}

// Forward and backward pass of one tile (loaded by load_tile) of a batch of
// B samples; what the gradients need goes to a.
__device__ inline void train_tile(SmemMlp &s, const Acts &a, int b0, int B)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u = lane + 32 * (warp & 1), b = warp >> 1;
    const int nb = min(kTile, B - b0);
    Pre pre;
    forward_tile(s, pre);
    if (threadIdx.x < nb) {
        const float d = output_of(s, threadIdx.x) - s.ys[threadIdx.x];
        const float g = 2.f * d / B;
        s.dout[threadIdx.x] = g;
        a.rows[static_cast<size_t>(kRowDout) * a.Bp + b0 + threadIdx.x] = g;
        a.loss[b0 + threadIdx.x] = d * d / B;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int k = (b + 8 * r) * kPitch + u;
        s.dz2[k] = b + 8 * r < nb ? s.dout[b + 8 * r] * s.W3[u] * gelu_grad(pre.z2[r], pre.t2[r]) : 0.f;
    }
    __syncthreads();
    float g[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int v = 0; v < kHidden; v += 4) {
        float w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = s.W2[(v + q) * kWPitch + u];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float4 d = *reinterpret_cast<const float4 *>(s.dz2 + (b + 8 * r) * kPitch + v);
            g[r] = fmaf(d.x, w[0], g[r]);
            g[r] = fmaf(d.y, w[1], g[r]);
            g[r] = fmaf(d.z, w[2], g[r]);
            g[r] = fmaf(d.w, w[3], g[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++) s.dz1[(b + 8 * r) * kPitch + u] = g[r] * gelu_grad(pre.z1[r], pre.t1[r]);
    __syncthreads();
    // out with the samples along the rows, a sample per lane
    if (lane < nb) {
        float *to = a.rows + b0 + lane;
        for (int k = warp; k < kHidden; k += kNt / 32) {
            to[static_cast<size_t>(k) * a.Bp] = s.h1[lane * kPitch + k];
            to[static_cast<size_t>(kRowDz1 + k) * a.Bp] = s.dz1[lane * kPitch + k];
            to[static_cast<size_t>(kRowDz2 + k) * a.Bp] = s.dz2[lane * kPitch + k];
            to[static_cast<size_t>(kRowH2 + k) * a.Bp] = s.h2[lane * kPitch + k];
        }
        if (warp < kFeat) to[static_cast<size_t>(kRowX + warp) * a.Bp] = s.xs[lane * kXPitch + warp];
    }
    __syncthreads();
}

__device__ inline void copy16(float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

// Starts the copy of chunk c of the batch for the rows of a CTA whose units
// begin at r0 (past the batch: an empty group), by the threads from T0 on.
template <int ROWS, int T0>
__device__ inline void stage_chunk(float *stage, const Acts &a, int r0, int c)
{
    const int t = static_cast<int>(threadIdx.x) - T0;
    if (c * kChunk < a.Bp && t >= 0) {
        float *dst = stage + static_cast<size_t>(c % kStages) * kStagedRows<ROWS> * kSPitch;
#pragma unroll 4
        for (int e = t; e < kStagedRows<ROWS> * (kChunk / 4); e += kNt - T0) {
            const int r = e / (kChunk / 4), q = e % (kChunk / 4), k = r - kRowDz1;
            const int src = k < 0 ? r : k == 3 * ROWS ? kRowDout : kRowDz1 + k / ROWS * kHidden + r0 + k % ROWS;
            copy16(dst + r * kSPitch + 4 * q, a.rows + static_cast<size_t>(src) * a.Bp + c * kChunk + 4 * q);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The steps of one epoch (or, without moments m, one full-batch gradient
// into G): samples idx[step B ..], Adam with the bias corrections cc[step].
// One cluster of 64 / ROWS CTAs; loss[step] receives the batch's mean squared
// error (blocks of 256 samples by a tree, the blocks in order).
template <int ROWS>
__global__ void __launch_bounds__(kNt)
    train_kernel(const float *x, const float *y, const int *idx, int steps, int B, float *P, float *m, float *v,
                 const float2 *cc, float lr, Acts a, float *loss, float *G)
{
    namespace cgr = cooperative_groups;
    cgr::cluster_group cl = cgr::this_cluster();
    constexpr int cs = kHidden / ROWS;
    const int rank = static_cast<int>(cl.block_rank()), t = threadIdx.x, r0 = rank * ROWS;
    extern __shared__ __align__(16) char smem[];
    SmemMlp &s = *reinterpret_cast<SmemMlp *>(smem);
    for (int e = t; e < kSPitch; e += kNt) s.ones[e] = 1.f;
    // The thread's two parameters (of the CTA's rows of W2 and W1, b1, b2, W3;
    // b3 on the first CTA): place in P, -1 none, and the staged rows of their
    // gradients' factors, one of them common to both (-1: the row of ones).
    constexpr int kH = ROWS / 2;
    constexpr int kW2 = kH * kHidden, kW1 = kW2 + kH * kFeat, kAll = kW1 + 3 * kH + 1;
    constexpr int kFetch = kNt - 192;   // the threads from here on copy chunks and fetch the next step's samples
    static_assert(kAll <= kNt && (ROWS > 4 || kAll <= kFetch), "");
    int par[2] = {-1, -1}, fu[2] = {0, 0}, fc = 0;
    if (t < kW2) {
        const int u = 2 * (t / kHidden), i = t % kHidden;
        fc = i;
        for (int q = 0; q < 2; q++) {
            par[q] = kMlpW2 + (r0 + u + q) * kHidden + i;
            fu[q] = kRowDz1 + ROWS + u + q;
        }
    } else if (t < kW1) {
        const int u = 2 * ((t - kW2) / kFeat), i = (t - kW2) % kFeat;
        fc = kRowX + i;
        for (int q = 0; q < 2; q++) {
            par[q] = kMlpW1 + (r0 + u + q) * kFeat + i;
            fu[q] = kRowDz1 + u + q;
        }
    } else if (t < kW1 + 3 * kH) {
        const int kind = (t - kW1) / kH, u = 2 * ((t - kW1) % kH);
        fc = kind == 2 ? kRowDz1 + 3 * ROWS : -1;
        for (int q = 0; q < 2; q++) {
            par[q] = (kind == 0 ? kMlpB1 : kind == 1 ? kMlpB2 : kMlpW3) + r0 + u + q;
            fu[q] = kRowDz1 + kind * ROWS + u + q;
        }
    } else if (t == kAll - 1 && rank == 0) {
        par[0] = kMlpB3;
        fu[0] = fu[1] = kRowDz1 + 3 * ROWS;
        fc = -1;
    }
    float pv[2], mv[2], vv[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        pv[q] = par[q] >= 0 ? P[par[q]] : 0.f;
        mv[q] = par[q] >= 0 && m ? m[par[q]] : 0.f;
        vv[q] = par[q] >= 0 && m ? v[par[q]] : 0.f;
    }
    bool fetched = false;
    for (int step = 0; step < steps; step++) {
        load_weights(s, P);
        for (int b0 = rank * kTile; b0 < B; b0 += cs * kTile) {
            if (!fetched)
                load_tile(s, x, y, idx ? idx + static_cast<size_t>(step) * B : nullptr, P, b0, min(kTile, B - b0), 0);
            fetched = false;
            train_tile(s, a, b0, B);
        }
        cl.sync();
        float g[2] = {0.f, 0.f};
#pragma unroll
        for (int c = 0; c < kStages - 1; c++) stage_chunk<ROWS, kFetch>(s.stage, a, r0, c);
        if (step + 1 < steps && rank * kTile < B) {
            load_tile(s, x, y, idx + static_cast<size_t>(step + 1) * B, P, rank * kTile, min(kTile, B - rank * kTile),
                      kFetch);
            fetched = true;
        }
        for (int c = 0; c * kChunk < a.Bp; c++) {
            // chunk c has landed, and the buffer of chunk c - 1 is free
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            __syncthreads();
            stage_chunk<ROWS, kFetch>(s.stage, a, r0, c + kStages - 1);
            const float *k = s.stage + static_cast<size_t>(c % kStages) * kStagedRows<ROWS> * kSPitch;
            if (par[0] >= 0) {
                const float4 *x0 = reinterpret_cast<const float4 *>(k + fu[0] * kSPitch);
                const float4 *x1 = reinterpret_cast<const float4 *>(k + fu[1] * kSPitch);
                const float4 *y4 = reinterpret_cast<const float4 *>(fc < 0 ? s.ones : k + fc * kSPitch);
#pragma unroll
                for (int b = 0; b < kChunk / 4; b++) {
                    const float4 u0 = x0[b], u1 = x1[b], w = y4[b];
                    g[0] = fmaf(u0.x, w.x, g[0]);
                    g[1] = fmaf(u1.x, w.x, g[1]);
                    g[0] = fmaf(u0.y, w.y, g[0]);
                    g[1] = fmaf(u1.y, w.y, g[1]);
                    g[0] = fmaf(u0.z, w.z, g[0]);
                    g[1] = fmaf(u1.z, w.z, g[1]);
                    g[0] = fmaf(u0.w, w.w, g[0]);
                    g[1] = fmaf(u1.w, w.w, g[1]);
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        const float2 c = m ? cc[step] : make_float2(1.f, 1.f);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (par[q] < 0) continue;
            if (m) {
                adam_update(pv[q], mv[q], vv[q], g[q], lr, 0.9f, 0.999f, 1e-8f, c.x, c.y);
                P[par[q]] = pv[q];
            } else {
                G[par[q]] = g[q];
            }
        }
        if (rank == cs - 1 && t >= kNt - 32) {
            const int lane = t & 31;
            float sum = 0.f;
            for (int k0 = 0; k0 < B; k0 += 256) {
                float q[8];
#pragma unroll
                for (int k = 0; k < 8; k++) q[k] = k0 + 32 * k + lane < B ? a.loss[k0 + 32 * k + lane] : 0.f;
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < o; k++) q[k] += q[k + o];
                float w = q[0];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
                sum += w;
            }
            if (lane == 0) loss[step] = sum;
        }
        cl.sync();
    }
#pragma unroll
    for (int q = 0; q < 2; q++)
        if (par[q] >= 0 && m) {
            m[par[q]] = mv[q];
            v[par[q]] = vv[q];
        }
}

// One device allocation, freed with its owner.
struct DevMem {
    char *p = nullptr;
    size_t used = 0;
    ~DevMem() { cudaFree(p); }
    template <class T>
    T *take(size_t n)
    {
        T *r = reinterpret_cast<T *>(p + used);
        used += (n * sizeof(T) + 255) & ~size_t(255);
        return r;
    }
};

// The batch's buffers, cleared (the rows' ends stay zero).
Acts take_acts(DevMem &d, int B)
{
    Acts a;
    a.Bp = static_cast<int>(batch_pitch(B));
    a.rows = d.take<float>(static_cast<size_t>(kRows) * a.Bp);
    a.loss = d.take<float>(B);
    cudaMemset(a.rows, 0, static_cast<size_t>(kRows) * a.Bp * sizeof(float));
    return a;
}
constexpr size_t act_floats(int B) { return kRows * batch_pitch(B) + B; }

using TrainKernel = void (*)(const float *, const float *, const int *, int, int, float *, float *, float *,
                             const float2 *, float, Acts, float *, float *);

// The training kernel's cluster: 16 CTAs of four units of a layer each, or 8
// of eight where the device runs no cluster of 16.
cudaError_t train_config(cudaLaunchConfig_t &lc, cudaLaunchAttribute *attr, TrainKernel &k)
{
    lc = {};
    lc.blockDim = dim3(kNt);
    lc.dynamicSmemBytes = sizeof(SmemMlp);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    for (unsigned cs : {16u, 8u}) {
        k = cs == 16 ? train_kernel<4> : train_kernel<8>;
        lc.gridDim = dim3(cs);
        attr[0].val.clusterDim.x = cs;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(sizeof(SmemMlp)));
        if (e == cudaSuccess && cs > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        int n = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, k, &lc);
        if (e == cudaSuccess && n > 0) return e;
        cudaGetLastError();
    }
    return cudaErrorInvalidConfiguration;
}

}  // namespace

int mlp_grad(const float *h_P, const float *h_x, const float *h_y, int n, float *h_loss, float *h_G)
{
    const size_t nx = static_cast<size_t>(n) * kFeat;
    cudaLaunchConfig_t lc;
    cudaLaunchAttribute attr[1];
    TrainKernel train_kernel_of = nullptr;
    cudaError_t e = train_config(lc, attr, train_kernel_of);
    if (e != cudaSuccess) return static_cast<int>(e);
    DevMem d;
    e = cudaMalloc(&d.p, (nx + n + 2 * kMlpFloats + act_floats(n)) * sizeof(float) + 16 * 256);
    if (e != cudaSuccess) return static_cast<int>(e);
    float *dx = d.take<float>(nx), *dy = d.take<float>(n), *dP = d.take<float>(kMlpFloats),
          *dG = d.take<float>(kMlpFloats), *dl = d.take<float>(1);
    const Acts a = take_acts(d, n);
    cudaMemcpy(dx, h_x, nx * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dy, h_y, n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dP, h_P, kMlpFloats * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(dG, 0, kMlpFloats * sizeof(float));
    e = cudaLaunchKernelEx(&lc, train_kernel_of, static_cast<const float *>(dx), static_cast<const float *>(dy),
                           static_cast<const int *>(nullptr), 1, n, dP, static_cast<float *>(nullptr),
                           static_cast<float *>(nullptr), static_cast<const float2 *>(nullptr), 0.f, a, dl, dG);
    if (e == cudaSuccess) e = cudaMemcpy(h_G, dG, kMlpFloats * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(h_loss, dl, sizeof(float), cudaMemcpyDeviceToHost);
    return static_cast<int>(e);
}

int mlp_predict(const float *h_P, const float *h_x, int n, float *h_out)
{
    const size_t nx = static_cast<size_t>(n) * kFeat;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(predict_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(offsetof(SmemMlp, stage)));
    if (e != cudaSuccess) return static_cast<int>(e);
    DevMem d;
    e = cudaMalloc(&d.p, (nx + n + kMlpFloats) * sizeof(float) + 3 * 256);
    if (e != cudaSuccess) return static_cast<int>(e);
    float *dx = d.take<float>(nx), *dP = d.take<float>(kMlpFloats), *dout = d.take<float>(n);
    cudaMemcpy(dx, h_x, nx * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dP, h_P, kMlpFloats * sizeof(float), cudaMemcpyHostToDevice);
    const int tiles = (n + kTile - 1) / kTile;
    predict_kernel<<<std::min(tiles, 2 * sms), kNt, offsetof(SmemMlp, stage)>>>(dx, dP, n, dout);
    e = cudaGetLastError();
    std::vector<float> out(n);
    if (e == cudaSuccess) e = cudaMemcpy(out.data(), dout, n * sizeof(float), cudaMemcpyDeviceToHost);
    for (int i = 0; i < n && e == cudaSuccess; i++) h_out[i] = out[i] * h_P[kMlpYSd] + h_P[kMlpYMu];
    return static_cast<int>(e);
}

int mlp_train(float *h_P, const float *h_x, const float *h_y, int n, int epochs, int batch, float lr, uint64_t seed,
              float *h_loss_hist)
{
    const int B = std::min(batch, n);
    const int steps = n / B;   // per epoch
    const size_t nx = static_cast<size_t>(n) * kFeat, total = static_cast<size_t>(steps) * epochs;
    cudaLaunchConfig_t lc;
    cudaLaunchAttribute attr[1];
    TrainKernel train_kernel_of = nullptr;
    cudaError_t e = train_config(lc, attr, train_kernel_of);
    if (e != cudaSuccess) return static_cast<int>(e);
    DevMem d;
    e = cudaMalloc(&d.p, (nx + n + 3 * kMlpFloats + act_floats(B) + total) * sizeof(float) +
                             static_cast<size_t>(n) * sizeof(int) + total * sizeof(float2) + 20 * 256);
    if (e != cudaSuccess) return static_cast<int>(e);
    float *dx = d.take<float>(nx), *dy = d.take<float>(n), *dP = d.take<float>(kMlpFloats),
          *dm = d.take<float>(kMlpFloats), *dv = d.take<float>(kMlpFloats), *dl = d.take<float>(total);
    int *di = d.take<int>(n);
    float2 *dcc = d.take<float2>(total);
    const Acts a = take_acts(d, B);
    std::vector<float2> cc(total);
    const float b1 = 0.9f, b2 = 0.999f;   // the decay rates of train_kernel's adam_update
    for (size_t t = 0; t < total; t++) {
        cc[t].x = 1.f - std::pow(b1, static_cast<float>(t + 1));
        cc[t].y = 1.f - std::pow(b2, static_cast<float>(t + 1));
    }
    cudaMemcpy(dx, h_x, nx * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dy, h_y, n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dP, h_P, kMlpFloats * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(dcc, cc.data(), total * sizeof(float2), cudaMemcpyHostToDevice);
    cudaMemset(dm, 0, kMlpFloats * sizeof(float));
    cudaMemset(dv, 0, kMlpFloats * sizeof(float));
    std::mt19937_64 rng(seed);
    std::vector<int> perm(n);
    std::iota(perm.begin(), perm.end(), 0);
    // The next epoch's order is shuffled while an epoch runs; its copy, in the
    // same stream, follows that epoch.
    for (int ep = 0; ep < epochs && e == cudaSuccess; ep++) {
        std::shuffle(perm.begin(), perm.end(), rng);
        e = cudaMemcpy(di, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) break;
        const size_t at = static_cast<size_t>(ep) * steps;
        e = cudaLaunchKernelEx(&lc, train_kernel_of, static_cast<const float *>(dx), static_cast<const float *>(dy),
                               static_cast<const int *>(di), steps, B, dP, dm, dv,
                               static_cast<const float2 *>(dcc + at), lr, a, dl + at, static_cast<float *>(nullptr));
    }
    std::vector<float> l(total);
    if (e == cudaSuccess) e = cudaMemcpy(l.data(), dl, total * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(h_P, dP, kMlpFloats * sizeof(float), cudaMemcpyDeviceToHost);
    for (int ep = 0; ep < epochs && h_loss_hist && e == cudaSuccess; ep++) {
        double loss = 0;
        for (int k = 0; k < steps; k++) loss += l[static_cast<size_t>(ep) * steps + k];
        h_loss_hist[ep] = static_cast<float>(loss / std::max(steps, 1));
    }
    return static_cast<int>(e);
}

}  // namespace psg
