// The learned warm start's network: a small fully connected MLP (GELU hidden layers,
// linear output) trained in FP32 on the device with hand-written forward, backward and
// Adam kernels. It maps (composition, temperature) to the zero-pressure lattice constant
// and initial C11, C12, C44, so that a production run can start near equilibrium.
//
// Sizes are small (inputs and widths of tens, a few thousand samples), so every kernel is
// FP32 FMA work with sums in a fixed order: no atomics, training is bit-for-bit repeatable.
// A network whose parameters, gradients and activations of 16 samples fit a block's shared
// memory (every network this package trains) takes a training step in two kernels, k_step_grad and
// k_step_update; larger ones run layer by layer, the step captured once as a CUDA graph and
// replayed.
//
// Parameter layout (also of gradients and of the host copies): for each layer l in order,
// W_l as in_l x out_l row-major (W[i * out + o]), then b_l (out_l).
#include <cuda_runtime.h>

#include <cmath>
#include <algorithm>
#include <cstring>
#include <random>
#include <vector>

#include "host_tables.h"
#include "kernels.cuh"
#include "mdelast.h"

using mdelast::clear_error;
using mdelast::fail;

namespace {

constexpr int kT = 256;

__device__ __forceinline__ float gelu(float z) {
    return 0.5f * z * (1.f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_d(float z) {
    // d/dz [z Phi(z)] = Phi(z) + z phi(z)
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) +
           z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// Z = X W + b; A = gelu(Z) for hidden layers, A = Z for the output layer
__global__ void k_fwd(const float *X, const float *W, const float *b, float *Z, float *A, int n,
                      int in, int out, int act) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n * out)
        return;
    int const s = k / out, o = k % out;
    float z = b[o];
    for (int i = 0; i < in; ++i)
        z = fmaf(X[s * in + i], W[i * out + o], z);
    Z[k] = z;
    A[k] = act ? gelu(z) : z;
}

// mean-squared error over n x out outputs: dY = 2 (Y - T) / (n out), loss in one block with
// a fixed-order tree
__global__ void k_loss(const float *Y, const float *Tg, float *dY, float *loss, int m) {
    __shared__ float part[kT];
    float const inv = 1.f / static_cast<float>(m);
    float acc = 0.f;
    for (int k = threadIdx.x; k < m; k += kT) {
        float const d = Y[k] - Tg[k];
        dY[k] = 2.f * d * inv;
        acc = fmaf(d, d, acc);
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int w = kT / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *loss = part[0] * inv;
}

// dZ = dA * gelu'(Z)
__global__ void k_bwd_act(const float *dA, const float *Z, float *dZ, int m) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m)
        dZ[k] = dA[k] * gelu_d(Z[k]);
}

// dX = dZ W^T
__global__ void k_bwd_dx(const float *dZ, const float *W, float *dX, int n, int in, int out) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n * in)
        return;
    int const s = k / in, i = k % in;
    float acc = 0.f;
    for (int o = 0; o < out; ++o)
        acc = fmaf(dZ[s * out + o], W[i * out + o], acc);
    dX[k] = acc;
}

// dW = X^T dZ, db = column sums of dZ (thread per parameter, samples in order)
__global__ void k_bwd_dw(const float *X, const float *dZ, float *dW, float *db, int n, int in,
                         int out) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < in * out) {
        int const i = k / out, o = k % out;
        float acc = 0.f;
        for (int s = 0; s < n; ++s)
            acc = fmaf(X[s * in + i], dZ[s * out + o], acc);
        dW[k] = acc;
    } else if (k < in * out + out) {
        int const o = k - in * out;
        float acc = 0.f;
        for (int s = 0; s < n; ++s)
            acc += dZ[s * out + o];
        db[o] = acc;
    }
}

// Adam (Kingma & Ba 2015) with bias correction; the step count lives on the device so that
// a captured graph can be replayed
__device__ __forceinline__ void adam(float *p, float *m1, float *m2, int k, float gk, float lr,
                                     float step) {
    float const b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float const c1 = 1.f - powf(b1, step), c2 = 1.f - powf(b2, step);
    float const a = b1 * m1[k] + (1.f - b1) * gk;
    float const v = b2 * m2[k] + (1.f - b2) * gk * gk;
    m1[k] = a;
    m2[k] = v;
    p[k] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}
__global__ void k_adam(float *p, const float *g, float *m1, float *m2, int np, float lr,
                       const int *t) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < np)
        adam(p, m1, m2, k, g[k], lr, static_cast<float>(*t + 1));
}

__global__ void k_step_inc(int *t) {
    if (threadIdx.x == 0 && blockIdx.x == 0)
        *t += 1;
}

// ------------------------------------------------------------------------------------
// A training step of a network that fits shared memory. Layer by layer, a step was 17
// launches whose weight-gradient kernel ran one thread per weight down a serial chain over
// all samples (2,048 samples: 0.55 of the step's 0.57 ms on a few blocks). Here each block takes tiles of
// kTile16 samples through forward, loss and backward out of shared memory, with the weight
// gradients of its tiles summed there in sample order; k_step_update adds the blocks' sums in block
// order and applies Adam. 2,048 samples fill 128 of the 148 SMs once. 2-64-64-64-4 network,
// 2,048 samples: 570 -> 22 us per training step; what bounds it now is latency inside one block
// per SM (16 warps, dot products of 64 out of shared memory between barriers).
constexpr int kTile16 = 16;      // samples per tile
constexpr int kTileP = 20;       // floats per activation row: 16-byte rows whose starts 8 lanes
                                 // apart fall on different banks
constexpr int kStepThreads = 512;
constexpr int kStepBlocks = 148; // one block per SM; more samples loop over tiles
constexpr size_t kStepSmemMax = 200 * 1024;

struct NetView {
    int L, np, n, wsum; // layers, parameters, samples, sum of all widths
    int w[MDELAST_MLP_MAX_LAYERS + 1], off_w[MDELAST_MLP_MAX_LAYERS];
};

// The step's own copy of the parameters and its gradients are laid out as they lie in shared
// memory: per layer w_l + 1 rows (the weights' and the bias) of w_{l+1} floats padded by one, so
// that lanes along either index read different banks, the whole rounded to 16 bytes. The blocks copy
// it in and their sums out with 16-byte accesses (copied element by element with the
// layout's arithmetic, that was 17,000 of k_step_grad's 41,000 cycles).
__host__ __device__ inline int padded_params(NetView const &v) {
    int k = 0;
    for (int l = 0; l < v.L; ++l)
        k += (v.w[l] + 1) * (v.w[l + 1] + 1);
    return (k + 3) / 4 * 4;
}
// index in the parameters' layout of padded entry k, -1 for a pad
__device__ __forceinline__ int unpadded(NetView const &v, int k) {
    for (int l = 0; l < v.L; ++l) {
        int const out = v.w[l + 1], row = out + 1, rows = (v.w[l] + 1) * row;
        if (k < rows) {
            int const i = k / row, o = k - i * row;
            return o < out ? v.off_w[l] + i * out + o : -1;
        }
        k -= rows;
    }
    return -1;
}
__host__ inline size_t step_smem(NetView const &v) {
    int wmax = 0;
    for (int l = 0; l <= v.L; ++l)
        wmax = std::max(wmax, v.w[l]);
    return sizeof(float) * (2 * static_cast<size_t>(padded_params(v)) +
                            2 * static_cast<size_t>(kTileP) * (v.wsum + wmax));
}

// the padded copy of the parameters
__global__ void k_step_params(NetView v, const float *p, float *pp) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < padded_params(v)) {
        int const u = unpadded(v, k);
        pp[k] = u >= 0 ? p[u] : 0.f;
    }
}

// Gradients of the mean-squared error summed over this block's tiles, to part[block] (in the
// padded layout) and its loss sum to part_loss[block]. count: the training step counter
// to advance (null outside training).
__global__ void __launch_bounds__(kStepThreads)
    k_step_grad(NetView v, const float *X, const float *Y, const float *pp, float *part,
                float *part_loss, int *count) {
    mdelast::chain_begin();
    extern __shared__ float4 s_net[];
    int const tid = threadIdx.x, T = kStepThreads, L = v.L;
    float *sW = reinterpret_cast<float *>(s_net); // layer l: (w_l + 1) rows of w_{l+1} + 1
    int const nW = padded_params(v);
    float *sG = sW + nW;            // gradients in the same layout
    float *sA = sG + nW;            // activations of layer l: rows of kTileP samples
    float *sD = sA + kTileP * v.wsum; // gelu'(z) of layer l
    int wmax = 0;
    for (int l = 0; l <= L; ++l)
        wmax = max(wmax, v.w[l]);
    float *sP = sD + kTileP * v.wsum; // dA or dZ of the layer above, and of the one below
    float *sQ = sP + kTileP * wmax;
    __shared__ float s_loss[kStepThreads];
    if (count && blockIdx.x == 0 && tid == 0)
        *count += 1;
#pragma unroll 8
    for (int k = tid; k < nW / 4; k += T) {
        reinterpret_cast<float4 *>(sW)[k] = reinterpret_cast<const float4 *>(pp)[k];
        reinterpret_cast<float4 *>(sG)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float const inv = 1.f / static_cast<float>(v.n * v.w[L]);
    float loss = 0.f;
    int const tiles = (v.n + kTile16 - 1) / kTile16;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        int const s0 = t * kTile16;
        __syncthreads(); // weights in place; the previous tile is done with
        for (int k = tid; k < kTile16 * v.w[0]; k += T) {
            int const s = k / v.w[0], i = k % v.w[0];
            sA[i * kTileP + s] = s0 + s < v.n ? X[static_cast<size_t>(s0 + s) * v.w[0] + i] : 0.f;
        }
        __syncthreads();
        // forward: a thread forms 2 samples of one output
        int a0 = 0, o0 = 0;
        for (int l = 0; l < L; ++l) {
            int const in = v.w[l], out = v.w[l + 1], row = out + 1;
            const float *x = sA + kTileP * a0;
            float *A = sA + kTileP * (a0 + in), *D = sD + kTileP * (a0 + in);
            for (int k = tid; k < out * (kTile16 / 2); k += T) {
                int const o = k % out, q = 2 * (k / out);
                const float *W = sW + o0 + o;
                float2 z = make_float2(W[in * row], W[in * row]);
#pragma unroll 8
                for (int i = 0; i < in; ++i) {
                    float const w = W[i * row];
                    float2 const a = *reinterpret_cast<const float2 *>(x + i * kTileP + q);
                    z.x = fmaf(a.x, w, z.x);
                    z.y = fmaf(a.y, w, z.y);
                }
                if (l + 1 < L) {
                    *reinterpret_cast<float2 *>(D + o * kTileP + q) =
                        make_float2(gelu_d(z.x), gelu_d(z.y));
                    z = make_float2(gelu(z.x), gelu(z.y));
                }
                *reinterpret_cast<float2 *>(A + o * kTileP + q) = z;
            }
            a0 += in;
            o0 += (in + 1) * row;
            __syncthreads();
        }
        // loss and its derivative
        for (int k = tid; k < kTile16 * v.w[L]; k += T) {
            int const s = k / v.w[L], o = k % v.w[L];
            float d = 0.f;
            if (s0 + s < v.n) {
                d = sA[(a0 + o) * kTileP + s] - Y[static_cast<size_t>(s0 + s) * v.w[L] + o];
                loss = fmaf(d, d, loss);
            }
            sP[o * kTileP + s] = 2.f * d * inv;
        }
        __syncthreads();
        // backward: sP holds dZ of layer l + 1
        for (int l = L - 1; l >= 0; --l) {
            int const in = v.w[l], out = v.w[l + 1], row = out + 1;
            a0 -= in;
            o0 -= (in + 1) * row;
            // weight gradients: lanes along the outputs, a thread every (T / out)-th input
            // (or, wider than the block, several outputs); the bias is the row after the inputs
            const float *x = sA + kTileP * a0;
            int const groups = max(1, T / out);
            for (int o = tid % out; o < out && tid < groups * out; o += T) {
                float dz[kTile16];
#pragma unroll
                for (int q = 0; q < kTile16; q += 4) {
                    float4 const d = *reinterpret_cast<const float4 *>(sP + o * kTileP + q);
                    dz[q] = d.x;
                    dz[q + 1] = d.y;
                    dz[q + 2] = d.z;
                    dz[q + 3] = d.w;
                }
                // two inputs at a time: two independent chains of FMAs in sample order
                for (int i = tid / out; i < in; i += 2 * groups) {
                    int const i1 = min(i + groups, in - 1);
                    float g = sG[o0 + i * row + o], g1 = sG[o0 + i1 * row + o];
#pragma unroll
                    for (int q = 0; q < kTile16; q += 4) {
                        float4 const a = *reinterpret_cast<const float4 *>(x + i * kTileP + q),
                                     b = *reinterpret_cast<const float4 *>(x + i1 * kTileP + q);
                        g = fmaf(a.x, dz[q], g);
                        g1 = fmaf(b.x, dz[q], g1);
                        g = fmaf(a.y, dz[q + 1], g);
                        g1 = fmaf(b.y, dz[q + 1], g1);
                        g = fmaf(a.z, dz[q + 2], g);
                        g1 = fmaf(b.z, dz[q + 2], g1);
                        g = fmaf(a.w, dz[q + 3], g);
                        g1 = fmaf(b.w, dz[q + 3], g1);
                    }
                    sG[o0 + i * row + o] = g;
                    if (i + groups < in)
                        sG[o0 + i1 * row + o] = g1;
                }
                if (tid < out || out > T) {
                    float g = sG[o0 + in * row + o];
#pragma unroll
                    for (int q = 0; q < kTile16; ++q)
                        g += dz[q];
                    sG[o0 + in * row + o] = g;
                }
            }
            // dZ of layer l = dA gelu'(z)
            if (l > 0) {
                const float *D = sD + kTileP * a0;
                for (int k = tid; k < in * (kTile16 / 2); k += T) {
                    int const i = k % in, q = 2 * (k / in);
                    const float *W = sW + o0 + i * row;
                    float2 a = make_float2(0.f, 0.f);
#pragma unroll 8
                    for (int o = 0; o < out; ++o) {
                        float const w = W[o];
                        float2 const d = *reinterpret_cast<const float2 *>(sP + o * kTileP + q);
                        a.x = fmaf(d.x, w, a.x);
                        a.y = fmaf(d.y, w, a.y);
                    }
                    float2 const g = *reinterpret_cast<const float2 *>(D + i * kTileP + q);
                    *reinterpret_cast<float2 *>(sQ + i * kTileP + q) =
                        make_float2(a.x * g.x, a.y * g.y);
                }
                __syncthreads();
                float *const u = sP;
                sP = sQ;
                sQ = u;
            }
        }
    }
    s_loss[tid] = loss;
    __syncthreads();
    for (int w = T / 2; w > 0; w >>= 1) {
        if (tid < w)
            s_loss[tid] += s_loss[tid + w];
        __syncthreads();
    }
    if (tid == 0)
        part_loss[blockIdx.x] = s_loss[0];
    float4 *out_p = reinterpret_cast<float4 *>(part + static_cast<size_t>(blockIdx.x) * nW);
    for (int k = tid; k < nW / 4; k += T)
        out_p[k] = reinterpret_cast<float4 *>(sG)[k];
}

// The blocks' gradients added in block order (4 threads of a parameter take every fourth block,
// their sums are added in order), then Adam (lr > 0) with the step counter k_step_grad advanced.
// Block 0 adds the loss sums.
constexpr int kUpdateThreads = 256;
__global__ void __launch_bounds__(kUpdateThreads)
    k_step_update(NetView v, const float *part, const float *part_loss, int n_part, float inv_m,
                  float *g, float *loss, float *p, float *pp, float *m1, float *m2, float lr,
                  const int *t) {
    mdelast::chain_begin();
    __shared__ float s_g[3][64];
    int const c = threadIdx.x & 63, q = threadIdx.x >> 6, np = padded_params(v);
    int const k = blockIdx.x * 64 + c;
    float a = 0.f;
    if (k < np)
#pragma unroll 16
        for (int b = q; b < n_part; b += 4)
            a += part[static_cast<size_t>(b) * np + k];
    if (q > 0)
        s_g[q - 1][c] = a;
    __syncthreads();
    int const u = q == 0 && k < np ? unpadded(v, k) : -1;
    if (u >= 0) {
        float const gk = ((a + s_g[0][c]) + s_g[1][c]) + s_g[2][c];
        g[u] = gk;
        if (lr > 0.f) {
            adam(p, m1, m2, u, gk, lr, static_cast<float>(*t));
            pp[k] = p[u];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x >= kUpdateThreads - 32) {
        float sum = 0.f;
        for (int b = threadIdx.x & 31; b < n_part; b += 32)
            sum += part_loss[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            sum += __shfl_down_sync(0xffffffffu, sum, o);
        if ((threadIdx.x & 31) == 0)
            *loss = sum * inv_m;
    }
}

unsigned blocks(long m) { return static_cast<unsigned>((m + kT - 1) / kT); }

} // namespace

#define MCK(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return fail(MDELAST_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_));            \
    } while (0)

struct mdelast_mlp_s {
    int device = 0;
    int L = 0;                  // layers
    std::vector<int> w;         // widths, L + 1
    std::vector<long> off_w, off_b;
    long np = 0;
    cudaStream_t stream = nullptr;
    float *p = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;
    int *t = nullptr;
    // activations for a batch of cap samples: per layer Z and A; A[0] is the input
    int cap = 0;
    std::vector<float *> Z, A, dA;
    float *Yt = nullptr, *dZ = nullptr, *loss = nullptr, *act = nullptr;
    // the two-kernel step: per-block gradients and loss sums (for the blocks of cap samples)
    bool fused = false;
    size_t fused_smem = 0;
    float *part = nullptr, *part_loss = nullptr, *pp = nullptr; // pp: the padded parameters
    NetView view(int n) const {
        NetView v{};
        v.L = L;
        v.np = static_cast<int>(np);
        v.n = n;
        for (int l = 0; l <= L; ++l) {
            v.w[l] = w[l];
            v.wsum += w[l];
            if (l < L)
                v.off_w[l] = static_cast<int>(off_w[l]);
        }
        return v;
    }
    // the padded copy of the current parameters, which the steps then keep
    void begin_fused() {
        NetView const v = view(1);
        k_step_params<<<(padded_params(v) + 255) / 256, 256, 0, stream>>>(v, p, pp);
    }
    // gradients into g and the loss; an Adam step when lr > 0
    int step_fused(int n, float lr) {
        int const nb = std::min((n + kTile16 - 1) / kTile16, kStepBlocks);
        NetView const v = view(n);
        MCK(mdelast::launch_chain(k_step_grad, nb, kStepThreads, fused_smem, stream, v, A[0], Yt,
                                  pp, part, part_loss, lr > 0.f ? t : nullptr));
        MCK(mdelast::launch_chain(k_step_update, (padded_params(v) + 63) / 64, kUpdateThreads, 0,
                                  stream, v, part, part_loss, nb,
                                  1.f / static_cast<float>(n * w[L]), g, loss, p, pp, m1, m2, lr,
                                  t));
        return MDELAST_OK;
    }
    cudaGraphExec_t graph = nullptr;
    int graph_n = -1;
    float graph_lr = 0.f;

    ~mdelast_mlp_s() {
        cudaSetDevice(device);
        if (graph)
            cudaGraphExecDestroy(graph);
        cudaFree(p);   // the slab of all that is sized by the parameters
        cudaFree(act); // ... and by the samples
        if (stream)
            cudaStreamDestroy(stream);
    }

    int reserve(int n) {
        if (n <= cap)
            return MDELAST_OK;
        if (graph) {
            cudaGraphExecDestroy(graph);
            graph = nullptr;
            graph_n = -1;
        }
        cudaFree(act);
        act = nullptr;
        cap = 0;
        // one allocation for everything sized by the samples (14 of them, and per-block sums for 148
        // blocks whatever the batch: creation and the first 200 steps of 2,048 samples 6.2 ms, now 5.3)
        int wmax = 0;
        size_t total = 0;
        auto at = [&](size_t floats) {
            size_t const o = total;
            total += (floats + 63) / 64 * 64;
            return o;
        };
        size_t const m = static_cast<size_t>(n);
        std::vector<size_t> oA, oD, oZ;
        for (int k = 0; k <= L; ++k) {
            oA.push_back(at(m * w[k]));
            oD.push_back(at(m * w[k]));
            oZ.push_back(k > 0 ? at(m * w[k]) : 0);
            wmax = std::max(wmax, w[k]);
        }
        size_t const oY = at(m * w[L]), odZ = at(m * wmax);
        size_t const nb = static_cast<size_t>(std::min((n + kTile16 - 1) / kTile16, kStepBlocks));
        size_t const oP = at(fused ? nb * padded_params(view(1)) : 0), oL = at(fused ? nb : 0);
        MCK(cudaMalloc(&act, sizeof(float) * total));
        Z.assign(L + 1, nullptr);
        A.assign(L + 1, nullptr);
        dA.assign(L + 1, nullptr);
        for (int k = 0; k <= L; ++k) {
            A[k] = act + oA[k];
            dA[k] = act + oD[k];
            if (k > 0)
                Z[k] = act + oZ[k];
        }
        Yt = act + oY;
        dZ = act + odZ;
        part = act + oP;
        part_loss = act + oL;
        cap = n;
        return MDELAST_OK;
    }

    void forward(int n, cudaStream_t s) {
        for (int l = 0; l < L; ++l)
            k_fwd<<<blocks(static_cast<long>(n) * w[l + 1]), kT, 0, s>>>(
                A[l], p + off_w[l], p + off_b[l], Z[l + 1], A[l + 1], n, w[l], w[l + 1],
                l + 1 < L);
    }

    // gradients of the mean-squared error of A[L] against Yt into g
    void backward(int n, cudaStream_t s) {
        k_loss<<<1, kT, 0, s>>>(A[L], Yt, dA[L], loss, n * w[L]);
        for (int l = L - 1; l >= 0; --l) {
            long const m = static_cast<long>(n) * w[l + 1];
            const float *dz = dA[l + 1];
            if (l + 1 < L) {
                k_bwd_act<<<blocks(m), kT, 0, s>>>(dA[l + 1], Z[l + 1], dZ, static_cast<int>(m));
                dz = dZ;
            }
            k_bwd_dw<<<blocks(static_cast<long>(w[l]) * w[l + 1] + w[l + 1]), kT, 0, s>>>(
                A[l], dz, g + off_w[l], g + off_b[l], n, w[l], w[l + 1]);
            if (l > 0)
                k_bwd_dx<<<blocks(static_cast<long>(n) * w[l]), kT, 0, s>>>(
                    dz, p + off_w[l], dA[l], n, w[l], w[l + 1]);
        }
    }

    int upload(const float *x, const float *y, int n) {
        if (int rc = reserve(n))
            return rc;
        MCK(cudaMemcpyAsync(A[0], x, sizeof(float) * static_cast<size_t>(n) * w[0],
                            cudaMemcpyHostToDevice, stream));
        if (y)
            MCK(cudaMemcpyAsync(Yt, y, sizeof(float) * static_cast<size_t>(n) * w[L],
                                cudaMemcpyHostToDevice, stream));
        return MDELAST_OK;
    }
};

extern "C" {

int mdelast_mlp_create(int32_t n_layers, const int32_t *widths, uint64_t seed, int32_t device,
                       mdelast_mlp **out) {
    clear_error();
    if (!widths || !out || n_layers < 1 || n_layers > MDELAST_MLP_MAX_LAYERS)
        return fail(MDELAST_ERR_ARGUMENT, "an MLP needs 1..%d layers", MDELAST_MLP_MAX_LAYERS);
    for (int k = 0; k <= n_layers; ++k)
        if (widths[k] < 1 || widths[k] > 4096)
            return fail(MDELAST_ERR_ARGUMENT, "layer width %d out of range", widths[k]);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(MDELAST_ERR_NO_DEVICE, "no CUDA device: the MLP kernels need one");
    }
    if (device < 0 || device >= ndev)
        return fail(MDELAST_ERR_ARGUMENT, "device %d not present", device);
    MCK(cudaSetDevice(device));
    auto *m = new mdelast_mlp_s();
    m->device = device;
    m->L = n_layers;
    m->w.assign(widths, widths + n_layers + 1);
    for (int l = 0; l < n_layers; ++l) {
        m->off_w.push_back(m->np);
        m->np += static_cast<long>(m->w[l]) * m->w[l + 1];
        m->off_b.push_back(m->np);
        m->np += m->w[l + 1];
    }
    // Glorot-normal weights, zero biases, from a 64-bit Mersenne Twister seeded by `seed`
    std::vector<float> h(static_cast<size_t>(m->np), 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < n_layers; ++l) {
        std::normal_distribution<double> nd(0., std::sqrt(2. / (m->w[l] + m->w[l + 1])));
        for (long k = 0; k < static_cast<long>(m->w[l]) * m->w[l + 1]; ++k)
            h[static_cast<size_t>(m->off_w[l] + k)] = static_cast<float>(nd(rng));
    }
    size_t const bytes = sizeof(float) * static_cast<size_t>(m->np);
    cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    // one allocation: p, g, m1, m2 (zero but p), the step counter, the loss, and the two-kernel
    // step's copy of the parameters
    m->fused_smem = step_smem(m->view(1));
    m->fused = m->fused_smem <= kStepSmemMax;
    size_t const np = (static_cast<size_t>(m->np) + 63) / 64 * 64,
                 npp = static_cast<size_t>(padded_params(m->view(1))),
                 extra = m->fused ? npp : 0;
    if (e == cudaSuccess)
        e = cudaMalloc(&m->p, sizeof(float) * (4 * np + 64 + extra));
    // in the order of the network's own stream, as everything that touches these buffers (that
    // stream does not wait for the legacy one), and complete on return
    if (e == cudaSuccess)
        e = cudaMemsetAsync(m->p, 0, sizeof(float) * (4 * np + 64), m->stream);
    m->g = m->p + np;
    m->m1 = m->p + 2 * np;
    m->m2 = m->p + 3 * np;
    m->t = reinterpret_cast<int *>(m->p + 4 * np);
    m->loss = m->p + 4 * np + 32;
    m->pp = m->p + 4 * np + 64;
    if (e == cudaSuccess && m->fused)
        e = cudaFuncSetAttribute(k_step_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kStepSmemMax));
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(m->p, h.data(), bytes, cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) {
        delete m;
        return fail(MDELAST_ERR_CUDA, "MLP set-up: %s", cudaGetErrorString(e));
    }
    *out = m;
    return MDELAST_OK;
}

void mdelast_mlp_destroy(mdelast_mlp *m) { delete m; }

int mdelast_mlp_n_params(const mdelast_mlp *m, int64_t *n) {
    clear_error();
    if (!m || !n)
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    *n = m->np;
    return MDELAST_OK;
}

int mdelast_mlp_get_params(mdelast_mlp *m, float *out) {
    clear_error();
    if (!m || !out)
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(m->device));
    MCK(cudaStreamSynchronize(m->stream));
    MCK(cudaMemcpy(out, m->p, sizeof(float) * static_cast<size_t>(m->np),
                   cudaMemcpyDeviceToHost));
    return MDELAST_OK;
}

int mdelast_mlp_set_params(mdelast_mlp *m, const float *in) {
    clear_error();
    if (!m || !in)
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(m->device));
    size_t const bytes = sizeof(float) * static_cast<size_t>(m->np);
    MCK(cudaMemcpyAsync(m->p, in, bytes, cudaMemcpyHostToDevice, m->stream));
    MCK(cudaMemsetAsync(m->m1, 0, bytes, m->stream)); // a new starting point resets the optimiser
    MCK(cudaMemsetAsync(m->m2, 0, bytes, m->stream));
    MCK(cudaMemsetAsync(m->t, 0, sizeof(int), m->stream));
    MCK(cudaStreamSynchronize(m->stream));
    return MDELAST_OK;
}

int mdelast_mlp_forward(mdelast_mlp *m, const float *x, int32_t n, float *y) {
    clear_error();
    if (!m || !x || !y || n < 1)
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(m->device));
    if (int rc = m->upload(x, nullptr, n))
        return rc;
    m->forward(n, m->stream);
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(y, m->A[m->L], sizeof(float) * static_cast<size_t>(n) * m->w[m->L],
                        cudaMemcpyDeviceToHost, m->stream));
    MCK(cudaStreamSynchronize(m->stream));
    return MDELAST_OK;
}

int mdelast_mlp_gradients(mdelast_mlp *m, const float *x, const float *y, int32_t n,
                          float *loss, float *grad) {
    clear_error();
    if (!m || !x || !y || n < 1)
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(m->device));
    if (int rc = m->upload(x, y, n))
        return rc;
    if (m->fused) {
        m->begin_fused();
        if (int rc = m->step_fused(n, 0.f))
            return rc;
    } else {
        m->forward(n, m->stream);
        m->backward(n, m->stream);
    }
    MCK(cudaGetLastError());
    if (loss)
        MCK(cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (grad)
        MCK(cudaMemcpyAsync(grad, m->g, sizeof(float) * static_cast<size_t>(m->np),
                            cudaMemcpyDeviceToHost, m->stream));
    MCK(cudaStreamSynchronize(m->stream));
    return MDELAST_OK;
}

int mdelast_mlp_train(mdelast_mlp *m, const float *x, const float *y, int32_t n,
                      int32_t steps, float lr, float *loss) {
    clear_error();
    if (!m || !x || !y || n < 1 || steps < 0 || !(lr > 0.f))
        return fail(MDELAST_ERR_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(m->device));
    if (int rc = m->upload(x, y, n))
        return rc;
    if (m->fused)
        m->begin_fused();
    for (int k = 0; m->fused && k < steps; ++k)
        if (int rc = m->step_fused(n, lr))
            return rc;
    if (!m->fused && (!m->graph || m->graph_n != n || m->graph_lr != lr)) {
        if (m->graph) {
            cudaGraphExecDestroy(m->graph);
            m->graph = nullptr;
        }
        cudaGraph_t gr = nullptr;
        MCK(cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
        m->forward(n, m->stream);
        m->backward(n, m->stream);
        k_adam<<<blocks(m->np), kT, 0, m->stream>>>(m->p, m->g, m->m1, m->m2,
                                                    static_cast<int>(m->np), lr, m->t);
        k_step_inc<<<1, 32, 0, m->stream>>>(m->t);
        cudaError_t const e = cudaStreamEndCapture(m->stream, &gr);
        if (e != cudaSuccess)
            return fail(MDELAST_ERR_CUDA, "capturing the training step: %s",
                        cudaGetErrorString(e));
        cudaError_t const e2 = cudaGraphInstantiate(&m->graph, gr, 0);
        cudaGraphDestroy(gr);
        if (e2 != cudaSuccess)
            return fail(MDELAST_ERR_CUDA, "instantiating the training step: %s",
                        cudaGetErrorString(e2));
        m->graph_n = n;
        m->graph_lr = lr;
    }
    for (int k = 0; !m->fused && k < steps; ++k)
        MCK(cudaGraphLaunch(m->graph, m->stream));
    if (loss) {
        // the loss of the parameters after the last step
        if (m->fused) {
            if (int rc = m->step_fused(n, 0.f))
                return rc;
        } else {
            m->forward(n, m->stream);
            m->backward(n, m->stream);
        }
        MCK(cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    }
    MCK(cudaStreamSynchronize(m->stream));
    return MDELAST_OK;
}

} // extern "C"
