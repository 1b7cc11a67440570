// Training kernels of the learned closure's MLP (5 -> 32 -> 32 -> 1, ReLU,
// linear output): FP32 forward, mean-squared-error loss and gradient, and
// the Adam update. The gradient is deterministic: a fixed grid of blocks
// takes 32-sample tiles in a fixed order, each block keeps its parameter
// partial sums in registers, and one final kernel adds the per-block
// partials in a fixed order.
//
// A mini-batch is small (4096 samples are 14 M multiply-adds): what bounds it
// is the chain of loads, layers and barriers of one tile, not the arithmetic.
// So a tile is small enough that a 4096-sample batch is one tile for each of
// 128 blocks, and a tile's layers are spread over 256 threads; the sums over
// samples and blocks run in parallel. Every sum over inputs or hidden units
// runs in index order. B200, 4096 samples: gradient 35 -> 7.2 us, its final sum
// 15 -> 4.1 us (one thread per sample with 128-sample tiles, one thread per
// parameter over the blocks, before); forward over 32768 samples 8.5 -> 6.4 us.
#include <cuda_runtime.h>

#include <cstdint>

#include "fc_lbm.h"

namespace {

constexpr int kIn = 5, kH = 32;
constexpr int kW1 = 0, kB1 = kW1 + kIn * kH, kW2 = kB1 + kH, kB2 = kW2 + kH * kH, kW3 = kB2 + kH, kB3 = kW3 + kH;
constexpr int kP = kB3 + 1;
static_assert(kP == FC_MLP_PARAMS, "parameter count must match the header");
constexpr int kTile = 32;          // samples per tile: one per lane
constexpr int kGradThreads = 256;  // 8 warps, 4 hidden units each
constexpr int kGradBlocks = 148;
constexpr int kRow = 36;           // padded row of kTile samples: 8 rows' 16-byte vectors cover all banks
constexpr int kForwardThreads = 128;
static_assert(kH == 4 * (kGradThreads / 32) && kTile == 32, "unit groups and lanes");
static_assert((size_t)kGradBlocks * kP + 2 * kGradBlocks <= FC_MLP_GRAD_SCRATCH, "scratch size");

__device__ __forceinline__ float relu(float z) { return z > 0.0f ? z : 0.0f; }

// One sample per thread; the weights come as uniform 16-byte loads, four
// hidden units each.
__global__ void __launch_bounds__(kForwardThreads) k_mlp_forward(const float* __restrict__ params,
                                                                const float* __restrict__ x, int64_t n,
                                                                float* __restrict__ y) {
    __shared__ __align__(16) float w1[kH][8];  // unit j: its five weights and bias
    __shared__ __align__(16) float w2[kH * kH], b2[kH], w3[kH];
    __shared__ float b3;
    // every load first: one trip to memory, not one per value
    constexpr int kLoads = (kP + kForwardThreads - 1) / kForwardThreads;
    float pv[kLoads];
#pragma unroll
    for (int r = 0; r < kLoads; ++r) {
        const int p = threadIdx.x + r * kForwardThreads;
        pv[r] = p < kP ? params[p] : 0.0f;
    }
#pragma unroll
    for (int r = 0; r < kLoads; ++r) {
        const int p = threadIdx.x + r * kForwardThreads;
        const float v = pv[r];
        if (p < kB1) w1[p % kH][p / kH] = v;
        else if (p < kW2) w1[p - kB1][kIn] = v;
        else if (p < kB2) w2[p - kW2] = v;
        else if (p < kW3) b2[p - kB2] = v;
        else if (p < kB3) w3[p - kW3] = v;
        else if (p == kB3) b3 = v;
    }
    __syncthreads();
    for (int64_t s = (int64_t)blockIdx.x * kForwardThreads + threadIdx.x; s < n;
         s += (int64_t)gridDim.x * kForwardThreads) {
        float xi[kIn], z2[kH];
        for (int i = 0; i < kIn; ++i) xi[i] = x[s * kIn + i];
#pragma unroll
        for (int k = 0; k < kH; ++k) z2[k] = b2[k];
#pragma unroll 4
        for (int j = 0; j < kH; ++j) {
            float z = w1[j][kIn];
#pragma unroll
            for (int i = 0; i < kIn; ++i) z = fmaf(xi[i], w1[j][i], z);
            const float h = relu(z);
#pragma unroll
            for (int k = 0; k < kH; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(w2 + j * kH + k);
                z2[k] = fmaf(h, w.x, z2[k]);
                z2[k + 1] = fmaf(h, w.y, z2[k + 1]);
                z2[k + 2] = fmaf(h, w.z, z2[k + 2]);
                z2[k + 3] = fmaf(h, w.w, z2[k + 3]);
            }
        }
        float o = b3;
#pragma unroll
        for (int k = 0; k < kH; ++k) o = fmaf(relu(z2[k]), w3[k], o);
        y[s] = o;
    }
}

// Layers: lane = sample, warp = four hidden units, activations as rows over
// the tile's samples. Parameter gradients: thread (j, k) sums over the
// samples of its rows, four k per thread.
__global__ void __launch_bounds__(kGradThreads) k_mlp_grad(const float* __restrict__ params,
                                                          const float* __restrict__ x, const float* __restrict__ y,
                                                          const int64_t* __restrict__ idx, int64_t n,
                                                          float* __restrict__ partial,
                                                          double* __restrict__ loss_partial) {
    __shared__ __align__(16) float w[kP + 3];       // as params; W2 (and b2, w3 behind it) on 16-byte boundaries
    __shared__ __align__(16) float w2t[kH * kH];    // W2 transposed: [k][j]
    __shared__ __align__(16) float sx[kIn][kRow];
    __shared__ __align__(16) float sh1[kH][kRow], sz1[kH][kRow];  // layer 1: value, dL/dz
    __shared__ __align__(16) float sh2[kH][kRow], sz2[kH][kRow];  // layer 2
    __shared__ __align__(16) float sd[kRow];                      // dL/dout
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, u0 = 4 * warp;
    static_assert(kW2 % 4 == 0 && kB1 % 4 == 0 && kB2 % 4 == 0, "vector loads of the weights");
    constexpr int kLoads = (kP + kGradThreads - 1) / kGradThreads;  // every load first, as in k_mlp_forward
    float pv[kLoads];
#pragma unroll
    for (int r = 0; r < kLoads; ++r) {
        const int p = threadIdx.x + r * kGradThreads;
        pv[r] = p < kP ? params[p] : 0.0f;
    }
#pragma unroll
    for (int r = 0; r < kLoads; ++r) {
        const int p = threadIdx.x + r * kGradThreads;
        if (p < kP) w[p] = pv[r];
        if (p >= kW2 && p < kB2) w2t[(p - kW2) % kH * kH + (p - kW2) / kH] = pv[r];
    }
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, acc1 = 0.0f, acc3 = 0.0f;
    double lsum = 0.0;
    const int64_t tiles = (n + kTile - 1) / kTile;
    const float inv_n = 1.0f / (float)n;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t s = tile * kTile + lane;
        const bool live = s < n;
        float yt = 0.0f;
        if (warp < kIn) {  // warps 0-4 take an input each, and warp 0 the target
            const int64_t row = live ? (idx ? idx[s] : s) : 0;
            sx[warp][lane] = live ? x[row * kIn + warp] : 0.0f;
            if (warp == 0 && live) yt = y[row];
        }
        __syncthreads();
        float z1[4], z2[4];
        for (int u = 0; u < 4; ++u) z1[u] = w[kB1 + u0 + u];
        for (int i = 0; i < kIn; ++i) {
            const float xi = sx[i][lane];
            const float4 v = *reinterpret_cast<const float4*>(w + kW1 + i * kH + u0);
            z1[0] = fmaf(xi, v.x, z1[0]);
            z1[1] = fmaf(xi, v.y, z1[1]);
            z1[2] = fmaf(xi, v.z, z1[2]);
            z1[3] = fmaf(xi, v.w, z1[3]);
        }
        for (int u = 0; u < 4; ++u) sh1[u0 + u][lane] = live ? relu(z1[u]) : 0.0f;
        __syncthreads();
        for (int u = 0; u < 4; ++u) z2[u] = w[kB2 + u0 + u];
#pragma unroll 8
        for (int j = 0; j < kH; ++j) {
            const float h = sh1[j][lane];
            const float4 v = *reinterpret_cast<const float4*>(w + kW2 + j * kH + u0);
            z2[0] = fmaf(h, v.x, z2[0]);
            z2[1] = fmaf(h, v.y, z2[1]);
            z2[2] = fmaf(h, v.z, z2[2]);
            z2[3] = fmaf(h, v.w, z2[3]);
        }
        for (int u = 0; u < 4; ++u) sh2[u0 + u][lane] = live ? relu(z2[u]) : 0.0f;
        __syncthreads();
        if (warp == 0) {
            float o = w[kB3], d = 0.0f;
#pragma unroll
            for (int k = 0; k < kH; ++k) o = fmaf(sh2[k][lane], w[kW3 + k], o);
            if (live) {
                const float e = o - yt;
                lsum += (double)e * (double)e;
                d = 2.0f * e * inv_n;
            }
            sd[lane] = d;
            for (int off = 16; off > 0; off >>= 1) d += __shfl_down_sync(0xffffffffu, d, off);
            acc3 += d;  // lane 0: the tile's sum, for b3
        }
        __syncthreads();
        const float d = sd[lane];
        for (int u = 0; u < 4; ++u) sz2[u0 + u][lane] = live && z2[u] > 0.0f ? d * w[kW3 + u0 + u] : 0.0f;
        __syncthreads();
        float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
        for (int k = 0; k < kH; ++k) {
            const float z = sz2[k][lane];
            const float4 v = *reinterpret_cast<const float4*>(w2t + k * kH + u0);
            g[0] = fmaf(v.x, z, g[0]);
            g[1] = fmaf(v.y, z, g[1]);
            g[2] = fmaf(v.z, z, g[2]);
            g[3] = fmaf(v.w, z, g[3]);
        }
        for (int u = 0; u < 4; ++u) sz1[u0 + u][lane] = live && z1[u] > 0.0f ? g[u] : 0.0f;
        // W2: unit j of layer 1 with units k, k + 8, k + 16, k + 24 of layer 2
        const int j = u0 + (lane >> 3), k = lane & 7;
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < kTile; q += 4) {
            const float4 h = *reinterpret_cast<const float4*>(&sh1[j][q]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float4 z = *reinterpret_cast<const float4*>(&sz2[k + 8 * c][q]);
                a[c] = fmaf(h.x, z.x, a[c]);
                a[c] = fmaf(h.y, z.y, a[c]);
                a[c] = fmaf(h.z, z.z, a[c]);
                a[c] = fmaf(h.w, z.w, a[c]);
            }
        }
        for (int c = 0; c < 4; ++c) acc[c] += a[c];
        __syncthreads();
        // the other parameters, a warp each: W1's rows, b1, b2, w3 (lane = unit)
        float b = 0.0f;
        const float* zr = warp == 6 ? sz2[lane] : (warp == 7 ? sh2[lane] : sz1[lane]);
        const float* fr = warp < kIn ? sx[warp] : sd;
        const bool plain = warp == 5 || warp == 6;  // biases: the sum of dL/dz
#pragma unroll
        for (int q = 0; q < kTile; q += 4) {
            const float4 z = *reinterpret_cast<const float4*>(zr + q);
            const float4 f = *reinterpret_cast<const float4*>(fr + q);
            b = fmaf(plain ? 1.0f : f.x, z.x, b);
            b = fmaf(plain ? 1.0f : f.y, z.y, b);
            b = fmaf(plain ? 1.0f : f.z, z.z, b);
            b = fmaf(plain ? 1.0f : f.w, z.w, b);
        }
        acc1 += b;
        __syncthreads();
    }
    float* out = partial + (size_t)blockIdx.x * kP;
    for (int c = 0; c < 4; ++c) out[kW2 + (u0 + (lane >> 3)) * kH + (lane & 7) + 8 * c] = acc[c];
    out[(warp < 6 ? kW1 + warp * kH : (warp == 6 ? kB2 : kW3)) + lane] = acc1;  // b1 follows W1's five rows
    if (warp == 0) {
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
        if (lane == 0) {
            out[kB3] = acc3;
            loss_partial[blockIdx.x] = lsum;
        }
    }
}

// A block per 32 parameters: warp v adds the partials of blocks v, v + 16,
// ..., then the sixteen sums are added in order. Block 0 also adds the losses.
constexpr int kSumWarps = 16;
__global__ void __launch_bounds__(32 * kSumWarps) k_mlp_grad_final(const float* __restrict__ partial,
                                                        const double* __restrict__ loss_partial, int blocks, int64_t n,
                                                        float* __restrict__ grad, double* __restrict__ loss) {
    __shared__ float sum[kSumWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    float g = 0.0f;
    if (p < kP) {
        constexpr int kMost = (kGradBlocks + kSumWarps - 1) / kSumWarps;
        float v[kMost];
#pragma unroll
        for (int r = 0; r < kMost; ++r) {
            const int b = warp + r * kSumWarps;
            v[r] = b < blocks ? partial[(size_t)b * kP + p] : 0.0f;
        }
#pragma unroll
        for (int r = 0; r < kMost; ++r) g += v[r];
    }
    sum[warp][lane] = g;
    __syncthreads();
    if (warp == 0 && p < kP) {
        for (int v = 1; v < kSumWarps; ++v) g += sum[v][lane];
        grad[p] = g;
    }
    if (blockIdx.x == 0 && warp == 1 && loss) {
        double l = 0.0;
        for (int b = lane; b < blocks; b += 32) l += loss_partial[b];
        for (int off = 16; off > 0; off >>= 1) l += __shfl_down_sync(0xffffffffu, l, off);
        if (lane == 0) *loss = l / (double)n;
    }
}

__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kP) return;
    const float gp = g[p];
    const float mp = b1 * m[p] + (1.0f - b1) * gp;
    const float vp = b2 * v[p] + (1.0f - b2) * gp * gp;
    m[p] = mp;
    v[p] = vp;
    w[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

}  // namespace

extern "C" {

FC_LBM_API int fc_lbm_mlp_forward(const float* params, const float* x, int64_t n, float* y, void* stream) {
    if (!params || (n > 0 && (!x || !y)) || n < 0) return FC_LBM_ERR_INVALID_ARG;
    if (n == 0) return FC_LBM_OK;
    const int64_t blocks = (n + kForwardThreads - 1) / kForwardThreads;
    k_mlp_forward<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), kForwardThreads, 0, (cudaStream_t)stream>>>(
        params, x, n, y);
    return cudaGetLastError() == cudaSuccess ? FC_LBM_OK : FC_LBM_ERR_CUDA;
}

FC_LBM_API int fc_lbm_mlp_grad(const float* params, const float* x, const float* y, const int64_t* idx, int64_t n,
                               float* grad, double* loss, float* scratch, void* stream) {
    if (!params || !x || !y || !grad || !scratch || n <= 0) return FC_LBM_ERR_INVALID_ARG;
    float* partial = scratch;
    double* lp = reinterpret_cast<double*>(scratch + (size_t)kGradBlocks * kP + ((size_t)kGradBlocks * kP) % 2);
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t tiles = (n + kTile - 1) / kTile;
    const int blocks = (int)(tiles < kGradBlocks ? tiles : kGradBlocks);
    k_mlp_grad<<<blocks, kGradThreads, 0, s>>>(params, x, y, idx, n, partial, lp);
    if (cudaGetLastError() != cudaSuccess) return FC_LBM_ERR_CUDA;
    k_mlp_grad_final<<<(kP + 31) / 32, 32 * kSumWarps, 0, s>>>(partial, lp, blocks, n, grad, loss);
    return cudaGetLastError() == cudaSuccess ? FC_LBM_OK : FC_LBM_ERR_CUDA;
}

FC_LBM_API int fc_lbm_mlp_adam(float* params, const float* grad, float* m, float* v, int32_t step, float lr,
                               float beta1, float beta2, float eps, void* stream) {
    if (!params || !grad || !m || !v || step < 1) return FC_LBM_ERR_INVALID_ARG;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    k_adam<<<(kP + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, lr, beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? FC_LBM_OK : FC_LBM_ERR_CUDA;
}

}  // extern "C"
