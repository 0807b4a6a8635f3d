// Kernels of the learned tracklet pre-filter: weight packing, tensor-core
// scoring of feature rows, and the training step (forward + backward on the
// CUDA cores with the inference path's BF16 roundings, then Adam).
#include <cstdio>

#include "sdl_mlp.h"

namespace sdlg {

namespace {

// FP32 parameters -> packed BF16 tiles [W1 b1], W2, b2 and the FP32 tail
// (BF16-rounded w3, b3, threshold)
__global__ void k_mlp_pack(const float* __restrict__ p, unsigned char* __restrict__ pack, float thr) {
    for (int e = threadIdx.x; e < kMlpHid * kMlpK1; e += blockDim.x) {
        const int n = e / kMlpK1, k = e % kMlpK1;
        const float w = k < kMlpIn ? p[kMlpW1 + n * kMlpIn + k] : (k == kMlpIn ? p[kMlpB1 + n] : 0.f);
        *reinterpret_cast<uint16_t*>(pack + kPackW1 + cm_offset(n, k, 2)) = bf16_bits(w);
    }
    for (int e = threadIdx.x; e < kMlpHid * kMlpK2; e += blockDim.x) {
        const int n = e / kMlpK2, k = e % kMlpK2;
        *reinterpret_cast<uint16_t*>(pack + kPackW2 + cm_offset(n, k, 8)) = bf16_bits(p[kMlpW2 + n * kMlpHid + k]);
    }
    for (int e = threadIdx.x; e < kMlpHid * 16; e += blockDim.x) {
        const int n = e / 16, k = e % 16;
        *reinterpret_cast<uint16_t*>(pack + kPackB2 + cm_offset(n, k, 2)) = k == 0 ? bf16_bits(p[kMlpB2 + n]) : (uint16_t)0;
    }
    for (int n = threadIdx.x; n < kMlpHid; n += blockDim.x) reinterpret_cast<float*>(pack + kPackW3)[n] = bf16_round(p[kMlpW3 + n]);
    if (threadIdx.x == 0) {
        float* tail = reinterpret_cast<float*>(pack + kPackB3);
        tail[0] = p[kMlpB3];
        tail[1] = thr;
        tail[2] = 0.f;
        tail[3] = 0.f;
    }
}

// logits of n feature rows (row-major n x 12), one 128-row tile per step
__global__ void __launch_bounds__(kMlpTile) k_mlp_score(const float* __restrict__ x, int64_t n,
                                                        const unsigned char* __restrict__ pack, float* __restrict__ logits,
                                                        unsigned int* __restrict__ status) {
    __shared__ MlpSmem sm;
    mlp_setup(sm, pack);
    MlpThread st;
    const int64_t ntile = (n + kMlpTile - 1) / kMlpTile;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int64_t r = tile * kMlpTile + threadIdx.x;
        float f[kMlpIn];
#pragma unroll
        for (int k = 0; k < kMlpIn; ++k) f[k] = r < n ? x[r * kMlpIn + k] : 0.f;
        const float z = mlp_tile(sm, f, st);
        if (r < n) logits[r] = z;
    }
    if (st.abort && threadIdx.x == 0) atomicOr(status, 1u);
    mlp_teardown(sm, st);
}

// ------------------------------------------------------------------ training
// A tile of 128 samples in six products on the FP32 cores (forward layers 1
// and 2, dLoss/da1, the gradients of W2 and W1), each thread holding a block
// of the result: 8 samples x 4 units of an activation, 4 x 4 of gW2, 1 x 3 of
// gW1.  Activations are kept unit by unit, samples consecutive (kLdM apart):
// the products over units read 8 samples of a unit, those over samples 4
// samples of a row, all as 16-byte loads without bank conflicts (a row is
// 4 banks past the one before).  Every activation is one thread's sum in
// index order, as written in the network's definition.  The weight gradients
// stay in registers over all of a CTA's tiles and reach memory by one atomic
// per CTA and parameter.  111 KB of shared memory: two CTAs per SM, so that one
// computes while the other waits.  Bound by the FP32 pipes: 98 us of
// multiply-adds for 262,144 samples, which take 190 us.  (A thread per sample
// with its units in shared memory took 1,023 us.)
constexpr int kTrainRows = 128;     // samples per tile
constexpr int kTrainThreads = 256;
constexpr int kLdM = kTrainRows + 4;

struct TrainSmem {
    float h1[kMlpHid][kLdM];     // BF16-rounded ReLU outputs of layer 1, then dLoss/da1
    float d2[kMlpHid][kLdM];     // partial logits, then dLoss/da2
    float x[kMlpIn][kLdM];       // BF16-rounded features
    float w2[kMlpHid][kMlpHid];  // BF16-rounded weights: W2[n][j]
    float w2t[kMlpHid][kMlpHid]; // W2[n][j] at [j][n]
    float w1t[kMlpIn][kMlpHid];  // W1[n][k] at [k][n]
    float b1[kMlpHid], b2[kMlpHid], w3[kMlpHid];
    float dz[kTrainRows];
};
constexpr int kNG = kTrainThreads / 16;  // unit groups of 4

__device__ __forceinline__ float sigmoid_f(float z) {
    if (z >= 0.f) return 1.f / (1.f + expf(-z));
    const float e = expf(z);
    return e / (1.f + e);
}
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
// acc[8 samples][4 units] += a[8 samples] x w[4 units]
__device__ __forceinline__ void outer8x4(float (&acc)[8][4], float4 a0, float4 a1, float4 w) {
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, b[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __fmaf_rn(b[j], a[i], acc[i][j]);
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
    c = __fmaf_rn(a.x, b.x, c);
    c = __fmaf_rn(a.y, b.y, c);
    c = __fmaf_rn(a.z, b.z, c);
    return __fmaf_rn(a.w, b.w, c);
}

// Forward and backward over `count` samples (ids order[start + i], or
// start + i when order is null); adds inv_norm * sum_i w_i dLoss_i/dparam
// into grad and the weighted loss sum into loss.  Weighted logistic loss:
// w_i * (softplus(z_i) - y_i z_i).  The BF16 roundings of the forward pass
// are treated as the identity in the backward pass.
__global__ void __launch_bounds__(kTrainThreads, 2)
    k_mlp_fwd_bwd(const float* __restrict__ X, const float* __restrict__ Y, const float* __restrict__ Wt,
                  const int32_t* __restrict__ order, int64_t start, int64_t count, float pos_weight, float inv_norm,
                  const float* __restrict__ params, float* __restrict__ grad, double* __restrict__ loss) {
    extern __shared__ __align__(16) unsigned char smraw[];
    TrainSmem& sm = *reinterpret_cast<TrainSmem*>(smraw);
    const int t = threadIdx.x, lane = t & 31;
    for (int e = t; e < kMlpHid * kMlpHid; e += kTrainThreads) {
        const float v = bf16_round(params[kMlpW2 + e]);
        sm.w2[e / kMlpHid][e % kMlpHid] = v;
        sm.w2t[e % kMlpHid][e / kMlpHid] = v;
    }
    for (int e = t; e < kMlpHid * kMlpIn; e += kTrainThreads) sm.w1t[e % kMlpIn][e / kMlpIn] = bf16_round(params[kMlpW1 + e]);
    if (t < kMlpHid) {
        sm.b1[t] = bf16_round(params[kMlpB1 + t]);
        sm.b2[t] = bf16_round(params[kMlpB2 + t]);
        sm.w3[t] = bf16_round(params[kMlpW3 + t]);
    }
    const float b3 = params[kMlpB3];
    // this thread's samples m0 .. m0 + 3 and m0 + 64 .. m0 + 67, units n0 .. n0 + 3
    const int m0 = (t % 16) * 4, n0 = (t / 16) * 4;
    // its block of gW2: rows n0 + r, columns (t % 16) + 16 c; of gW1: row t / 4, columns 3 (t % 4) + c
    float g2[4][4] = {}, g1[3] = {}, gw3[4] = {}, gb2[4] = {}, gb1[4] = {}, gb3 = 0.f;
    double ls = 0.0;
    const int64_t ntile = (count + kTrainRows - 1) / kTrainRows;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        __syncthreads();  // the weights are there; the previous tile's products have read h1 and x
        float y = 0.f, wt = 0.f;
        if (t < kTrainRows) {
            const int64_t i = tile * kTrainRows + t;
            float f[kMlpIn] = {};
            if (i < count) {
                const int64_t id = order ? (int64_t)order[start + i] : start + i;
                y = Y[id];
                wt = Wt ? Wt[id] : (y > 0.5f ? pos_weight : 1.f);
#pragma unroll
                for (int k = 0; k < kMlpIn; k += 4) *reinterpret_cast<float4*>(f + k) = ld4(X + id * kMlpIn + k);
            }
#pragma unroll
            for (int k = 0; k < kMlpIn; ++k) sm.x[k][t] = bf16_round(f[k]);
        }
        __syncthreads();
        // layer 1
        float acc[8][4] = {};
#pragma unroll
        for (int k = 0; k < kMlpIn; ++k) outer8x4(acc, ld4(&sm.x[k][m0]), ld4(&sm.x[k][m0 + 64]), ld4(&sm.w1t[k][n0]));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = bf16_round(fmaxf(__fadd_rn(acc[i][j], sm.b1[n0 + j]), 0.f));
            st4(&sm.h1[n0 + j][m0], v);
            st4(&sm.h1[n0 + j][m0 + 64], v + 4);
        }
        __syncthreads();
        // layer 2 and this thread's share of the logits (h2 stays in acc)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 8
        for (int j = 0; j < kMlpHid; ++j) outer8x4(acc, ld4(&sm.h1[j][m0]), ld4(&sm.h1[j][m0 + 64]), ld4(&sm.w2t[j][n0]));
        {
            float z[8] = {};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaxf(__fadd_rn(acc[i][j], sm.b2[n0 + j]), 0.f);
                    z[i] = __fmaf_rn(sm.w3[n0 + j], acc[i][j], z[i]);
                }
            st4(&sm.d2[t / 16][m0], z);
            st4(&sm.d2[t / 16][m0 + 64], z + 4);
        }
        __syncthreads();
        if (t < kTrainRows) {
            float z = b3;
#pragma unroll
            for (int g = 0; g < kNG; ++g) z += sm.d2[g][t];
            const bool valid = tile * kTrainRows + t < count;
            const float dz = valid ? wt * (sigmoid_f(z) - y) * inv_norm : 0.f;
            sm.dz[t] = dz;
            gb3 += dz;
            if (valid) ls += (double)(wt * (softplus_f(z) - y * z));
        }
        __syncthreads();
        // dLoss/da2
        {
            const float4 za = ld4(&sm.dz[m0]), zb = ld4(&sm.dz[m0 + 64]);
            const float dz[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    gw3[j] = __fmaf_rn(dz[i], acc[i][j], gw3[j]);
                    v[i] = acc[i][j] > 0.f ? dz[i] * sm.w3[n0 + j] : 0.f;
                    gb2[j] += v[i];
                }
                st4(&sm.d2[n0 + j][m0], v);
                st4(&sm.d2[n0 + j][m0 + 64], v + 4);
            }
        }
        __syncthreads();
        // dLoss/da1
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 8
        for (int n = 0; n < kMlpHid; ++n) outer8x4(acc, ld4(&sm.d2[n][m0]), ld4(&sm.d2[n][m0 + 64]), ld4(&sm.w2[n][n0]));
        // gW2[n][j] += sum_m d2[m][n] h1[m][j]
#pragma unroll 2
        for (int m = 0; m < kTrainRows; m += 4) {
            float4 d[4], h[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                d[r] = ld4(&sm.d2[n0 + r][m]);
                h[r] = ld4(&sm.h1[t % 16 + 16 * r][m]);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) g2[r][c] = dot4(d[r], h[c], g2[r][c]);
        }
        // dLoss/da1 past the ReLU, in place of h1
        float v[4][8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 ha = ld4(&sm.h1[n0 + j][m0]), hb = ld4(&sm.h1[n0 + j][m0 + 64]);
            const float h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[j][i] = h[i] > 0.f ? acc[i][j] : 0.f;
                gb1[j] += v[j][i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            st4(&sm.h1[n0 + j][m0], v[j]);
            st4(&sm.h1[n0 + j][m0 + 64], v[j] + 4);
        }
        __syncthreads();
        // gW1[n][k] += sum_m d1[m][n] x[m][k]
#pragma unroll 4
        for (int m = 0; m < kTrainRows; m += 4) {
            const float4 d = ld4(&sm.h1[t / 4][m]);
#pragma unroll
            for (int c = 0; c < 3; ++c) g1[c] = dot4(d, ld4(&sm.x[3 * (t % 4) + c][m]), g1[c]);
        }
    }
    // the CTA's sums: sixteen threads (half a warp) share a unit group, the rest are one thread's
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            gw3[j] += __shfl_xor_sync(0xffffffffu, gw3[j], o);
            gb2[j] += __shfl_xor_sync(0xffffffffu, gb2[j], o);
            gb1[j] += __shfl_xor_sync(0xffffffffu, gb1[j], o);
        }
    for (int o = 16; o > 0; o >>= 1) {
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
        ls += __shfl_xor_sync(0xffffffffu, ls, o);
    }
    if (lane == 0 && t < kTrainRows) {
        atomicAdd(grad + kMlpB3, gb3);
        atomicAdd(loss, ls);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int c = 0; c < 4; ++c) atomicAdd(grad + kMlpW2 + (n0 + r) * kMlpHid + t % 16 + 16 * c, g2[r][c]);
        if (t % 16 == 0) {
            atomicAdd(grad + kMlpW3 + n0 + r, gw3[r]);
            atomicAdd(grad + kMlpB2 + n0 + r, gb2[r]);
            atomicAdd(grad + kMlpB1 + n0 + r, gb1[r]);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(grad + kMlpW1 + (t / 4) * kMlpIn + 3 * (t % 4) + c, g1[c]);
}

// Adam step on the FP32 master parameters; clears the gradient
__global__ void k_mlp_adam(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                           float lr, float c1, float c2) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < kMlpParams; e += gridDim.x * blockDim.x) {
        const float gr = g[e];
        const float mm = b1 * m[e] + (1.f - b1) * gr;
        const float vv = b2 * v[e] + (1.f - b2) * gr * gr;
        m[e] = mm;
        v[e] = vv;
        p[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
        g[e] = 0.f;
    }
}

}  // namespace

size_t mlp_train_smem() { return sizeof(TrainSmem); }

void launch_mlp_pack(const float* params, unsigned char* pack, float thr, cudaStream_t s) {
    k_mlp_pack<<<1, 256, 0, s>>>(params, pack, thr);
}

void launch_mlp_score(const float* x, int64_t n, const unsigned char* pack, float* logits, unsigned int* status, int n_sm,
                      cudaStream_t s) {
    if (n <= 0) return;
    const int64_t ntile = (n + kMlpTile - 1) / kMlpTile;
    const int64_t grid = ntile < (int64_t)n_sm * 4 ? ntile : (int64_t)n_sm * 4;
    k_mlp_score<<<(unsigned)grid, kMlpTile, 0, s>>>(x, n, pack, logits, status);
}

cudaError_t launch_mlp_fwd_bwd(const float* X, const float* Y, const float* W, const int32_t* order, int64_t start,
                               int64_t count, float pos_weight, float inv_norm, const float* params, float* grad,
                               double* loss, int n_sm, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_fwd_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
    if (e != cudaSuccess) return e;
    const int64_t ntile = (count + kTrainRows - 1) / kTrainRows;
    const unsigned grid = (unsigned)(ntile < 2 * (int64_t)n_sm ? ntile : 2 * (int64_t)n_sm);
    k_mlp_fwd_bwd<<<grid, kTrainThreads, sizeof(TrainSmem), s>>>(X, Y, W, order, start, count, pos_weight, inv_norm, params,
                                                                 grad, loss);
    return cudaGetLastError();
}

void launch_mlp_adam(float* p, float* g, float* m, float* v, float lr, float c1, float c2, cudaStream_t s) {
    k_mlp_adam<<<(kMlpParams + 255) / 256, 256, 0, s>>>(p, g, m, v, lr, c1, c2);
}

}  // namespace sdlg
