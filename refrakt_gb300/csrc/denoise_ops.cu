// Elementwise kernels of the learned density estimator (a small U-Net whose convolutions run on the
// tensor cores, conv.cu): the optimiser and the input features.  Activations are NHWC with the
// channel count a multiple of 8, so every pixel's channels are whole 16-byte vectors of bf16.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "denoise_ops.h"

namespace rfk {

namespace {

// Adam on the FP32 master weights of every layer in one launch (blockIdx.y = layer): w, g, m, v are
// flat over the network (each layer's weights, then its biases).  Refreshes the bf16 copy used as
// the forward operand (w16, [cout x K]) and the flipped transpose used by the input gradient
// (wf16[ci][tap' * cout + co] = w[co][(8 - tap') * C + ci], C = K / 9), or for a 1x1 layer (taps = 1)
// the plain transpose wf16[ci][co] = w[co][ci] with its row stride ldf.
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, const __grid_constant__ AdamLayers L, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
    const AdamLayer& l = L.layer[blockIdx.y];
    const uint32_t nw = l.cout * l.K, n = nw + l.cout;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t o = l.offset + i;
        float wi = w[o];
        if (lr > 0.0f) {
            const float gi = g[o];
            const float mi = b1 * m[o] + (1.0f - b1) * gi;
            const float vi = b2 * v[o] + (1.0f - b2) * gi * gi;
            m[o] = mi;
            v[o] = vi;
            wi -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
            w[o] = wi;
        }
        if (i >= nw) continue;  // a bias
        const __nv_bfloat16 b = __float2bfloat16_rn(wi);
        l.w16[i] = b;
        const uint32_t co = i / l.K, k = i % l.K;
        const uint32_t C = l.K / l.taps, tap = k / C, ci = k % C;
        l.wf16[(uint64_t)ci * l.ldf + (uint64_t)(l.taps - 1 - tap) * l.cout + co] = b;
    }
}

// input features of a histogram (RGBA sums float4 per bin, W x H): 8 bf16 channels
//   [0] l = log10(1 + a * k2), [1..3] colour * l / a — the tonemap's log-density scaling
//   (tonemap.glsl:18-26) without the gamma step; [4..6] the plain path's tonemapped RGB of the
//   same histogram (base, may be null: zeros), on which the network predicts a residual;
//   [7] `level`, the caller's code of the run's sample count (the noise level)
__global__ void features_kernel(const float4* __restrict__ bins, uint64_t n, float k2, const double* __restrict__ stats,
                                const float4* __restrict__ base, float level, __nv_bfloat16* __restrict__ out) {
    const float k = k2 > 0.0f ? k2 : (float)((double)n / fmax(stats[0], 1e-30));
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float4 c = bins[i];
        __align__(16) __nv_bfloat16 f[8];
        float l = 0.0f, s = 0.0f;
        if (c.w > 0.0f) {
            l = log10f(1.0f + c.w * k);
            s = l / c.w;
        }
        f[0] = __float2bfloat16_rn(l);
        f[1] = __float2bfloat16_rn(c.x * s);
        f[2] = __float2bfloat16_rn(c.y * s);
        f[3] = __float2bfloat16_rn(c.z * s);
        const float4 bb = base ? base[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        f[4] = __float2bfloat16_rn(bb.x);
        f[5] = __float2bfloat16_rn(bb.y);
        f[6] = __float2bfloat16_rn(bb.z);
        f[7] = __float2bfloat16_rn(level);
        *reinterpret_cast<uint4*>(out + i * 8) = *reinterpret_cast<const uint4*>(f);
    }
}

unsigned grid_for(uint64_t n, unsigned threads) {
    const uint64_t g = (n + threads - 1) / threads;
    return (unsigned)(g < 152ull * 32 ? (g ? g : 1) : 152ull * 32);
}

}  // namespace

cudaError_t launch_adam(float* w, const float* g, float* m, float* v, const AdamLayers& L, uint32_t layers, float lr,
                        float b1, float b2, float eps, uint32_t t, cudaStream_t st) {
    const float c1 = 1.0f - powf(b1, (float)(t ? t : 1)), c2 = 1.0f - powf(b2, (float)(t ? t : 1));
    adam_kernel<<<dim3(64, layers), 256, 0, st>>>(w, g, m, v, L, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

cudaError_t launch_features(const float4* bins, uint64_t n, float k2, const double* stats, const float4* base,
                            float level, __nv_bfloat16* out, cudaStream_t st) {
    features_kernel<<<grid_for(n, 256), 256, 0, st>>>(bins, n, k2, stats, base, level, out);
    return cudaGetLastError();
}

}  // namespace rfk
