// Launchers of the learned density estimator's elementwise and data-movement kernels
// (denoise_ops.cu).  NHWC activations, channel counts multiples of 8.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace rfk {

struct AdamLayer {
    uint32_t offset;  // of the layer's weights (then its biases) in the flat parameter arrays
    uint32_t cout, K, taps, ldf;
    __nv_bfloat16 *w16, *wf16;
};
constexpr int kMaxAdamLayers = 16;
struct AdamLayers {
    AdamLayer layer[kMaxAdamLayers];
};
// lr = 0 refreshes the bf16 copies only
cudaError_t launch_adam(float* w, const float* g, float* m, float* v, const AdamLayers& L, uint32_t layers, float lr,
                        float b1, float b2, float eps, uint32_t t, cudaStream_t st);
cudaError_t launch_features(const float4* bins, uint64_t n, float k2, const double* stats, const float4* base,
                            float level, __nv_bfloat16* out, cudaStream_t st);

}  // namespace rfk
