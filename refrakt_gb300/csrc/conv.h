// Tensor-core convolutions of the learned density estimator (conv.cu): 3x3 and 1x1, forward,
// input gradient and weight gradient, with the layer's elementwise work in their epilogues.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace rfk {

// What happens to a finished tile of outputs v[pixel][column]
enum ConvEpilogue : int {
    kConvStoreF32,    // C = v
    kConvAtomicF32,   // C += v
    kConvStoreBF16,   // C = relu(v + bias) as bf16; `pool` (may be null) its 2x2 averages
    kConvHead,        // out = clamp(base + v + bias, 0, 1), base = feature channels 4..6
    kConvL1,          // L1 loss of base + v + bias against target: dz = sign / (3 pixels), loss
    kConvMask,        // dz = v where y > 0 (ReLU backward), gb += its sums
    kConvConcat,      // columns < nlow: summed over 2x2 blocks, then as kConvMask at half
                      // resolution; the others to dskip
    kConvPool,        // dz = (dskip + v / 4) where y > 0 at twice the resolution, gb += its sums
};

struct ConvArgs {
    // input: NHWC, channels [0, ca) from xa (at half resolution, nearest-neighbour upsampled, when
    // up), [ca, ca + cb) from xb; zero outside the image
    const __nv_bfloat16* xa;
    const __nv_bfloat16* xb;
    uint32_t ca, cb;
    int up;
    uint32_t n, h, w;
    uint32_t taps;             // 9 (3x3) or 1 (1x1)
    const __nv_bfloat16* B;    // weights [N x taps (ca + cb)], row stride ldb, column tap (ca + cb) + c
    uint32_t N, ldb;
    // store modes
    void* C;                   // [pixels x N], row stride ldc
    uint32_t ldc;
    const float* bias;
    int relu;
    __nv_bfloat16* pool;
    // gradient modes; y, dz, dskip have as many channels as the columns they serve
    const __nv_bfloat16* y;
    __nv_bfloat16* dz;
    float* gb;
    float* dskip;
    uint32_t nlow;
    // head modes
    const __nv_bfloat16* feats;
    const float* target;
    float* out;
    double* loss;
    int* error;                // the caller's ErrorWord (error_word.h): conv_error's codes
};

// whether launch_conv takes the shape: ca + cb a multiple of 16 (or 8 channels in all), a tile's
// operands within an SM's shared memory and no more column groups than a grid has rows
bool conv_supported(uint32_t channels, uint32_t N, uint32_t taps);
cudaError_t launch_conv(const ConvArgs& a, ConvEpilogue epi, cudaStream_t st);
// what the wait that a code of ConvArgs.error names was for
inline const char* conv_error(int code) {
    return code == 1 ? "a stage to load" : code == 2 ? "an accumulator's release" : code == 3 ? "a loaded stage" : "an accumulator";
}

// gw[co][tap (ca + cb) + c] += sum over pixels of dz[p][co] x[p shifted by tap][c] for every task in
// one launch; of `conv` xa, xb, ca, cb, up, n, h, w, taps and dz (ldz channels per
// pixel, a multiple of 8, ldz >= cout) are read (a 1x1 kernel: w a multiple of 8)
struct WgradTask {
    ConvArgs conv;
    uint32_t cout, ldz;
    float* gw;
};
constexpr int kMaxWgradLayers = 16;
// with bias_dz (8 channels per pixel, the head's dz) also the head's bias gradient into bias_gb[0..2]
cudaError_t launch_conv_wgrad(const WgradTask* tasks, uint32_t count, const __nv_bfloat16* bias_dz, uint64_t bias_pixels,
                              float* bias_gb, int* error, cudaStream_t st);

}  // namespace rfk
