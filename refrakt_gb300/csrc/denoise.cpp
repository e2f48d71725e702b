// Learned density estimation (no reference counterpart): a U-Net that maps a short-run histogram
// to the converged, tonemapped image.  Four levels of 32-48-64-96 channels, two 3x3 convolutions
// + ReLU per level, 2x2 average pooling down, nearest-neighbour upsampling and channel-concatenated
// skip connections up, a 1x1 output convolution to RGB.  Weights are FP32 masters with BF16 copies;
// every convolution and both of its gradients are tcgen05 BF16 kernels with FP32 accumulation
// (conv.cu) whose epilogues carry the elementwise work of the layer: bias, ReLU and the pooled copy
// going forward; the loss at the head; and going back the ReLU mask, the adjoints of pooling,
// upsampling and concatenation and the bias gradients, so each layer's output gradient is written
// once, as the BF16 operand that its weight- and input-gradient kernels read.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <algorithm>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "conv.h"
#include "denoise_ops.h"
#include "error_word.h"
#include "internal.h"
#include "kernels.h"
#include "scratch.h"
#include "refrakt.h"

using namespace rfk;

namespace {

struct Conv {
    uint32_t ca, cb, cout, taps;  // inputs: ca channels (upsampled when up) + cb skip channels
    int up, relu, level;
    int src_a, src_b;             // activation indices (-1 = network input / none)
    uint32_t K() const { return taps * (ca + cb); }
    uint32_t ldf() const { return (taps * cout + 7) & ~7u; }  // row stride of the flipped transpose
    size_t offset = 0;            // of the weights [cout x K], then the biases, in the flat parameter arrays
    float *b = nullptr, *gw = nullptr, *gb = nullptr;
    __nv_bfloat16 *w16 = nullptr, *wf16 = nullptr;
};

struct Act {  // one activation tensor (the output of conv i or of a pool)
    uint32_t c;
    int level;
    bool skip = false;           // also read by a decoder layer
    __nv_bfloat16* x = nullptr;  // bf16 [P_level x c]
    __nv_bfloat16* dz = nullptr; // gradient before the ReLU, same shape (the head: 8 channels per pixel)
    float* dskip = nullptr;      // FP32 gradient from the decoder layer that reads it, same shape
};

constexpr uint32_t kIn = 8;  // input feature channels (4 used)
const uint32_t kCh[4] = {32, 48, 64, 96};

}  // namespace

struct rf_denoiser {
    rf_denoiser_desc d{};
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<Conv> convs;
    std::vector<Act> acts;          // acts[i] = output of convs[i]; pools appended after
    int out_conv = -1;
    uint64_t P0 = 0;                // pixels at level 0 (max)
    uint32_t H = 0, W = 0, N = 0;   // current shape
    // parameters, gradients and Adam moments, flat over the layers (weights, then biases, of each)
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    AdamLayers adam{};
    double* loss = nullptr;
    uint32_t step = 0;
    ErrorWord error;                // of every convolution and weight-gradient launch
    std::vector<void*> allocs;
};

namespace {

int cuda_fail(cudaError_t e, const char* what) { return fail(RF_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)); }

// waits for the denoiser's stream; RF_ERR_TIMEOUT when a bounded wait of a kernel launched before ran out
int sync(rf_denoiser* D, const char* fn) {
    const cudaError_t e = cudaStreamSynchronize(D->stream);
    if (e != cudaSuccess) return cuda_fail(e, fn);
    if (const int code = D->error.take())
        return fail(RF_ERR_TIMEOUT, std::string(fn) + ": a convolution's wait for " + conv_error(code) + " ran out; the results are invalid");
    return RF_OK;
}

template <class T>
cudaError_t dalloc(rf_denoiser* d, T** p, size_t n, bool zero = false) {
    cudaError_t e = cudaMalloc((void**)p, n * sizeof(T) + 16);
    if (e == cudaSuccess) {
        d->allocs.push_back(*p);
        if (zero) e = cudaMemset(*p, 0, n * sizeof(T) + 16);
    }
    return e;
}

uint64_t level_pixels(uint32_t n, uint32_t h, uint32_t w, int level) {
    return (uint64_t)n * (h >> level) * (w >> level);
}

void build_graph(rf_denoiser* D) {
    auto conv = [&](uint32_t ca, uint32_t cb, uint32_t cout, int level, int src_a, int src_b, int up, uint32_t taps,
                    int relu) {
        Conv c{};
        c.ca = ca;
        c.cb = cb;
        c.cout = cout;
        c.level = level;
        c.src_a = src_a;
        c.src_b = src_b;
        c.up = up;
        c.taps = taps;
        c.relu = relu;
        D->convs.push_back(c);
        Act a{};
        a.c = cout;
        a.level = level;
        D->acts.push_back(a);
        return (int)D->convs.size() - 1;
    };
    // encoder
    int prev = -1;
    uint32_t cin = kIn;
    std::vector<int> skip(4, -1);
    for (int l = 0; l < 4; l++) {
        int a = conv(cin, 0, kCh[l], l, prev, -1, 0, 9, 1);
        int b = conv(kCh[l], 0, kCh[l], l, a, -1, 0, 9, 1);
        skip[l] = b;
        prev = b;
        cin = kCh[l];
    }
    // decoder
    int low = skip[3];
    for (int l = 2; l >= 0; l--) {
        int a = conv(kCh[l + 1], kCh[l], kCh[l], l, low, skip[l], 1, 9, 1);
        D->acts[skip[l]].skip = true;
        int b = conv(kCh[l], 0, kCh[l], l, a, -1, 0, 9, 1);
        low = b;
    }
    D->out_conv = conv(kCh[0], 0, 3, 0, low, -1, 0, 1, 0);
    // pooled activations: the input of encoder conv 'a' at levels 1..3
    for (int l = 1; l < 4; l++) {
        Act p{};
        p.c = kCh[l - 1];
        p.level = l;
        D->acts.push_back(p);
        const int pi = (int)D->acts.size() - 1;
        // encoder conv 'a' of level l is convs[2 l]; its input is the pool of level l - 1's output
        D->convs[2 * l].src_a = pi;
    }
}

// ---- forward ---------------------------------------------------------------------------------
// the input side of layer i's convolution at the current shape
ConvArgs layer_input(rf_denoiser* D, size_t i, const __nv_bfloat16* input) {
    const Conv& c = D->convs[i];
    ConvArgs a{};
    a.xa = c.src_a < 0 ? input : D->acts[c.src_a].x;
    a.xb = c.src_b < 0 ? nullptr : D->acts[c.src_b].x;
    a.ca = c.ca;
    a.cb = c.cb;
    a.up = c.up;
    a.n = D->N;
    a.h = D->H >> c.level;
    a.w = D->W >> c.level;
    a.taps = c.taps;
    a.error = D->error.get();
    return a;
}

// every layer; the head writes the image to `out`, or with a target the loss and its gradient
int forward(rf_denoiser* D, const __nv_bfloat16* input, float* out, const float* target) {
    for (size_t i = 0; i < D->convs.size(); i++) {
        Conv& c = D->convs[i];
        ConvArgs a = layer_input(D, i, input);
        a.B = c.w16;
        a.ldb = c.K();
        a.N = c.cout;
        a.bias = c.b;
        ConvEpilogue epi = kConvStoreBF16;
        if ((int)i == D->out_conv) {
            epi = target ? kConvL1 : kConvHead;
            a.feats = input;
            a.target = target;
            a.out = out;
            a.dz = D->acts[i].dz;
            a.loss = D->loss;
        } else {
            a.C = D->acts[i].x;
            a.ldc = c.cout;
            a.relu = c.relu;
            // an encoder layer whose output is pooled for the level below
            const int pooled = i < 6 && i % 2 == 1 ? D->convs[i + 1].src_a : -1;
            if (pooled >= 0) a.pool = D->acts[pooled].x;
        }
        const cudaError_t e = launch_conv(a, epi, D->stream);
        if (e != cudaSuccess) return cuda_fail(e, "convolution");
    }
    return RF_OK;
}

// ---- backward + Adam -------------------------------------------------------------------------
int update(rf_denoiser* D, float lr, uint32_t step) {
    const cudaError_t e = launch_adam(D->w, D->g, D->m, D->v, D->adam, (uint32_t)D->convs.size(), lr, 0.9f, 0.999f, 1e-8f,
                                      step, D->stream);
    if (e != cudaSuccess) return cuda_fail(e, "adam");
    return RF_OK;
}

int train(rf_denoiser* D, const __nv_bfloat16* input, const float* target, float lr) {
    cudaError_t e = cudaMemsetAsync(D->g, 0, rf_denoiser_num_params(D) * sizeof(float), D->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(D->loss, 0, sizeof(double), D->stream);
    if (e != cudaSuccess) return cuda_fail(e, "gradient clear");
    if (int rc = forward(D, input, nullptr, target)) return rc;
    std::vector<WgradTask> tasks;
    for (int i = (int)D->convs.size() - 1; i >= 0; i--) {
        Conv& c = D->convs[i];
        const uint32_t ldz = i == D->out_conv ? 8 : c.cout;  // the head's gradient is padded to 8 channels
        tasks.push_back(WgradTask{layer_input(D, (size_t)i, input), c.cout, ldz, c.gw});
        tasks.back().conv.dz = D->acts[i].dz;
        if (c.src_a < 0) continue;  // first layer: no input gradient
        // input gradient: dX = conv(dz, flipped transposed weights)
        ConvArgs gx{};
        gx.xa = D->acts[i].dz;
        gx.ca = ldz;
        gx.n = D->N;
        gx.h = D->H >> c.level;
        gx.w = D->W >> c.level;
        gx.taps = c.taps;
        gx.B = c.wf16;
        gx.ldb = c.ldf();
        gx.N = c.ca + c.cb;
        gx.error = D->error.get();
        ConvEpilogue epi = kConvMask;
        int into = c.src_a;  // the layer whose output gradient this completes
        if (c.cb > 0) {
            epi = kConvConcat;
            gx.nlow = c.ca;
            gx.dskip = D->acts[c.src_b].dskip;
        } else if (c.src_a >= (int)D->convs.size()) {
            epi = kConvPool;
            into = 2 * (c.level - 1) + 1;  // the last encoder layer of the level above
            gx.dskip = D->acts[into].dskip;
        }
        gx.y = D->acts[into].x;
        gx.dz = D->acts[into].dz;
        gx.gb = D->convs[into].gb;
        e = launch_conv(gx, epi, D->stream);
        if (e != cudaSuccess) return cuda_fail(e, "input gradient");
    }
    const Conv& head = D->convs[D->out_conv];
    e = launch_conv_wgrad(tasks.data(), (uint32_t)tasks.size(), D->acts[D->out_conv].dz, level_pixels(D->N, D->H, D->W, 0),
                          head.gb, D->error.get(), D->stream);
    if (e != cudaSuccess) return cuda_fail(e, "weight gradients");
    return update(D, lr, ++D->step);
}

int refresh_bf16(rf_denoiser* D) { return update(D, 0.0f, 1); }

int check_shape(rf_denoiser* D, uint32_t n, uint32_t h, uint32_t w) {
    if (n == 0 || h == 0 || w == 0 || h % 8 || w % 8)
        return fail(RF_ERR_INVALID_ARG, "denoiser: batch >= 1 and height, width multiples of 8 required");
    if ((uint64_t)n * h * w > D->P0) return fail(RF_ERR_CAPACITY, "denoiser: batch x height x width over the created capacity");
    D->N = n;
    D->H = h;
    D->W = w;
    return RF_OK;
}

}  // namespace

extern "C" {

int rf_denoiser_create(const rf_denoiser_desc* desc, rf_denoiser** out) {
    if (!desc || !out || desc->max_pixels == 0) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_create: bad arguments");
    *out = nullptr;
    auto* D = new rf_denoiser();
    D->d = *desc;
    D->device = desc->device;
    D->P0 = desc->max_pixels;
    auto bail = [&](int rc) { rf_denoiser_destroy(D); return rc; };
    if (cudaSetDevice(D->device) != cudaSuccess) return bail(fail(RF_ERR_NO_DEVICE, "rf_denoiser_create: no such device"));
    cudaError_t e = cudaStreamCreateWithFlags(&D->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return bail(cuda_fail(e, "stream"));
    if (!D->error.acquire()) return bail(cuda_fail(cudaErrorMemoryAllocation, "rf_denoiser_create: error word"));
    build_graph(D);
    // parameters, He-normal initialisation from a seeded generator
    const size_t np = rf_denoiser_num_params(D);
    std::vector<float> hp;
    hp.reserve(np);
    std::mt19937_64 gen(desc->seed);
    for (auto& c : D->convs) {
        const size_t nw = (size_t)c.cout * c.K();
        std::vector<float> hw(nw);
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)c.K()));
        for (size_t k = 0; k < nw; k++) hw[k] = nd(gen);
        if (c.taps == 9 && c.src_a < 0)  // network input: zero the padding channel's weights
            for (uint32_t co = 0; co < c.cout; co++)
                for (uint32_t t = 0; t < 9; t++) hw[(size_t)co * c.K() + t * kIn + kIn - 1] = 0.0f;
        if (c.taps == 1)  // the output layer starts at zero: the first prediction is the plain image
            std::fill(hw.begin(), hw.end(), 0.0f);
        c.offset = hp.size();
        hp.insert(hp.end(), hw.begin(), hw.end());
        hp.insert(hp.end(), c.cout, 0.0f);  // biases
        if (e == cudaSuccess) e = dalloc(D, &c.w16, nw);
        if (e == cudaSuccess) e = dalloc(D, &c.wf16, (size_t)(c.ca + c.cb) * c.ldf(), true);  // padding columns stay zero
    }
    if (e == cudaSuccess) e = dalloc(D, &D->w, np);
    if (e == cudaSuccess) e = dalloc(D, &D->g, np, true);
    if (e == cudaSuccess) e = dalloc(D, &D->m, np, true);
    if (e == cudaSuccess) e = dalloc(D, &D->v, np, true);
    // (the copy runs behind the clears on the default stream and returns when it is done)
    if (e == cudaSuccess) e = cudaMemcpy(D->w, hp.data(), np * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return bail(cuda_fail(e, "rf_denoiser_create: parameters"));
    for (size_t i = 0; i < D->convs.size(); i++) {
        Conv& c = D->convs[i];
        const size_t nw = (size_t)c.cout * c.K();
        c.b = D->w + c.offset + nw;
        c.gw = D->g + c.offset;
        c.gb = c.gw + nw;
        D->adam.layer[i] = AdamLayer{(uint32_t)c.offset, c.cout, c.K(), c.taps, c.ldf(), c.w16, c.wf16};
    }
    // activations and their gradients at the maximum size
    for (size_t i = 0; i < D->acts.size(); i++) {
        Act& a = D->acts[i];
        const uint64_t P = D->P0 >> (2 * a.level);
        const bool head = (int)i == D->out_conv;
        if (e == cudaSuccess && !head) e = dalloc(D, &a.x, P * a.c);
        if (e == cudaSuccess && i < D->convs.size()) e = dalloc(D, &a.dz, P * (head ? 8 : a.c));
        if (e == cudaSuccess && a.skip) e = dalloc(D, &a.dskip, P * a.c);
    }
    if (e == cudaSuccess) e = dalloc(D, &D->loss, 1);
    if (e != cudaSuccess) return bail(cuda_fail(e, "rf_denoiser_create: activations"));
    if (int rc = refresh_bf16(D)) return bail(rc);
    e = cudaStreamSynchronize(D->stream);
    if (e != cudaSuccess) return bail(cuda_fail(e, "rf_denoiser_create"));
    *out = D;
    return RF_OK;
}

int rf_denoiser_destroy(rf_denoiser* D) {
    if (!D) return RF_OK;
    cudaSetDevice(D->device);
    if (D->stream) cudaStreamSynchronize(D->stream);
    for (void* p : D->allocs) cudaFree(p);
    scratch_trim();
    if (D->stream) cudaStreamDestroy(D->stream);
    delete D;
    return RF_OK;
}

int rf_denoiser_set_stream(rf_denoiser* D, void* stream) {
    if (!D) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_set_stream: null");
    D->stream = static_cast<cudaStream_t>(stream);  // the caller's stream from here on
    return RF_OK;
}

int rf_denoiser_sync(rf_denoiser* D) {
    if (!D) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_sync: null");
    cudaSetDevice(D->device);
    return sync(D, "rf_denoiser_sync");
}

int rf_denoiser_num_layers(const rf_denoiser* D) { return D ? (int)D->convs.size() : -1; }

int rf_denoiser_layer(const rf_denoiser* D, int i, rf_denoiser_layer_info* out) {
    if (!D || !out || i < 0 || i >= (int)D->convs.size()) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_layer: bad index");
    const Conv& c = D->convs[i];
    out->in_a = c.ca;
    out->in_b = c.cb;
    out->out = c.cout;
    out->taps = c.taps;
    out->upsample = c.up;
    out->relu = c.relu;
    out->level = c.level;
    auto src = [&](int s) {
        if (s < 0) return -1;
        if (s < (int)D->convs.size()) return s;
        return -100 - (D->acts[s].level);  // pooled output of the level above's last conv
    };
    out->src_a = src(c.src_a);
    out->src_b = src(c.src_b);
    return RF_OK;
}

size_t rf_denoiser_num_params(const rf_denoiser* D) {
    if (!D) return 0;
    size_t n = 0;
    for (auto& c : D->convs) n += (size_t)c.cout * c.K() + c.cout;
    return n;
}

int rf_denoiser_get_params(rf_denoiser* D, float* host, size_t cap) {
    if (!D || !host || cap < rf_denoiser_num_params(D)) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_get_params: bad arguments");
    cudaSetDevice(D->device);
    if (int rc = sync(D, "rf_denoiser_get_params")) return rc;
    const cudaError_t e = cudaMemcpy(host, D->w, rf_denoiser_num_params(D) * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "rf_denoiser_get_params");
    return RF_OK;
}

int rf_denoiser_set_params(rf_denoiser* D, const float* host, size_t count) {
    if (!D || !host || count != rf_denoiser_num_params(D)) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_set_params: bad arguments");
    cudaSetDevice(D->device);
    if (int rc = sync(D, "rf_denoiser_set_params")) return rc;
    const cudaError_t e = cudaMemcpy(D->w, host, count * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "rf_denoiser_set_params");
    return refresh_bf16(D);
}

int rf_denoiser_features(const float* bins_rgba, uint32_t width, uint32_t height, float k2, const float* base_rgba,
                         float level, void* out_bf16, void* stream) {
    if (!bins_rgba || !out_bf16 || !width || !height) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_features: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* stats = nullptr;
    cudaError_t e = cudaSuccess;
    if (!(k2 > 0.0f)) {
        e = scratch_alloc(&stats, 3, st);
        if (e == cudaSuccess) e = launch_stats(reinterpret_cast<const float4*>(bins_rgba), width, height, stats, st);
    }
    if (e == cudaSuccess)
        e = launch_features(reinterpret_cast<const float4*>(bins_rgba), (uint64_t)width * height, k2, stats,
                            reinterpret_cast<const float4*>(base_rgba), level, static_cast<__nv_bfloat16*>(out_bf16), st);
    if (stats) cudaFreeAsync(stats, st);
    if (e != cudaSuccess) return cuda_fail(e, "rf_denoiser_features");
    return RF_OK;
}

int rf_denoiser_infer(rf_denoiser* D, const void* feats, uint32_t n, uint32_t h, uint32_t w, float* out_rgb) {
    if (!D || !feats || !out_rgb) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_infer: null argument");
    if (int rc = check_shape(D, n, h, w)) return rc;
    cudaSetDevice(D->device);
    if (int rc = forward(D, static_cast<const __nv_bfloat16*>(feats), out_rgb, nullptr)) return rc;
    return RF_OK;
}

int rf_denoiser_train_step(rf_denoiser* D, const void* feats, const float* target_rgb, uint32_t n, uint32_t h,
                           uint32_t w, float lr, double* loss) {
    if (!D || !feats || !target_rgb) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_train_step: null argument");
    if (int rc = check_shape(D, n, h, w)) return rc;
    cudaSetDevice(D->device);
    if (int rc = train(D, static_cast<const __nv_bfloat16*>(feats), target_rgb, lr)) return rc;
    if (loss) {
        double l = 0;
        cudaError_t e = cudaMemcpyAsync(&l, D->loss, sizeof(double), cudaMemcpyDeviceToHost, D->stream);
        if (e != cudaSuccess) return cuda_fail(e, "rf_denoiser_train_step");
        if (int rc = sync(D, "rf_denoiser_train_step")) return rc;
        *loss = l / (3.0 * (double)n * h * w);
    }
    return RF_OK;
}

int rf_denoiser_gradients(rf_denoiser* D, float* host, size_t cap) {
    if (!D || !host || cap < rf_denoiser_num_params(D)) return fail(RF_ERR_INVALID_ARG, "rf_denoiser_gradients: bad arguments");
    cudaSetDevice(D->device);
    if (int rc = sync(D, "rf_denoiser_gradients")) return rc;
    const cudaError_t e = cudaMemcpy(host, D->g, rf_denoiser_num_params(D) * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "rf_denoiser_gradients");
    return RF_OK;
}

}  // extern "C"
