// Host path of the tensor-core kernels' bounded waits, without a GPU: the entry points of the GEMM, the convolution
// and the learned estimator over a fake CUDA runtime and fake launches, of which the test makes one "run out" by
// writing the word it was given, as the kernels do.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>

#include "../../refrakt_gb300/csrc/denoise.cpp"
#include "../../refrakt_gb300/csrc/error_word.cpp"
#include "../../refrakt_gb300/csrc/gemm_api.cpp"

static std::string g_message;
static std::function<void()> g_at_sync;  // runs once, inside the next stream synchronisation
static int g_conv_code = 0, g_wgrad_code = 0, g_gemm_code = 0, g_streams = 0;

// ---- fake runtime ----
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = aligned_alloc(64, (n + 63) / 64 * 64); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "a CUDA error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(intptr_t)++g_streams; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (auto f = std::move(g_at_sync)) { g_at_sync = nullptr; f(); }
    return cudaSuccess;
}
}

// ---- fake launches ----
namespace rfk {
int fail(int status, const std::string& m) { g_message = m; return status; }
static void write(int* word, int& code) {
    if (code && word) *(volatile int*)word = code;
    code = 0;
}
bool conv_supported(uint32_t c, uint32_t, uint32_t) { return c % 16 == 0; }
cudaError_t launch_conv(const ConvArgs& a, ConvEpilogue, cudaStream_t) { write(a.error, g_conv_code); return a.error ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t launch_conv_wgrad(const WgradTask*, uint32_t, const __nv_bfloat16*, uint64_t, float*, int* error, cudaStream_t) {
    write(error, g_wgrad_code);
    return error ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t launch_gemm(GemmArgs g, uint32_t, cudaStream_t) { write(g.error, g_gemm_code); return g.error ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t launch_gemm_conv(GemmArgs g, cudaStream_t) { return launch_gemm(g, 1, nullptr); }
cudaError_t launch_adam(float*, const float*, float*, float*, const AdamLayers&, uint32_t, float, float, float, float, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_stats(const float4*, uint32_t, uint32_t, double*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_features(const float4*, uint64_t, float, const double*, const float4*, float, __nv_bfloat16*, cudaStream_t) { return cudaSuccess; }
cudaError_t scratch_alloc(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t scratch_trim() { return cudaSuccess; }
}  // namespace rfk

#define CHECK(x) do { if (!(x)) { printf("line %d: %s (%s)\n", __LINE__, #x, g_message.c_str()); return 1; } } while (0)

alignas(16) static unsigned char g_buf[1 << 16];
static int gemm() { return rf_gemm_bf16(g_buf, g_buf, g_buf, 8, 8, 8, 8, 8, 8, RF_GEMM_STORE_F32, nullptr, 0, 1, nullptr); }
static int conv(uint32_t c) { return rf_conv3x3_bf16(g_buf, c, 0, nullptr, 0, 1, 8, 8, g_buf, 8, 9 * c, g_buf, 8, RF_GEMM_STORE_F32, nullptr, 0, nullptr); }

int main() {
    const rf_denoiser_desc desc{4096, 1, 0};
    rf_denoiser *a = nullptr, *b = nullptr;
    CHECK(rf_denoiser_create(&desc, &a) == RF_OK && rf_denoiser_create(&desc, &b) == RF_OK);
    std::string host(rf_denoiser_num_params(a) * sizeof(float), '\0');
    float* params = reinterpret_cast<float*>(&host[0]);
    const size_t n = rf_denoiser_num_params(a);
    double loss = 0;
    auto train = [&](rf_denoiser* d, double* l) { return rf_denoiser_train_step(d, g_buf, (const float*)g_buf, 1, 64, 64, 1e-3f, l); };
    CHECK(train(a, &loss) == RF_OK && gemm() == RF_OK && conv(16) == RF_OK && conv(24) == RF_OK);

    // a step whose convolution or weight gradient gives up says so, once
    g_conv_code = 3;
    CHECK(train(a, &loss) == RF_ERR_TIMEOUT && g_message.find("a loaded stage") != std::string::npos);
    CHECK(train(a, &loss) == RF_OK);
    g_wgrad_code = 4;
    CHECK(train(a, &loss) == RF_ERR_TIMEOUT && train(a, &loss) == RF_OK);
    // without a loss nothing is waited for: the next call that does reports it, whichever it is
    using Call = std::function<int()>;
    const Call calls[] = {[&] { return rf_denoiser_sync(a); }, [&] { return rf_denoiser_get_params(a, params, n); },
                          [&] { return rf_denoiser_gradients(a, params, n); }, [&] { return rf_denoiser_set_params(a, params, n); }};
    for (const Call& call : calls) {
        g_wgrad_code = 1;
        CHECK(train(a, nullptr) == RF_OK && call() == RF_ERR_TIMEOUT && call() == RF_OK);
    }
    // another denoiser's and the GEMM's calls do not take it
    g_conv_code = 2;
    CHECK(rf_denoiser_infer(a, g_buf, 1, 8, 8, (float*)g_buf) == RF_OK);
    CHECK(train(b, &loss) == RF_OK && rf_denoiser_sync(b) == RF_OK && gemm() == RF_OK && conv(16) == RF_OK);
    CHECK(rf_denoiser_sync(a) == RF_ERR_TIMEOUT && rf_denoiser_sync(a) == RF_OK);

    // the single calls, and which wait it was
    g_gemm_code = 7;
    CHECK(gemm() == RF_ERR_CUDA && g_message.find("code 7") != std::string::npos && gemm() == RF_OK);
    g_gemm_code = 2;
    CHECK(conv(24) == RF_ERR_CUDA && g_message.find("code 2") != std::string::npos && conv(24) == RF_OK);
    g_conv_code = 2;
    CHECK(conv(16) == RF_ERR_CUDA && g_message.find("accumulator's release") != std::string::npos && conv(16) == RF_OK);
    // a call that another one overlaps keeps its own failure
    int inner = -1;
    g_gemm_code = 5;
    g_at_sync = [&] { inner = gemm(); };
    CHECK(gemm() == RF_ERR_CUDA && inner == RF_OK);
    rf_denoiser_destroy(a);
    rf_denoiser_destroy(b);
    // words come back: as many calls as there are words in several pages
    for (int k = 0; k < 1000; k++) CHECK(gemm() == RF_OK);
    printf("OK\n");
    return 0;
}
