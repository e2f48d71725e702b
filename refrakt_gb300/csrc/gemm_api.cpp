// C-ABI entries of the tensor-core GEMM and implicit 3x3 convolution (no reference counterpart):
// let a caller, and the tests, run the contractions of the learned density estimator on their own.
#include <cuda_runtime.h>

#include <string>

#include "conv.h"
#include "error_word.h"
#include "gemm.h"
#include "internal.h"
#include "refrakt.h"

using namespace rfk;

namespace {

// waits for the launch, then takes the call's error word; conv: the code is one of conv.cu's
int finish(const char* fn, cudaError_t e, cudaStream_t st, ErrorWord& word, bool conv) {
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(RF_ERR_CUDA, std::string(fn) + ": " + cudaGetErrorString(e));
    const int code = word.take();
    if (!code) return RF_OK;
    return fail(RF_ERR_CUDA, std::string(fn) + ": an mbarrier wait ran out (" +
                                 (conv ? "for " + std::string(conv_error(code)) : "code " + std::to_string(code)) + ")");
}
int no_word(const char* fn) { return fail(RF_ERR_CUDA, std::string(fn) + ": " + cudaGetErrorString(cudaErrorMemoryAllocation)); }

}  // namespace

extern "C" int rf_gemm_bf16(const void* A, const void* B, void* C, uint32_t M, uint32_t N, uint32_t K, uint32_t lda,
                            uint32_t ldb, uint32_t ldc, int mode, const float* bias, int relu, uint32_t splits,
                            void* stream) {
    if (!A || !B || !C || M == 0 || N == 0) return fail(RF_ERR_INVALID_ARG, "rf_gemm_bf16: null operand or empty shape");
    if (K % 8 || lda % 8 || ldb % 8 || lda < K || ldb < K || ldc < N)
        return fail(RF_ERR_INVALID_ARG, "rf_gemm_bf16: K and the operand strides must be multiples of 8, strides >= K");
    if ((((uintptr_t)A) | ((uintptr_t)B)) & 15) return fail(RF_ERR_INVALID_ARG, "rf_gemm_bf16: operands must be 16-byte aligned");
    if (mode < RF_GEMM_STORE_F32 || mode > RF_GEMM_ATOMIC_F32) return fail(RF_ERR_INVALID_ARG, "rf_gemm_bf16: bad mode");
    if (splits > 1 && mode != RF_GEMM_ATOMIC_F32) return fail(RF_ERR_INVALID_ARG, "rf_gemm_bf16: split K needs RF_GEMM_ATOMIC_F32");
    GemmArgs g{};
    g.A = static_cast<const __nv_bfloat16*>(A);
    g.B = static_cast<const __nv_bfloat16*>(B);
    g.M = M;
    g.N = N;
    g.K = K;
    g.lda = lda;
    g.ldb = ldb;
    g.C = C;
    g.ldc = ldc;
    g.mode = mode;
    g.bias = bias;
    g.relu = relu;
    ErrorWord word;
    if (!word.acquire()) return no_word("rf_gemm_bf16");
    g.error = word.get();
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return finish("rf_gemm_bf16", launch_gemm(g, splits, st), st, word, false);
}

extern "C" int rf_conv3x3_bf16(const void* xa, uint32_t ca, int up, const void* xb, uint32_t cb, uint32_t n,
                               uint32_t h, uint32_t w, const void* B, uint32_t N, uint32_t ldb, void* C, uint32_t ldc,
                               int mode, const float* bias, int relu, void* stream) {
    if (!xa || !B || !C || (cb && !xb) || n == 0 || h == 0 || w == 0 || N == 0)
        return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: null operand or empty shape");
    if (ca % 8 || cb % 8 || ca + cb == 0 || ldb % 8 || ldb < 9 * (ca + cb) || ldc < N)
        return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: channels and ldb must be multiples of 8, ldb >= 9 (ca + cb)");
    if (h > 65535 || w > 65535 || (uint64_t)n * h * w > 0xFFFFFFFFull)
        return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: image too large");
    if (up && (h % 2 || w % 2)) return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: an upsampled input needs even h, w");
    if ((((uintptr_t)xa) | ((uintptr_t)xb) | ((uintptr_t)B)) & 15)
        return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: operands must be 16-byte aligned");
    if (mode < RF_GEMM_STORE_F32 || mode > RF_GEMM_ATOMIC_F32) return fail(RF_ERR_INVALID_ARG, "rf_conv3x3_bf16: bad mode");
    ErrorWord word;
    if (!word.acquire()) return no_word("rf_conv3x3_bf16");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // channels in whole K steps and a tile's operands within shared memory: the staged-tile kernel
    // (conv.cu); other channel counts gather im2col rows (gemm.cu)
    if (conv_supported(ca + cb, N, 9)) {
        ConvArgs a{};
        a.xa = static_cast<const __nv_bfloat16*>(xa);
        a.xb = static_cast<const __nv_bfloat16*>(xb);
        a.ca = ca;
        a.cb = cb;
        a.up = up;
        a.n = n;
        a.h = h;
        a.w = w;
        a.taps = 9;
        a.B = static_cast<const __nv_bfloat16*>(B);
        a.N = N;
        a.ldb = ldb;
        a.C = C;
        a.ldc = ldc;
        a.bias = bias;
        a.relu = relu;
        a.error = word.get();
        const ConvEpilogue epi = mode == RF_GEMM_STORE_F32 ? kConvStoreF32 : mode == RF_GEMM_ATOMIC_F32 ? kConvAtomicF32 : kConvStoreBF16;
        return finish("rf_conv3x3_bf16", launch_conv(a, epi, st), st, word, true);
    }
    GemmArgs g{};
    g.xa = static_cast<const __nv_bfloat16*>(xa);
    g.xb = static_cast<const __nv_bfloat16*>(xb);
    g.ca = ca;
    g.cb = cb;
    g.n = n;
    g.h = h;
    g.w = w;
    g.up = up;
    g.B = static_cast<const __nv_bfloat16*>(B);
    g.M = n * h * w;
    g.N = N;
    g.K = 9 * (ca + cb);
    g.ldb = ldb;
    g.C = C;
    g.ldc = ldc;
    g.mode = mode;
    g.bias = bias;
    g.relu = relu;
    g.error = word.get();
    return finish("rf_conv3x3_bf16", launch_gemm_conv(g, st), st, word, false);
}
