// 3x3 and 1x1 convolutions of the learned density estimator on the 5th-generation tensor cores.
//
// Layout.  A CTA takes tiles of 8 x 16 output pixels (the MMA's M = 128 rows, one 8-pixel row group
// per tile row).  The tile's input, with a one-pixel halo for a 3x3 kernel (10 x 18 pixels), is
// staged once in shared memory, pixel-fastest: plane q holds channels 8q .. 8q + 7 of every staged
// pixel, 16 bytes each.  In that layout any 8 consecutive pixels of a plane are one K-major core
// matrix of the no-swizzle layout (umma.cuh), so each tap's A operand is the same staged tile with
// the descriptor's start moved by (dy * pitch + dx) * 16 bytes, row groups a staged row apart
// (SBO = pitch * 16) and K chunks a plane apart (LBO = plane): the input crosses L2 -> shared memory
// 1.4 times instead of 9 (an im2col gather), and no tap is decoded per element.
// For the weight gradient the same planes are the MN-major core matrices of x^T (8 pixels of K by
// 8 channels of M), again shifted per tap, and the output gradient's planes those of the other
// operand: no transposed copy of either is ever made.
//
// Roles (576 threads, persistent over the tiles): warps 0-7 load (cp.async, a ring of tile stages);
// warps 8 and 9 each have one lane issue the MMAs of every other tile into an accumulator of its own,
// so that one's waits and commits (about 1,000 cycles a tile) pass under the other's MMAs; warps 10-13
// and 14-17 each drain one of the accumulators.  The weights of the
// CTA's columns stay in shared memory for all of its tiles; a layer whose weights do not fit beside
// two stages is cut into column groups (grid.y).
//
// The K order (taps outermost, 16 channels per MMA) is that of the im2col GEMM (gemm.cu, conv mode).
//
// Bound: the copies' shared-memory writes, a wavefront per 16 bytes (72 copies of 41 wavefronts per tile
// of 80 channels, of its 2,930 cycles; the 45 MMAs' operand reads, 40 wavefronts each, take 1,800).
// Measured, bf16, one call: 48 upsampled + 32 channels to 32 at 1920 x 1080 885 us as a gathered im2col
// GEMM, 192 us here; 32 to 32 at 16 x 256 x 256 (the kernel) 238 -> 59 us.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "conv.h"
#include "gemm.h"
#include "umma.cuh"

namespace rfk {

namespace {

constexpr uint32_t kTileX = 8, kTileY = 16;  // output pixels per tile: 8 rows of a core matrix by 16 groups
constexpr int kThreads = 576;
constexpr int kLoaders = 256;
constexpr int kLoadWarps = kLoaders / 32, kMmaWarp = kLoadWarps, kDrainWarp = kMmaWarp + 2;
constexpr int kMaxStages = 4;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr size_t kMaxSmem = 227 * 1024;

struct Geom {
    uint32_t tiles_x, tiles_y, tiles;
    uint32_t chunks;   // 8-channel planes of the input
    uint32_t hx, hy;   // staged pixels per tile
    uint32_t plane;    // bytes of a plane
    uint32_t stage;    // bytes of a stage
    uint32_t stages;
    uint32_t np;       // columns of a CTA, rounded to 16
    uint32_t kchunks;  // 8-wide K chunks of the weights, rounded to 2
    uint32_t wbytes;   // bytes of the weights (conv) before the stages
    uint32_t zero;     // offset of the zero plane (odd chunk count), else 0
    uint32_t bars;     // offset of the mbarriers
    uint32_t cols;     // tensor-memory columns of one accumulator
};

// The tiles of one CTA, blockIdx.x, blockIdx.x + gridDim.x, ..., without a division per tile
struct Tile {
    uint32_t img, ty, tx;
    uint32_t simg, sty, stx;  // the step
    int y0, x0;
    __device__ __forceinline__ Tile(const Geom& G, uint32_t first, uint32_t step) {
        const uint32_t per = G.tiles_x * G.tiles_y;
        img = first / per;
        ty = (first - img * per) / G.tiles_x;
        tx = first - img * per - ty * G.tiles_x;
        simg = step / per;
        sty = (step - simg * per) / G.tiles_x;
        stx = step - simg * per - sty * G.tiles_x;
        place();
    }
    __device__ __forceinline__ void place() {
        y0 = (int)(ty * kTileY);
        x0 = (int)(tx * kTileX);
    }
    __device__ __forceinline__ void next(const Geom& G) {
        tx += stx;
        ty += sty;
        img += simg;
        if (tx >= G.tiles_x) { tx -= G.tiles_x; ty++; }
        if (ty >= G.tiles_y) { ty -= G.tiles_y; img++; }
        place();
    }
};

// A loading thread's share of every tile: in each of its pixel octets (warp, warp + 8, warp + 16) one
// pixel and every fourth plane, so a quarter warp writes 128 contiguous bytes of shared memory and
// reads 64 contiguous bytes of 8 pixels; a one-plane input takes a pixel per lane.  The pixels'
// offsets from the tile's origin are the same for every tile.
// (The copies cost a shared-memory wavefront per 16 bytes.  Loads into registers and 16-byte stores
// cost a third of that but were latency bound: 138 us against 95 for 80 channels at 16 x 256 x 256.)
template <bool HALO>
struct PixelLoader {
    static constexpr uint32_t HX = kTileX + (HALO ? 2u : 0u), HY = kTileY + (HALO ? 2u : 0u), PX = HX * HY;
    static constexpr uint32_t PLANE = PX * 16u;
    static constexpr int kItems = (int)((PX + 8 * kLoadWarps - 1) / (8 * kLoadWarps));
    const __nv_bfloat16 *xa, *xb;
    uint32_t ca, cb, na, nb;  // channels, planes of each input
    uint32_t h, w, up, q0;
    int32_t ra[kItems], rb[kItems], dy[kItems], dx[kItems];
    uint32_t dst[kItems];  // ~0u: no pixel

    __device__ __forceinline__ PixelLoader(const ConvArgs& A, int tid)
        : xa(A.xa), xb(A.xb), ca(A.ca), cb(A.cb), na(A.ca >> 3), nb(A.cb >> 3), h(A.h), w(A.w), up(A.up ? 1u : 0u) {
        const uint32_t lane = tid & 31u, warp = tid >> 5;
        const bool one = na + nb == 1;
        q0 = one ? 0u : lane >> 3;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const uint32_t g = warp + kLoadWarps * k, p = one ? g * 32u + lane : g * 8u + (lane & 7u);
            const uint32_t py = p / HX, px = p - py * HX;
            dy[k] = (int)py - (HALO ? 1 : 0);
            dx[k] = (int)px - (HALO ? 1 : 0);
            ra[k] = ((dy[k] >> up) * (int)(w >> up) + (dx[k] >> up)) * (int)ca + 8 * (int)q0;
            rb[k] = (dy[k] * (int)w + dx[k]) * (int)cb + 8 * (int)q0;
            dst[k] = p < PX ? q0 * PLANE + p * 16u : ~0u;
        }
    }
    __device__ __forceinline__ void planes(uint32_t d, const __nv_bfloat16* src, uint32_t n, uint32_t bytes) const {
#pragma unroll 4
        for (uint32_t q = q0; q < n; q += 4, d += 4 * PLANE, src += bytes ? 32 : 0) umma::cp_async16(d, src, bytes);
    }
    __device__ __forceinline__ void operator()(const Tile& t, uint32_t stage) const {
        const __nv_bfloat16* ta = xa + (((size_t)t.img * (h >> up) + ((uint32_t)t.y0 >> up)) * (w >> up) + ((uint32_t)t.x0 >> up)) * ca;
        const __nv_bfloat16* tb = xb + (((size_t)t.img * h + (uint32_t)t.y0) * w + (uint32_t)t.x0) * cb;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            if (dst[k] == ~0u) continue;
            const bool ok = (uint32_t)(t.y0 + dy[k]) < h && (uint32_t)(t.x0 + dx[k]) < w;
            const uint32_t bytes = ok ? 16u : 0u, d = stage + dst[k];
            planes(d, ok ? ta + ra[k] : xa, na, bytes);
            if (nb) planes(d + na * PLANE, ok ? tb + rb[k] : xb, nb, bytes);
        }
    }
};

__device__ __forceinline__ void cp_wait_pending(uint32_t left) {
    switch (left) {
    case 0: umma::cp_async_wait<0>(); break;
    case 1: umma::cp_async_wait<1>(); break;
    default: umma::cp_async_wait<2>(); break;
    }
}

// barriers: full[stages], empty[stages], acc_full[2], acc_empty[2]
struct Bars {
    uint64_t *full, *empty, *acc_full, *acc_empty;
    uint32_t* tmem;
    int* fail;
    int* error;  // the host's error word
};
// b.error gets 1 a stage to load, 2 an accumulator's release, 3 a loaded stage, 4 an accumulator (conv_error)
__device__ __forceinline__ void conv_fail(const Bars& b, int code) {
    *reinterpret_cast<volatile int*>(b.fail) = 1;
    umma::report_error(b.error, code);
}
__device__ __forceinline__ bool conv_failed(const int* s_fail) { return *reinterpret_cast<const volatile int*>(s_fail) != 0; }

__device__ __forceinline__ Bars bars_at(unsigned char* p, int* error) {
    Bars b;
    b.full = reinterpret_cast<uint64_t*>(p);
    b.empty = b.full + kMaxStages;
    b.acc_full = b.empty + kMaxStages;
    b.acc_empty = b.acc_full + 2;
    b.tmem = reinterpret_cast<uint32_t*>(b.acc_empty + 2);
    b.fail = reinterpret_cast<int*>(b.tmem + 1);
    b.error = error;
    return b;
}
constexpr uint32_t kBarBytes = (2 * kMaxStages + 4) * 8 + 16;

// `loaders`: threads that fill a stage; `issuers`: threads whose MMAs read it
__device__ __forceinline__ void bars_init(const Bars& b, uint32_t loaders, uint32_t issuers) {
    for (int s = 0; s < kMaxStages; s++) {
        umma::mbar_init(&b.full[s], loaders);
        umma::mbar_init(&b.empty[s], issuers);
    }
    for (int k = 0; k < 2; k++) {
        umma::mbar_init(&b.acc_full[k], issuers);
        umma::mbar_init(&b.acc_empty[k], 4);  // one arrival per draining warp
    }
    *b.fail = 0;
    umma::fence_mbar_init();
}

// The loading threads' loop over this CTA's `count` tiles: `issue(stage)` starts the next tile's copies.
// A thread announces a tile (full) once its own copies of it have landed, S - 1 tiles behind the one
// it issues, and before it waits for that one's stage, so the issuing lanes always have the next tile.
template <class Issue>
__device__ __forceinline__ void load_loop(const Bars& b, uint32_t count, uint32_t S, Issue issue) {
    uint32_t st = 0, use = 0, told = 0, announced = 0;  // stage of tile i and its use, stage of the next tile to announce
    for (uint32_t i = 0; i < count; i++) {
        if (i + 1 >= S) {
            cp_wait_pending(S - 2);
            umma::fence_proxy_async_smem();
            umma::mbar_arrive(&b.full[told]);
            if (++told == S) told = 0;
            announced++;
        }
        if (use > 0 && !umma::mbar_wait(&b.empty[st], (use - 1) & 1u, kWaitLimit)) {
            conv_fail(b, 1);
            break;
        }
        if (conv_failed(b.fail)) break;
        issue(st);
        umma::cp_async_commit();
        if (++st == S) { st = 0; use++; }
    }
    umma::cp_async_wait<0>();
    umma::fence_proxy_async_smem();
    if (!conv_failed(b.fail))
        for (; announced < count; announced++) {
            umma::mbar_arrive(&b.full[told]);
            if (++told == S) told = 0;
        }
}

// ---- epilogue -----------------------------------------------------------------------------------

__device__ __forceinline__ void st_v8(void* p, const uint32_t (&u)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(u[0]), "r"(u[1]), "r"(u[2]),
                 "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7])
                 : "memory");
}
__device__ __forceinline__ void ld_v8(const void* p, uint32_t (&u)[8]) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "l"(p));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

// sums of 16 columns over the warp's 32 lanes: lane l (even) returns the sum of column l / 2
// (recursive halving, 16 shuffles)
__device__ __forceinline__ float column_sums(const float (&v)[16], uint32_t lane) {
    float a[8], b[4], c[2];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const bool up = lane & 16u;
        const float keep = up ? v[8 + j] : v[j], give = up ? v[j] : v[8 + j];
        a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const bool up = lane & 8u;
        const float keep = up ? a[4 + j] : a[j], give = up ? a[j] : a[4 + j];
        b[j] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const bool up = lane & 4u;
        const float keep = up ? b[2 + j] : b[j], give = up ? b[j] : b[2 + j];
        c[j] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
    const bool up = lane & 2u;
    float s = (up ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, up ? c[0] : c[1], 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// 16 gradient values g of one pixel: dz = g where the activation y is positive, as bf16 at element
// offset o; g is masked in place.  (y has the layout of dz.)
__device__ __forceinline__ void mask_store(const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ dz, size_t o,
                                           float (&g)[16]) {
    uint32_t m[8], u[8];
    ld_v8(y + o, m);
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (!(bf_lo(m[j]) > 0.0f)) g[2 * j] = 0.0f;
        if (!(bf_hi(m[j]) > 0.0f)) g[2 * j + 1] = 0.0f;
        u[j] = pack_bf16(g[2 * j], g[2 * j + 1]);
    }
    st_v8(dz + o, u);
}

// state a reading thread keeps over its tiles (kConvL1)
struct HeadSums {
    double loss = 0.0;
};

// 16 columns n .. n + 15 of this thread's pixel (every lane of the warp calls it; ok = inside the
// image).  s_gb: the warp's column sums in shared memory, indexed from the CTA's first column.
template <int EPI>
__device__ __forceinline__ void finish16(const ConvArgs& A, float (&v)[16], uint32_t n, uint32_t col, bool ok,
                                         uint32_t img, int y, int x, uint32_t lane, float* s_gb, const float* s_bias,
                                         HeadSums& hs, bool wide) {
    const size_t p = ((size_t)img * A.h + (uint32_t)y) * A.w + (uint32_t)x;
    if constexpr (EPI == kConvStoreF32 || EPI == kConvAtomicF32) {
        if (!ok) return;
        float* c = static_cast<float*>(A.C) + p * A.ldc + n;
        if (EPI == kConvStoreF32 && wide && n + 16 <= A.N) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                uint32_t u[8];
#pragma unroll
                for (int j = 0; j < 8; j++) u[j] = __float_as_uint(v[8 * q + j]);
                st_v8(c + 8 * q, u);
            }
        } else {
            for (int j = 0; j < 16; j++) {
                if (n + j >= A.N) break;
                if (EPI == kConvAtomicF32) atomicAdd(c + j, v[j]);
                else c[j] = v[j];
            }
        }
    } else if constexpr (EPI == kConvStoreBF16) {
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const float s = v[j] + s_bias[col + j];
            v[j] = A.relu ? fmaxf(s, 0.0f) : s;
        }
        __nv_bfloat16* c = static_cast<__nv_bfloat16*>(A.C) + p * A.ldc + n;
        if (wide && n + 16 <= A.N) {
            uint32_t u[8];
#pragma unroll
            for (int j = 0; j < 8; j++) u[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
            if (ok) st_v8(c, u);
            if (A.pool) {  // the 2x2 average of the stored values, FP32, in the block's row order
                uint32_t r[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint32_t b = __shfl_down_sync(0xffffffffu, u[j], 1), d = __shfl_down_sync(0xffffffffu, u[j], 8),
                                   e = __shfl_down_sync(0xffffffffu, u[j], 9);
                    r[j] = pack_bf16(0.25f * (bf_lo(u[j]) + bf_lo(b) + bf_lo(d) + bf_lo(e)),
                                     0.25f * (bf_hi(u[j]) + bf_hi(b) + bf_hi(d) + bf_hi(e)));
                }
                if (ok && !((lane & 1u) | (lane & 8u)))
                    st_v8(A.pool + (((size_t)img * (A.h >> 1) + ((uint32_t)y >> 1)) * (A.w >> 1) + ((uint32_t)x >> 1)) * A.N + n,
                          r);
            }
        } else if (ok) {
            for (int j = 0; j < 16; j++)
                if (n + j < A.N) c[j] = __float2bfloat16_rn(v[j]);
        }
    } else if constexpr (EPI == kConvHead) {
        if (!ok) return;
        for (int ch = 0; ch < 3; ch++)
            A.out[p * 3 + ch] = fminf(fmaxf(__bfloat162float(A.feats[p * 8 + 4 + ch]) + v[ch] + A.bias[ch], 0.0f), 1.0f);
    } else if constexpr (EPI == kConvL1) {
        if (!ok) return;
        const float inv = 1.0f / (3.0f * (float)((uint64_t)A.n * A.h * A.w));
        __align__(16) __nv_bfloat16 g8[8];
#pragma unroll
        for (int q = 0; q < 8; q++) g8[q] = __float2bfloat16_rn(0.0f);
#pragma unroll
        for (int ch = 0; ch < 3; ch++) {
            const float d = __bfloat162float(A.feats[p * 8 + 4 + ch]) + v[ch] + A.bias[ch] - A.target[p * 3 + ch];
            hs.loss += fabs((double)d);
            g8[ch] = __float2bfloat16_rn(d > 0.0f ? inv : (d < 0.0f ? -inv : 0.0f));
        }
        *reinterpret_cast<uint4*>(A.dz + p * 8) = *reinterpret_cast<const uint4*>(g8);
    } else if constexpr (EPI == kConvMask) {
        if (ok) mask_store(A.y, A.dz, p * A.N + n, v);
        else
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = 0.0f;
        const float s = column_sums(v, lane);
        if (!(lane & 1u)) s_gb[col + (lane >> 1)] += s;
    } else if constexpr (EPI == kConvConcat) {
        if (n >= A.nlow) {
            if (!ok) return;
            float* c = A.dskip + p * (A.N - A.nlow) + (n - A.nlow);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                uint32_t u[8];
#pragma unroll
                for (int j = 0; j < 8; j++) u[j] = __float_as_uint(v[8 * q + j]);
                st_v8(c + 8 * q, u);
            }
            return;
        }
        const bool own = ok && !((lane & 1u) | (lane & 8u));
#pragma unroll
        for (int j = 0; j < 16; j++) {  // the adjoint of nearest-neighbour upsampling
            const float b = __shfl_down_sync(0xffffffffu, v[j], 1), d = __shfl_down_sync(0xffffffffu, v[j], 8),
                        e = __shfl_down_sync(0xffffffffu, v[j], 9);
            v[j] = own ? v[j] + b + d + e : 0.0f;
        }
        if (own)
            mask_store(A.y, A.dz,
                       (((size_t)img * (A.h >> 1) + ((uint32_t)y >> 1)) * (A.w >> 1) + ((uint32_t)x >> 1)) * A.nlow + n, v);
        const float s = column_sums(v, lane);
        if (!(lane & 1u)) s_gb[col + (lane >> 1)] += s;
    } else if constexpr (EPI == kConvPool) {
        float sum[16];
#pragma unroll
        for (int j = 0; j < 16; j++) sum[j] = 0.0f;
        if (ok) {
            for (int q = 0; q < 4; q++) {  // the four pixels that were averaged
                const size_t o = (((size_t)img * (2u * A.h) + 2u * (uint32_t)y + (q >> 1)) * (2u * A.w) + 2u * (uint32_t)x +
                                  (q & 1)) * A.N + n;
                uint32_t u[8];
                float g[16];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    ld_v8(A.dskip + o + 8 * k, u);
#pragma unroll
                    for (int j = 0; j < 8; j++) g[8 * k + j] = __uint_as_float(u[j]) + 0.25f * v[8 * k + j];
                }
                mask_store(A.y, A.dz, o, g);
#pragma unroll
                for (int j = 0; j < 16; j++) sum[j] += g[j];
            }
        }
        const float s = column_sums(sum, lane);
        if (!(lane & 1u)) s_gb[col + (lane >> 1)] += s;
    }
}

// The MMAs of one tile: taps outermost, then pairs of planes; only the descriptors' low words move.
// (A step is a few additions in uniform registers; computing each tap's descriptor afresh took 200
// cycles per tap, and unrolling over the taps spilled and missed the instruction cache.)
struct MmaSteps {
    uint32_t d, alo, ahi, blo, bhi, idesc;
    uint32_t da, db, pitch;  // descriptor steps of a plane pair (operands A, B) and of a staged row
};
__device__ __forceinline__ void mma_tile(const MmaSteps& m, uint32_t side, uint32_t pairs) {
    uint32_t row = m.alo, b = m.blo, acc = 0;
#pragma unroll 1
    for (uint32_t dy = 0; dy < side; dy++, row += m.pitch) {
#pragma unroll 1
        for (uint32_t dx = 0; dx < side; dx++) {
            uint32_t a = row + dx;
#pragma unroll 1
            for (uint32_t q = 0; q < pairs; q++, a += m.da, b += m.db) {
                umma::mma_bf16(m.d, a, m.ahi, b, m.bhi, m.idesc, acc);
                acc = 1;
            }
        }
    }
}

// ---- forward and input gradient -------------------------------------------------------------------

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1) conv_kernel(const __grid_constant__ ConvArgs A, const __grid_constant__ Geom G) {
    constexpr bool kSums = EPI == kConvMask || EPI == kConvConcat || EPI == kConvPool;
    extern __shared__ __align__(128) unsigned char smem[];
    const Bars B = bars_at(smem + G.bars, A.error);
    float* s_gb = reinterpret_cast<float*>(smem + G.bars + kBarBytes);  // 8 warps x np (kSums)
    const uint32_t base = umma::smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t lane = tid & 31u;
    const uint32_t n0 = blockIdx.y * G.np;
    const uint32_t nt = min(G.np, ((A.N - n0) + 15u) & ~15u);  // this CTA's columns, rounded to 16
    const uint32_t count = blockIdx.x < G.tiles ? (G.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;

    if (warp == kMmaWarp) umma::tmem_alloc(B.tmem, 2 * G.cols);
    if (tid == 0) bars_init(B, kLoaders, 1);
    if (kSums)
        for (uint32_t i = tid; i < 8 * G.np; i += kThreads) s_gb[i] = 0.0f;
    float* s_bias = s_gb + (kSums ? 8 * G.np : 0u);
    if (EPI == kConvStoreBF16)
        for (uint32_t i = tid; i < nt; i += kThreads) s_bias[i] = A.bias && n0 + i < A.N ? A.bias[n0 + i] : 0.0f;
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *B.tmem;

    if (warp < kLoadWarps) {
        // the weights, K chunk q's rows 16 bytes apart (rows past N and chunks past K zero), and the
        // zero plane: part of the first tile's copies
        const uint32_t kc = A.taps * G.chunks;
        for (uint32_t g = warp; g * 8 < nt; g += kLoadWarps) {
            const uint32_t r = g * 8 + (lane & 7u);
            const bool row = n0 + r < A.N;
            const __nv_bfloat16* src = A.B + (size_t)(row ? n0 + r : 0u) * A.ldb;
            for (uint32_t q = lane >> 3; q < G.kchunks; q += 4)
                umma::cp_async16(base + (q * nt + r) * 16u, q < kc ? src + 8 * q : A.B, row && q < kc ? 16u : 0u);
        }
        if (G.zero)
            for (uint32_t o = tid * 16u; o < G.plane; o += kLoaders * 16u) umma::cp_async16(base + G.zero + o, A.B, 0u);
        const uint32_t ring = base + G.wbytes;
        Tile t(G, blockIdx.x, gridDim.x);
        if (A.taps == 9) {
            const PixelLoader<true> load(A, tid);
            load_loop(B, count, G.stages, [&](uint32_t st) {
                load(t, ring + st * G.stage);
                t.next(G);
            });
        } else {
            const PixelLoader<false> load(A, tid);
            load_loop(B, count, G.stages, [&](uint32_t st) {
                load(t, ring + st * G.stage);
                t.next(G);
            });
        }
    } else if (warp < kDrainWarp) {
        if (umma::elect_one()) {
            const uint32_t buf = (uint32_t)(warp - kMmaWarp), idesc = umma::idesc_bf16_f32(128, nt);
            const uint32_t sbo = G.hx * 16u, wq = nt * 16u;
            uint32_t st = buf % G.stages, use = buf / G.stages;
            for (uint32_t i = buf; i < count; i += 2) {
                const uint32_t u = i >> 1;
                if (conv_failed(B.fail)) break;
                if (u > 0 && !umma::mbar_wait(&B.acc_empty[buf], (u - 1) & 1u, kWaitLimit)) {
                    conv_fail(B, 2);
                    break;
                }
                if (!umma::mbar_wait(&B.full[st], use & 1u, kWaitLimit)) {
                    conv_fail(B, 3);
                    break;
                }
                umma::fence_after_sync();
                const uint32_t a0 = base + G.wbytes + st * G.stage, d = tmem + buf * G.cols;
                if (G.zero) {  // one plane: a K step is two taps; the odd last chunk pairs with zeros
                    for (uint32_t q = 0; q < G.kchunks; q += 2) {
                        const uint32_t s0 = (q / 3) * G.hx + q % 3, s1 = ((q + 1) / 3) * G.hx + (q + 1) % 3;
                        const uint32_t a = a0 + s0 * 16u;
                        const uint32_t lbo = q + 1 < A.taps ? (s1 - s0) * 16u : base + G.zero - a;
                        umma::mma_bf16(d, umma::smem_desc(a, lbo, sbo), umma::smem_desc(base + q * wq, wq, 128u), idesc,
                                       q != 0u);
                    }
                } else {
                    const uint64_t da = umma::smem_desc(a0, G.plane, sbo), db = umma::smem_desc(base, wq, 128u);
                    const MmaSteps m{d, (uint32_t)da, (uint32_t)(da >> 32), (uint32_t)db, (uint32_t)(db >> 32), idesc,
                                     G.plane >> 3, wq >> 3, G.hx};
                    mma_tile(m, A.taps == 9 ? 3u : 1u, G.chunks >> 1);
                }
                umma::mma_commit(&B.empty[st]);
                umma::mma_commit(&B.acc_full[buf]);
                if ((st += 2) >= G.stages) { st -= G.stages; use++; }
            }
        }
    } else {
        const uint32_t q4 = (uint32_t)warp & 3u, m = 32u * q4 + lane;  // tensor-memory lane quarter, pixel of the tile
        const uint32_t ty = m >> 3, tx = m & 7u;
        const uint32_t buf = (uint32_t)(warp - kDrainWarp) >> 2;        // this group's accumulator
        float* gbw = s_gb + (warp - kDrainWarp) * G.np;
        HeadSums hs;
        bool wide = true;  // whole 32-byte pieces of the output
        if constexpr (EPI == kConvStoreF32)
            wide = ((reinterpret_cast<uintptr_t>(A.C) & 31u) == 0) && A.ldc % 8u == 0;
        if constexpr (EPI == kConvStoreBF16)
            wide = ((reinterpret_cast<uintptr_t>(A.C) & 31u) == 0) && A.ldc % 16u == 0;
        Tile t(G, blockIdx.x + buf * gridDim.x, 2 * gridDim.x);
        for (uint32_t i = buf; i < count; i += 2, t.next(G)) {
            if (!umma::mbar_wait_warp(&B.acc_full[buf], (i >> 1) & 1u, kWaitLimit)) {
                conv_fail(B, 4);
                break;
            }
            umma::fence_after_sync();
            const int y = t.y0 + (int)ty, x = t.x0 + (int)tx;
            const bool ok = y < (int)A.h && x < (int)A.w;
            for (uint32_t c = 0; c < nt; c += 16) {
                float v[16];
                umma::tmem_ld16(tmem + buf * G.cols + ((32u * q4) << 16) + c, v);
                if (c + 16 >= nt) {  // the accumulator is in registers: release it
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(&B.acc_empty[buf]);
                }
                finish16<EPI>(A, v, n0 + c, c, ok, t.img, y, x, lane, gbw, s_bias, hs, wide);
            }
        }
        if constexpr (EPI == kConvL1) {
            double s = hs.loss;
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0 && count) atomicAdd(A.loss, s);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) umma::tmem_free(tmem, 2 * G.cols);
    if (kSums && count) {
        const uint32_t last = EPI == kConvConcat ? A.nlow : A.N;
        for (uint32_t c = tid; c < nt; c += kThreads) {
            float s = 0.0f;
            for (int k = 0; k < 8; k++) s += s_gb[k * G.np + c];
            if (n0 + c < last) atomicAdd(A.gb + n0 + c, s);
        }
    }
}

// ---- weight gradients -----------------------------------------------------------------------------

// All of the network's weight gradients in one launch.  One CTA is one chain of one layer, the pixels
// of one split in order:
//   D[dx][dy, c][co] = sum over the split's pixels p of x[p + (dy, dx)][c] dz[p][co]
// accumulated in tensor memory in FP32, 16 consecutive pixels per MMA, and added to gw at the end --
// the splits and the order of a split-K GEMM over the im2col matrix, without building either operand.
//
// A stage is a segment of 128 (or 64) consecutive pixels: of the input the image rows that the CTA's
// kernel rows read (all three, or one), as sets of planes one after another, and of the output
// gradient its planes.  M runs over the stacked rows and channels (dy, c) -- 96 of 128 for 32
// channels, one MMA for three taps -- in tiles of 128 (rows past the last plane read whatever lies
// there and are dropped), and dx moves the operand's start by one pixel: no pixel is staged once per
// tap.  A CTA takes one kernel row where three need more tensor memory than there is, or where the
// layer has so few splits that whole ones would finish late.
// Where the width is a multiple of 8 every group of 8 pixels lies in one image row, and 2^k groups of
// one row form a window staged with its two neighbours (kWindows, the widest that divides the row).
// Other widths (the coarse levels of an odd-sized crop) have groups across row ends, whose columns
// see different neighbours: there a CTA serves one dx and stages exactly its pixels (kPerTap).
//
// Roles: warps 0-15 load and at the end drain, three warps issue (one thread's waits and commits alone
// take as long as the MMAs of a segment).
// Bound: instruction issue of the loading warps (49 % of the issue slots; their copies are a
// shared-memory wavefront per 16 bytes) and the issuing warps' waits; the MMAs read 35 % of the
// shared-memory bandwidth.  All 15 layers of a 16 x 256 x 256 step: 0.81 ms, against 14.5 ms of im2col
// transposes and 1.6 ms of split-K GEMMs before.
struct WgradLayer {
    const __nv_bfloat16 *xa, *xb, *dz;
    float* gw;
    uint32_t ca, cb, up, h, w, taps, cout, ldz;
    uint32_t mode, segment, groups;  // staging, pixels per stage, pixel groups per window
    uint32_t pixels, chain;          // pixels in all, and per split
    uint32_t np, mtiles, dys, dxs, cols, stages;  // dys, dxs: kernel rows and columns per CTA
    uint32_t first;                  // CTA index of this layer's first chain
};
struct WgradArgs {
    WgradLayer layer[kMaxWgradLayers];
    uint32_t layers, bars;
    int* error;
    // the head's bias gradient, by the grid's first bias_first CTAs
    uint32_t bias_first;
    const __nv_bfloat16* bias_dz;
    float* bias_out;
    uint32_t bias_pixels;
};
constexpr int kWgradLoadWarps = 16, kWgradIssuers = 3, kWgradThreads = 32 * (kWgradLoadWarps + kWgradIssuers);
constexpr uint32_t kBiasCtas = 4;
enum : uint32_t { kPlain, kWindows, kPerTap };  // staging of the pixels: 1x1 kernel; as above

// bytes of a plane: windows of 8 `groups` pixels and two neighbours
__host__ __device__ constexpr uint32_t wgrad_plane(uint32_t mode, uint32_t segment, uint32_t groups) {
    return (segment + (mode == kWindows ? segment / (8 * groups) * 2 : 0)) * 16u;
}

// A loading thread's share of every segment: one pixel of its warp's octet (if the segment has one for
// the warp) and every fourth plane of each input and of the output gradient, and where the octet
// begins or ends a window one plane of a neighbour.  Addresses and image coordinates advance by a
// segment, without a multiplication or a division; only an upsampled input's are computed per row.
template <uint32_t MODE>
struct SegmentLoader {
    // one lane's pixel in one of the inputs
    struct Source {
        const __nv_bfloat16* base;
        int64_t at;        // element offset of the pixel in the CTA's first image row, at this lane's first plane
        uint32_t c, n;     // channels, planes this lane copies (every fourth)
        uint32_t dst;      // of the first plane
    };
    uint32_t p0, p1;     // of the next segment; end of the chain
    uint32_t x, y, img;  // the octet's first pixel; kPerTap: this lane's pixel
    uint32_t seg, sx, sy, simg, h, w, up, dys;
    uint32_t plane, set;  // bytes of a plane, of one image row's planes
    int dy, dx;           // of the CTA's first kernel row; kPerTap: its column
    Source a, b, e, z;    // the two inputs, the window neighbour, the output gradient
    uint32_t e_up, edge, edges, e_more;
    int ecol;

    __device__ __forceinline__ SegmentLoader(const WgradLayer& L, uint32_t first, uint32_t end, int dy_, int dx_, int tid)
        : p0(first), p1(end), seg(L.segment), h(L.h), w(L.w), up(L.up), dys(L.dys), plane(wgrad_plane(MODE, L.segment, L.groups)),
          dy(dy_), dx(dx_) {
        const uint32_t lane = tid & 31u, g = tid >> 5, pl = lane & 7u, q0 = lane >> 3;
        const uint32_t na = L.ca >> 3, nb = L.cb >> 3, chunks = na + nb, gmask = L.groups - 1;
        set = chunks * plane;
        const uint32_t r = seg / w;
        sx = seg - r * w;
        simg = r / h;
        sy = r - simg * h;
        const uint32_t p = p0 + 8u * g + (MODE == kPerTap ? pl : 0u), row = p / w;
        x = p - row * w;
        img = row / h;
        y = row - img * h;
        // slot of the octet's first pixel in a plane
        const uint32_t slot = MODE == kWindows ? (g / L.groups) * (8 * L.groups + 2) + 8 * (g & gmask) + 1 : 8 * g;
        const int64_t lin = (int64_t)p0 + 8 * g + pl, line = lin + (int64_t)dy * w + (MODE == kPerTap ? dx : 0);
        const auto lanes = [&](const __nv_bfloat16* base, int64_t pixel, uint32_t c, uint32_t n, uint32_t dst) {
            return Source{base, pixel * c + 8 * q0, c, n > q0 ? (n - q0 + 3) / 4 : 0u, dst};
        };
        a = lanes(L.xa, line, L.ca, na, q0 * plane + (slot + pl) * 16u);
        b = lanes(L.xb, line, L.cb, nb, (na + q0) * plane + (slot + pl) * 16u);
        z = lanes(L.dz, lin, L.ldz, L.ldz >> 3, dys * set + (q0 * seg + 8u * g + pl) * 16u);
        // a window's neighbours: lanes 0-15 left of its first octet, 16-31 right of its last, a plane each
        const uint32_t right = lane >> 4, q = lane & 15u;
        edges = MODE == kWindows && ((g & gmask) == 0 || (g & gmask) == gmask);
        edge = MODE == kWindows && (g & gmask) == (right ? gmask : 0u) && q < chunks;
        e_more = chunks > 16;
        const bool in_a = q < na;
        e = Source{in_a ? L.xa : L.xb, 0, in_a ? L.ca : L.cb, 0, q * plane + (slot + (right ? 8u : ~0u)) * 16u};
        e.at = (line - pl + (right ? 8 : -1)) * (int64_t)e.c + 8 * (in_a ? q : q - na);
        e_up = in_a ? up : 0u;
    }
    // element offset of column `col` of image row yy in an upsampled input
    __device__ __forceinline__ uint64_t up_at(const Source& s, int yy, int col) const {
        return (uint64_t)((img * (h >> 1) + ((uint32_t)yy >> 1)) * (w >> 1) + ((uint32_t)col >> 1)) * s.c;
    }
    __device__ __forceinline__ static void copy(const Source& s, uint64_t at, bool ok, uint32_t d, uint32_t dstep) {
        const __nv_bfloat16* src = s.base + (ok ? at : 0);
        const uint32_t bytes = ok ? 16u : 0u, inc = ok ? 32u : 0u;
        for (uint32_t j = 0; j < s.n; j++, d += dstep, src += inc) umma::cp_async16(d, src, bytes);
    }
    __device__ __forceinline__ void operator()(const WgradLayer& L, uint32_t dst, int tid) {
        const uint32_t lane = tid & 31u, g = tid >> 5, pl = lane & 7u;
        if (8u * g < seg) {
            const bool in = p0 + 8u * g + (MODE == kPerTap ? pl : 0u) < p1;
            const int col = (int)x + (MODE == kPerTap ? dx : (int)pl);
            ecol = (int)x + (lane & 16u ? 8 : -1);
            const bool col_ok = in && (MODE != kPerTap || (uint32_t)col < w);
            int yy = (int)y + dy;
            uint32_t d = dst;
            int64_t off = 0;  // of the image row, in pixels
            for (uint32_t r = 0; r < dys; r++, yy++, d += set, off += w) {
                const bool row_ok = (uint32_t)yy < h, ok = row_ok && col_ok;
                copy(a, up ? up_at(a, yy, col) + 8 * (lane >> 3) : (uint64_t)(a.at + off * a.c), ok, d + a.dst, 4 * plane);
                if (b.n) copy(b, (uint64_t)(b.at + off * b.c), ok, d + b.dst, 4 * plane);
                if (MODE == kWindows && edges) {
                    const bool eok = row_ok && in && (uint32_t)ecol < w;
                    const __nv_bfloat16* src = e.base;
                    if (eok && edge) src += e_up ? up_at(e, yy, ecol) + 8 * (lane & 15u) : (uint64_t)(e.at + off * e.c);
                    if (edge) umma::cp_async16(d + e.dst, src, eok ? 16u : 0u);
                    if (e_more) more_edges(L, d, r, yy, eok, lane);
                }
            }
            copy(z, (uint64_t)z.at, p0 + 8u * g + pl < p1, dst + z.dst, 4 * seg * 16u);
            a.at += (int64_t)seg * a.c;
            b.at += (int64_t)seg * b.c;
            e.at += (int64_t)seg * e.c;
            z.at += (int64_t)seg * z.c;
            x += sx;
            y += sy;
            img += simg;
            if (x >= w) { x -= w; y++; }
            if (y >= h) { y -= h; img++; }
        }
        p0 += seg;
    }
    // the neighbours' planes 16 and up
    __device__ __forceinline__ void more_edges(const WgradLayer& L, uint32_t d, uint32_t r, int yy, bool ok, uint32_t lane) const {
        const uint32_t na = L.ca >> 3, chunks = na + (L.cb >> 3), right = lane >> 4;
        for (uint32_t q = 16u + (lane & 15u); q < chunks; q += 16) {
            const bool in_a = q < na;
            const uint32_t c = in_a ? L.ca : L.cb;
            const __nv_bfloat16* src = in_a ? L.xa : L.xb;
            const uint32_t pixel = in_a && up ? (img * (h >> 1) + ((uint32_t)yy >> 1)) * (w >> 1) + ((uint32_t)ecol >> 1)
                                              : (img * h + (uint32_t)yy) * w + (uint32_t)ecol;
            if (ok) src += (uint64_t)pixel * c + 8 * (in_a ? q : q - na);
            if ((warp_window(L) & (1u << right)) != 0)
                umma::cp_async16(d + q * plane + (e.dst - (lane & 15u) * plane), src, ok ? 16u : 0u);
        }
    }
    // bit 0: the warp's octet begins a window, bit 1: it ends one
    __device__ __forceinline__ static uint32_t warp_window(const WgradLayer& L) {
        const uint32_t g = threadIdx.x >> 5, gmask = L.groups - 1;
        return ((g & gmask) == 0 ? 1u : 0u) | ((g & gmask) == gmask ? 2u : 0u);
    }
};

template <uint32_t MODE>
__device__ __forceinline__ void load_segments(const Bars& B, const WgradLayer& L, uint32_t p0, uint32_t p1, uint32_t count,
                                              uint32_t ring, uint32_t stage, int dy, int dx, int tid) {
    SegmentLoader<MODE> load(L, p0, p1, dy, dx, tid);
    load_loop(B, count, L.stages, [&](uint32_t st) { load(L, ring + st * stage, tid); });
}

// gb[ch] += sum of sign(dz) / (3 pixels), one FP32 addition per 32 consecutive pixels
__device__ __forceinline__ void head_bias(const WgradArgs& W, uint32_t cta, int tid) {
    const uint32_t lane = tid & 31u, warps = kBiasCtas * (kWgradThreads / 32);
    const float inv = 1.0f / (3.0f * (float)W.bias_pixels);
    for (uint32_t g = cta * (kWgradThreads / 32) + (tid >> 5); g * 32u < W.bias_pixels; g += warps) {
        const uint32_t p = g * 32u + lane;
        uint2 u = make_uint2(0, 0);
        if (p < W.bias_pixels) u = *reinterpret_cast<const uint2*>(W.bias_dz + (size_t)p * 8);
        const float z[3] = {bf_lo(u.x), bf_hi(u.x), bf_lo(u.y)};
#pragma unroll
        for (int ch = 0; ch < 3; ch++) {
            float d = z[ch] > 0.0f ? inv : (z[ch] < 0.0f ? -inv : 0.0f);
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (lane == 0) atomicAdd(W.bias_out + ch, d);
        }
    }
}

__global__ void __launch_bounds__(kWgradThreads, 1) conv_wgrad_kernel(const __grid_constant__ WgradArgs W) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t lane = tid & 31u;
    if (blockIdx.x < W.bias_first) {
        head_bias(W, blockIdx.x, tid);
        return;
    }
    const Bars B = bars_at(smem + W.bars, W.error);
    const uint32_t base = umma::smem_u32(smem);
    uint32_t li = 0;
    while (li + 1 < W.layers && blockIdx.x >= W.layer[li + 1].first) li++;
    const WgradLayer L = W.layer[li];  // in registers: read through the parameters each field was a load per use
    // the CTA's split and its kernel rows dy0 .. and columns dx0 .. of side x side
    const uint32_t side = L.taps == 9 ? 3u : 1u, parts_x = side / L.dxs, parts = side / L.dys * parts_x;
    const uint32_t job = blockIdx.x - L.first, split = job / parts, part = job - split * parts;
    const uint32_t dy0 = part / parts_x * L.dys, dx0 = part % parts_x * L.dxs;
    const uint32_t p0 = split * L.chain, p1 = min(L.pixels, p0 + L.chain);
    const uint32_t seg = L.segment, count = (p1 - p0 + seg - 1) / seg;
    const uint32_t plane = wgrad_plane(L.mode, seg, L.groups), C = L.ca + L.cb, chunks = C >> 3;
    const uint32_t xbytes = L.dys * chunks * plane, stage = xbytes + (L.ldz >> 3) * (seg * 16u);

    if (warp == kWgradLoadWarps) umma::tmem_alloc(B.tmem, L.cols);
    if (tid == 0) bars_init(B, 32 * kWgradLoadWarps, kWgradIssuers);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *B.tmem;

    if (warp < kWgradLoadWarps) {
        const int dy = L.taps == 9 ? (int)dy0 - 1 : 0, dx = (int)dx0 - 1;
        if (L.mode == kWindows) load_segments<kWindows>(B, L, p0, p1, count, base, stage, dy, dx, tid);
        else if (L.mode == kPerTap) load_segments<kPerTap>(B, L, p0, p1, count, base, stage, dy, dx, tid);
        else load_segments<kPlain>(B, L, p0, p1, count, base, stage, dy, dx, tid);
        // the accumulators into gw: a warp its tensor-memory lane quarter and every fourth 16 columns
        const uint32_t q4 = (uint32_t)warp & 3u, share = (uint32_t)warp >> 2;
        if (count && !umma::mbar_wait_warp(&B.acc_full[0], 0u, kWaitLimit)) conv_fail(B, 4);
        umma::fence_after_sync();
        if (count && !__any_sync(0xffffffffu, conv_failed(B.fail))) {
            const uint32_t K = L.taps * C;
            for (uint32_t mt = 0; mt < L.mtiles; mt++) {
                const uint32_t m = mt * 128u + 32u * q4 + lane, dy = m / C, c = m - dy * C;
                if (mt * 128u + 32u * q4 >= L.dys * C) break;
                for (uint32_t k = 0; k < L.dxs; k++)
                    for (uint32_t n = 16u * share; n < L.np; n += 64) {
                        float v[16];
                        umma::tmem_ld16(tmem + (mt * L.dxs + k) * L.np + ((32u * q4) << 16) + n, v);
#pragma unroll
                        for (uint32_t j = 0; j < 16; j++)
                            if (dy < L.dys && n + j < L.cout)
                                atomicAdd(L.gw + (size_t)(n + j) * K + ((dy0 + dy) * side + dx0 + k) * C + c, v[j]);
                    }
            }
        }
    } else if (umma::elect_one()) {
        const uint32_t mine = (uint32_t)(warp - kWgradLoadWarps);
        const uint32_t idesc = umma::idesc_bf16_f32(128, L.np) | umma::kTransposeA | umma::kTransposeB;
        // K groups (8 pixels) are contiguous within a window; windows of one group are a pitch apart
        const bool narrow = L.mode == kWindows && L.groups == 1;
        const uint32_t lbo = narrow ? 160u : 128u, step = narrow ? 20u : 16u;
        const uint32_t wmask = L.mode == kWindows && !narrow ? (L.groups >> 1) - 1 : ~0u;  // steps per window - 1
        bool ok = true;
        uint32_t st = 0, use = 0;
        for (uint32_t i = 0; i < count; i++) {
            if (conv_failed(B.fail)) { ok = false; break; }
            if (!umma::mbar_wait(&B.full[st], use & 1u, kWaitLimit)) {
                conv_fail(B, 3);
                ok = false;
                break;
            }
            umma::fence_after_sync();
            const uint32_t x = base + st * stage, z = x + xbytes;
            const uint64_t db = umma::smem_desc(z, 128u, seg * 16u);
            for (uint32_t job2 = mine; job2 < L.mtiles * L.dxs; job2 += kWgradIssuers) {
                const uint32_t mt = job2 / L.dxs, k = job2 - mt * L.dxs;
                const uint32_t shift = L.mode == kWindows ? (dx0 + k) * 16u : 0u;
                const uint64_t da = umma::smem_desc(x + mt * 16u * plane + shift, lbo, plane);
                uint32_t a = (uint32_t)da, b = (uint32_t)db;
#pragma unroll 1
                for (uint32_t s = 0; s < seg / 16; s++, b += 16u) {
                    umma::mma_bf16(tmem + job2 * L.np, a, (uint32_t)(da >> 32), b, (uint32_t)(db >> 32), idesc, (i | s) != 0u);
                    a += step;
                    if (wmask != ~0u && ((s + 1) & wmask) == 0) a += 2;
                }
            }
            umma::mma_commit(&B.empty[st]);
            if (++st == L.stages) { st = 0; use++; }
        }
        if (ok && count) umma::mma_commit(&B.acc_full[0]);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kWgradLoadWarps) umma::tmem_free(tmem, L.cols);
}

// ---- host -----------------------------------------------------------------------------------------

uint32_t pow2_cols(uint32_t n) {
    uint32_t c = 32;
    while (c < n) c <<= 1;
    return c;
}

int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 152;
    return sms;
}

void geom_tiles(Geom& G, uint32_t n, uint32_t h, uint32_t w, uint32_t taps, uint32_t channels) {
    G.tiles_x = (w + kTileX - 1) / kTileX;
    G.tiles_y = (h + kTileY - 1) / kTileY;
    G.tiles = n * G.tiles_x * G.tiles_y;
    G.chunks = channels / 8;
    G.hx = kTileX + (taps == 9 ? 2 : 0);
    G.hy = kTileY + (taps == 9 ? 2 : 0);
    G.plane = G.hx * G.hy * 16;
}

// the columns per CTA and stages of a convolution: as few column groups as leave room for two stages
// (every group reads the input again), then as many stages as fit
bool conv_geom(Geom& G, uint32_t channels, uint32_t N, uint32_t taps, size_t* smem) {
    if (channels == 0 || channels % 8 || (channels % 16 && channels != 8)) return false;
    G.kchunks = (taps * G.chunks + 1) & ~1u;
    const uint32_t n16 = (N + 15) / 16;
    G.stage = (G.chunks * G.plane + 127) & ~127u;
    for (uint32_t groups = (n16 + 15) / 16; groups <= n16; groups++) {
        G.np = (n16 + groups - 1) / groups * 16;
        G.wbytes = (G.kchunks * G.np * 16 + 127) & ~127u;
        const size_t fixed = (size_t)G.wbytes + (channels == 8 ? G.plane : 0) + kBarBytes + 8 * G.np * 4 + 128;
        if (fixed + 2 * (size_t)G.stage > kMaxSmem) continue;
        G.stages = (uint32_t)std::min<size_t>(kMaxStages, (kMaxSmem - fixed) / G.stage);
        const uint32_t end = G.wbytes + G.stages * G.stage;
        G.zero = channels == 8 ? end : 0;
        G.bars = (end + (channels == 8 ? G.plane : 0) + 127) & ~127u;
        G.cols = pow2_cols(G.np);
        *smem = (size_t)G.bars + kBarBytes + 8 * G.np * 4;
        return true;
    }
    return false;
}

template <int EPI>
cudaError_t launch_epi(const ConvArgs& a, const Geom& G, dim3 grid, size_t smem, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(conv_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    conv_kernel<EPI><<<grid, kThreads, smem, st>>>(a, G);
    return cudaGetLastError();
}

}  // namespace

bool conv_supported(uint32_t channels, uint32_t N, uint32_t taps) {
    Geom G{};
    size_t smem = 0;
    geom_tiles(G, 1, 1, 1, taps, channels);
    return N > 0 && conv_geom(G, channels, N, taps, &smem) && (N - 1) / G.np < 65535;  // column groups: grid.y
}

cudaError_t launch_conv(const ConvArgs& a, ConvEpilogue epi, cudaStream_t st) {
    if (!a.error || (a.taps != 9 && a.taps != 1) || a.n == 0 || a.h == 0 || a.w == 0 || a.N == 0 || a.ca % 8 || a.cb % 8 || a.ldb % 8 ||
        a.ldb < a.taps * (a.ca + a.cb) || (((uintptr_t)a.xa | (uintptr_t)a.xb | (uintptr_t)a.B) & 15))
        return cudaErrorInvalidValue;
    Geom G{};
    size_t smem = 0;
    geom_tiles(G, a.n, a.h, a.w, a.taps, a.ca + a.cb);
    if (!conv_geom(G, a.ca + a.cb, a.N, a.taps, &smem)) return cudaErrorInvalidValue;
    // the fused epilogues write whole 16-column pieces
    if ((epi == kConvMask || epi == kConvConcat || epi == kConvPool || (epi == kConvStoreBF16 && a.pool)) &&
        (a.N % 16 || (epi == kConvConcat && a.nlow % 16)))
        return cudaErrorInvalidValue;
    const uint32_t groups = (a.N + G.np - 1) / G.np;
    const uint32_t resident = (uint32_t)sm_count();  // one CTA per SM
    const dim3 grid(std::min(G.tiles, std::max(1u, resident / groups)), groups);
    switch (epi) {
    case kConvStoreF32: return launch_epi<kConvStoreF32>(a, G, grid, smem, st);
    case kConvAtomicF32: return launch_epi<kConvAtomicF32>(a, G, grid, smem, st);
    case kConvStoreBF16: return launch_epi<kConvStoreBF16>(a, G, grid, smem, st);
    case kConvHead: return launch_epi<kConvHead>(a, G, grid, smem, st);
    case kConvL1: return launch_epi<kConvL1>(a, G, grid, smem, st);
    case kConvMask: return launch_epi<kConvMask>(a, G, grid, smem, st);
    case kConvConcat: return launch_epi<kConvConcat>(a, G, grid, smem, st);
    case kConvPool: return launch_epi<kConvPool>(a, G, grid, smem, st);
    }
    return cudaErrorInvalidValue;
}

// tensor memory, segment, windows and stages of a layer whose CTAs take L.dys x L.dxs taps (one row
// where three do not fit); *bytes grows to the shared memory it needs
static bool wgrad_shape(WgradLayer& L, size_t* bytes) {
    const uint32_t C = L.ca + L.cb;
    for (;; L.dys = 1) {
        L.mtiles = (L.dys * C + 127) / 128;
        L.cols = pow2_cols(L.mtiles * L.dxs * L.np);
        L.stages = 0;
        for (L.segment = 128; L.segment >= 64 && L.cols <= 512; L.segment /= 2) {
            L.groups = 1;
            if (L.mode == kWindows)  // the widest windows that divide a row and a chain
                for (L.groups = L.segment / 8; L.w % (8 * L.groups) || L.chain % (8 * L.groups); L.groups /= 2) {}
            const uint32_t plane = wgrad_plane(L.mode, L.segment, L.groups);
            const size_t xbytes = (size_t)L.dys * C / 8 * plane, stage = xbytes + (L.ldz / 8) * (L.segment * 16);
            // an operand's unused rows (stacked rows up to a multiple of 128, columns up to np) are read past
            // the stage's planes: keep them inside the allocation
            const size_t over = std::max<size_t>((size_t)L.mtiles * 16 * plane + 32, xbytes + L.np / 8 * (L.segment * 16));
            const size_t pad = over > stage ? over - stage : 0;
            for (L.stages = kMaxStages; L.stages >= 2 && L.stages * stage + pad + kBarBytes + 128 > kMaxSmem;) L.stages--;
            if (L.stages >= 2) {
                *bytes = std::max(*bytes, L.stages * stage + pad);
                return true;
            }
        }
        if (L.dys == 1) return false;
    }
}
// of one CTA, in copies: every pixel's planes
static uint64_t wgrad_cost(const WgradLayer& L) {
    return (uint64_t)L.chain / L.segment * ((uint64_t)L.dys * (L.ca + L.cb) / 8 * wgrad_plane(L.mode, L.segment, L.groups) / 16 + L.ldz / 8 * L.segment);
}
static uint32_t wgrad_parts(const WgradLayer& L) {
    const uint32_t side = L.taps == 9 ? 3 : 1;
    return side / L.dys * (side / L.dxs);
}

cudaError_t launch_conv_wgrad(const WgradTask* tasks, uint32_t count, const __nv_bfloat16* bias_dz, uint64_t bias_pixels,
                              float* bias_gb, int* error, cudaStream_t st) {
    if (!error || count == 0 || count > (uint32_t)kMaxWgradLayers || bias_pixels > 0x7fffffffull) return cudaErrorInvalidValue;
    WgradArgs W{};
    W.error = error;
    W.layers = count;
    W.bias_first = bias_dz ? kBiasCtas : 0;
    W.bias_dz = bias_dz;
    W.bias_out = bias_gb;
    W.bias_pixels = (uint32_t)bias_pixels;
    size_t bytes = 0;
    uint64_t cost[kMaxWgradLayers], total = 0;
    uint32_t order[kMaxWgradLayers];
    WgradLayer layer[kMaxWgradLayers];
    for (uint32_t i = 0; i < count; i++) {
        const WgradTask& t = tasks[i];
        const ConvArgs& a = t.conv;
        const uint64_t pixels = (uint64_t)a.n * a.h * a.w;
        const uint32_t C = a.ca + a.cb;
        if ((a.taps != 9 && (a.taps != 1 || a.w % 8)) || pixels == 0 || pixels > 0x7fffffffull || a.ca % 8 || a.cb % 8 || C == 0 ||
            t.ldz % 8 || t.ldz < t.cout || t.cout == 0 || t.cout > 256 || (((uintptr_t)a.xa | (uintptr_t)a.xb | (uintptr_t)a.dz) & 15))
            return cudaErrorInvalidValue;
        WgradLayer& L = layer[i];
        L = WgradLayer{};
        L.xa = a.xa;
        L.xb = a.xb;
        L.dz = a.dz;
        L.gw = t.gw;
        L.ca = a.ca;
        L.cb = a.cb;
        L.up = a.up ? 1 : 0;
        L.h = a.h;
        L.w = a.w;
        L.taps = a.taps;
        L.cout = t.cout;
        L.ldz = t.ldz;
        L.pixels = (uint32_t)pixels;
        // chains of at least 256 blocks of 64 pixels, at most 64 of them
        const uint32_t kb = (L.pixels + 63) / 64, splits = std::min(64u, std::max(1u, kb / 256)), side = a.taps == 9 ? 3 : 1;
        L.chain = (kb + splits - 1) / splits * 64;
        L.np = (t.cout + 15) & ~15u;
        L.mode = a.taps == 1 ? kPlain : a.w % 8 == 0 ? kWindows : kPerTap;
        L.dxs = L.mode == kPerTap ? 1 : side;
        L.dys = side;
        if (!wgrad_shape(L, &bytes)) return cudaErrorInvalidValue;
        total += wgrad_cost(L) * wgrad_parts(L) * ((L.pixels + L.chain - 1) / L.chain);
        order[i] = i;
    }
    // whole chains that would take over a third of an even share of the work go a kernel row at a time
    // (the output gradient is then read three times)
    const uint64_t share = total / (uint64_t)sm_count();
    for (uint32_t i = 0; i < count; i++) {
        WgradLayer& L = layer[i];
        if (L.dys > 1 && wgrad_cost(L) > share / 3) {
            L.dys = 1;
            if (!wgrad_shape(L, &bytes)) return cudaErrorInvalidValue;
        }
        cost[i] = wgrad_cost(L);
    }
    // the costliest chains first, so that the last ones to finish are short
    std::stable_sort(order, order + count, [&](uint32_t x, uint32_t y) { return cost[x] > cost[y]; });
    uint32_t ctas = W.bias_first;
    for (uint32_t k = 0; k < count; k++) {
        WgradLayer& L = W.layer[k] = layer[order[k]];
        L.first = ctas;
        ctas += (L.pixels + L.chain - 1) / L.chain * wgrad_parts(L);
    }
    W.bars = (uint32_t)((bytes + 127) & ~(size_t)127);
    const size_t smem = (size_t)W.bars + kBarBytes;
    cudaError_t e = cudaFuncSetAttribute(conv_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    conv_wgrad_kernel<<<ctas, kWgradThreads, smem, st>>>(W);
    return cudaGetLastError();
}

}  // namespace rfk
