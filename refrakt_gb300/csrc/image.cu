// Image passes after the chaos game: adaptive density estimation, FP64 histogram statistics
// and the log-density tonemap with a supersample box filter.
//
// The reference does density estimation as a GL point-sprite raster pass with additive
// blending (src/main.cpp:490-515, shaders/density_vert.glsl:26-63, density_frag.glsl:9-18):
// every non-empty bin becomes a sprite of radius r = max(min, min(R, int(R / a^curve))) whose
// fragments add color * (1 - d^2) * (2/pi) / r^2.  Here each warp owns an output tile and gathers it
// from the tile and its halo staged in shared memory, sweeping the sources that reach it (radii above
// kDeMaxSweepR gather from global memory).  The disc is the symmetric restatement
// 4 (dx^2 + dy^2) <= (2r + 1)^2 with
// d^2 = (dx^2 + dy^2) / (r + 0.5)^2 (the GL sprite's sub-pixel centring depends on point
// rasterisation rules).  Radii come from thresholds on a, computed on the host in FP64, and the
// kernel weights are those of a per-radius FP64 table rounded to FP32, so every radius and weight is
// exactly defined.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "kernels.h"
#include "scratch.h"
#include "umma.cuh"

namespace rfk {

constexpr int kDeMaxSmemR = 12;   // radius of the fused path: a tile and its whole halo in shared memory
constexpr int kDeMaxSweepR = 56;  // radius up to which de_weight_params reproduces the weight table

struct DeTables {
    float thr[101];      // thr[k-1]: bin radius >= k  <=>  a <= thr (curve > 0) or a >= thr (curve < 0)
    int R, min_r, mode;  // mode 0: curve > 0, 1: curve < 0, 2: curve == 0 (radius R)
    int wbase[102];      // offset of radius r's (r+1)^2 weights
    double wsum[101];    // the weights of a whole disc of radius r, summed in FP64
};

// the weight coefficients (de_weight_params) of radii up to kDeMaxSmemR
struct DeSmallParams {
    float4 r[kDeMaxSmemR + 1];
};

__device__ __forceinline__ int de_radius(float a, const DeTables& T) {
    int r;
    if (T.mode == 2) r = T.R;
    else if (T.R <= 16) {
        // thresholds are monotone: the number that hold.  Every lane reads the same threshold; the search below
        // reads another one per lane, which the constant cache serves one after another
        r = 0;
        for (int k = 0; k < T.R; k++) r += (T.mode == 0 ? a <= T.thr[k] : a >= T.thr[k]) ? 1 : 0;
    } else {
        // thresholds are monotone: binary search for the largest k with the condition true
        int lo = 0, hi = T.R;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const bool ok = (T.mode == 0) ? (a <= T.thr[mid - 1]) : (a >= T.thr[mid - 1]);
            if (ok) lo = mid; else hi = mid - 1;
        }
        r = lo;
    }
    return r > T.min_r ? r : T.min_r;  // max(min, min(R, int(R / a^curve))), density_vert.glsl:35-44
}

// The densities of a thread's next AHEAD bins, loaded together: with one load in flight per thread the passes
// over all bins are bound by memory latency (8.3 M bins: the radii 31 -> 27 us, the statistics 62 -> 43, also for
// want of FP64 rate; 20 us at the copy bandwidth).  Below kAheadBins a thread has few bins or one: 1.
constexpr size_t kAheadBins = 1u << 20;
template <int AHEAD>
__device__ __forceinline__ void load_densities(const float4* __restrict__ in, size_t i, size_t stride, size_t n,
                                               float (&a)[AHEAD]) {
#pragma unroll
    for (int u = 0; u < AHEAD; u++) a[u] = i + u * stride < n ? in[i + u * stride].w : 0.0f;
}

// CTAs of 256 threads for a pass over n bins
static unsigned pass_ctas(size_t n) { return (unsigned)std::min<size_t>(1024, (n + 255) / 256); }

// pass 1: radius per bin (255 = empty)
template <int AHEAD>
__global__ void de_radius_kernel(const float4* __restrict__ in, size_t n, const __grid_constant__ DeTables T,
                                 uint8_t* __restrict__ rad) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += AHEAD * stride) {
        float a[AHEAD];
        load_densities(in, i, stride, n, a);
#pragma unroll
        for (int u = 0; u < AHEAD; u++)
            if (i + u * stride < n)
                rad[i + u * stride] = (a[u] == 0.0f || a[u] != a[u]) ? (uint8_t)255 : (uint8_t)de_radius(a[u], T);
    }
}

static void launch_radius(const float4* in, size_t n, const DeTables& T, uint8_t* rad, cudaStream_t st) {
    if (n >= kAheadBins) de_radius_kernel<4><<<pass_ctas(n), 256, 0, st>>>(in, n, T, rad);
    else de_radius_kernel<1><<<pass_ctas(n), 256, 0, st>>>(in, n, T, rad);
}

// block-wide FP64 sum, added to *out by one thread per block (blockDim.x a multiple of 32, <= 1024)
__device__ __forceinline__ void block_sum_to(double s, double* out) {
    __shared__ double part[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) part[wid] = s;
    __syncthreads();
    if (wid == 0) {
        s = lane < (int)(blockDim.x >> 5) ? part[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) atomicAdd(out, s);
    }
}

// pass 1 of the fused image tail: the radius per bin, and the total density of the estimator's
// output, sum_out a = sum over bins of a * (the kernel weights of its disc inside the grid) — the
// log-density scale's sum (k2 = W * H / sum a) without a pass over the output.  A whole disc's
// weights come from T.wsum; a disc cut by the grid's edge adds, per row inside the grid,
// the difference of two prefix sums of that row's FP32 weights, staged per CTA in shared memory
// for every radius up to kDeMaxSmemR (the fused path's radii), from the weights' coefficients: reading the table
// from a kernel parameter, a lane at a time, took a third of the pass on small grids (512 x 512: 13 -> 9 us;
// 3840 x 2160 45 us, bound by the instructions per bin).
constexpr int kRowPrefixFloats = 1638;  // sum over r <= 12 of (r + 1) rows of 2r + 2 prefix sums

__global__ void de_radius_sum_kernel(const float4* __restrict__ in, uint32_t w, uint32_t h, const __grid_constant__ DeTables T,
                                     const __grid_constant__ DeSmallParams P, uint8_t* __restrict__ rad,
                                     double* __restrict__ sum_out) {
    __shared__ float s_pre[kRowPrefixFloats];
    __shared__ int s_pbase[kDeMaxSmemR + 1];
    __shared__ float4 s_par[kDeMaxSmemR + 1];
    if (threadIdx.x <= kDeMaxSmemR) s_par[threadIdx.x] = P.r[threadIdx.x];
    const int rmax = min(kDeMaxSmemR, T.R > T.min_r ? T.R : T.min_r);
    if (threadIdx.x == 0) {
        int off = 0;
        for (int r = 0; r <= kDeMaxSmemR; r++) {
            s_pbase[r] = off;
            off += (r + 1) * (2 * r + 2);
        }
    }
    __syncthreads();
    // row (r, ay): pre[j] = sum of the disc's weights at dx = -r .. -r + j - 1
    for (int q = threadIdx.x; q < (rmax + 1) * (rmax + 1); q += blockDim.x) {
        const int r = q / (rmax + 1), ay = q % (rmax + 1);
        if (r < 1 || ay > r) continue;
        float* pre = s_pre + s_pbase[r] + ay * (2 * r + 2);
        const float4 c = s_par[r];
        const float ny2 = -(float)(ay * ay);
        float acc = 0.0f;
        pre[0] = 0.0f;
        for (int dx = -r; dx <= r; dx++) {  // the table's weights as the sweep computes them (de_add)
            const float nx2 = -(float)(dx * dx);
            acc += fmaxf(fmaf(ny2, c.y, fmaf(nx2, c.y, c.x)) + fmaf(ny2, c.w, fmaf(nx2, c.w, c.z)), 0.0f);
            pre[dx + r + 1] = acc;
        }
    }
    __syncthreads();
    // a thread's bins (a few dozen) are summed in FP32, the partial sums in FP64 (this part's
    // FP64 rate is a small fraction of its FP32 rate)
    __shared__ float s_wsum[kDeMaxSmemR + 1];
    for (int r = threadIdx.x; r <= kDeMaxSmemR; r += blockDim.x) s_wsum[r] = (float)T.wsum[r];
    __syncthreads();
    const uint32_t n = w * h;  // < 2^32 (the caller's grids hold fewer bins)
    float s = 0.0f;
    const size_t stride = (size_t)gridDim.x * blockDim.x, first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float ahead[2] = {first < n ? in[first].w : 0.0f, first + stride < n ? in[first + stride].w : 0.0f};  // the next two
    for (size_t i = first; i < n; i += stride) {
        const float a = ahead[0];
        ahead[0] = ahead[1];
        ahead[1] = i + 2 * stride < n ? in[i + 2 * stride].w : 0.0f;
        if (a == 0.0f || a != a) {
            rad[i] = 255;
            continue;
        }
        const int r = de_radius(a, T);
        rad[i] = (uint8_t)r;
        const int y = (int)((uint32_t)i / w), x = (int)((uint32_t)i - (uint32_t)y * w);
        if (x >= r && y >= r && x + r < (int)w && y + r < (int)h) {  // the whole disc (r = 0: weight 1)
            s = fmaf(a, s_wsum[r], s);
            continue;
        }
        const int dx0 = max(-r, -x), dx1 = min(r, (int)w - 1 - x);
        float ws = 0.0f;
        for (int dy = max(-r, -y); dy <= min(r, (int)h - 1 - y); dy++) {
            const float* pre = s_pre + s_pbase[r] + (dy < 0 ? -dy : dy) * (2 * r + 2);
            ws += pre[dx1 + r + 1] - pre[dx0 + r];
        }
        s = fmaf(a, ws, s);
    }
    block_sum_to((double)s, sum_out);
}

// tonemap.glsl:26: the per-bin log-density scale 0.5*brightness*log10(1 + a*k)/a (a > 0)
__device__ __forceinline__ float tonemap_log_scale(float a, float k, float brightness) {
    return 0.5f * brightness * log1pf(a * k) * 0.434294481903251827651128918916f / a;
}

// tonemap.glsl:28-37 on a filtered (r, g, b, a): z = a^(1/gamma), rgb = clamp(mix(rgb^(1/gamma),
// (z/a)*rgb, vibrancy)), alpha 1; no density is opaque black
__device__ __forceinline__ float4 tonemap_finish(float r, float g, float b, float a, float gamma, float vibrancy) {
    if (!(a > 0.0f)) return make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    const float ig = 1.0f / gamma;
    const float gf = powf(a, ig) / a;
    const float rgb[3] = {r, g, b};
    float res[3];
    for (int q = 0; q < 3; q++) {
        // at vibrancy 1 the first term is zero where the power is finite, as it is of every finite colour at
        // gamma >= 1 (a negative one's NaN clamps to 0, as its second term does): three of a pixel's four
        // powers are not needed.  A power that overflows makes the sum NaN, which clamps to 0
        const bool plain = vibrancy == 1.0f && gamma >= 1.0f && fabsf(rgb[q]) < INFINITY;
        const float v = (plain ? 0.0f : powf(rgb[q], ig) * (1.0f - vibrancy)) + gf * rgb[q] * vibrancy;
        res[q] = fminf(fmaxf(v, 0.0f), 1.0f);
    }
    return make_float4(res[0], res[1], res[2], 1.0f);
}

// tonemap.glsl:18-38 for one output pixel from its ss x ss block of bins (rows `stride` apart):
// per bin c *= 0.5*brightness*log10(1 + a*k)/a, mean over the block, then tonemap_finish.
__device__ __forceinline__ float4 tonemap_block(const float4* src, size_t stride, uint32_t ss, float k, float gamma,
                                                float brightness, float vibrancy) {
    float4 acc = make_float4(0, 0, 0, 0);
    for (uint32_t j = 0; j < ss; j++) {
        const float4* row = src + (size_t)j * stride;
        for (uint32_t i = 0; i < ss; i++) {
            const float4 c = row[i];
            if (c.w > 0.0f) {
                const float ls = tonemap_log_scale(c.w, k, brightness);
                acc.x = fmaf(c.x, ls, acc.x);
                acc.y = fmaf(c.y, ls, acc.y);
                acc.z = fmaf(c.z, ls, acc.z);
                acc.w = fmaf(c.w, ls, acc.w);
            }
        }
    }
    const float inv = 1.0f / (float)(ss * ss);
    return tonemap_finish(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv, gamma, vibrancy);
}

// the log-density scale: k2 when given, else bins / sum(a) from the FP64 statistics
__device__ __forceinline__ float tonemap_scale(float k2, const double* stats, uint32_t w, uint32_t h) {
    if (k2 > 0.0f) return k2;
    const double sum = stats ? stats[0] : 0.0;
    return sum > 0.0 ? (float)((double)w * (double)h / sum) : 1.0f;
}

__device__ __forceinline__ uchar4 to_rgba8(float4 o) {
    return make_uchar4((unsigned char)lrintf(o.x * 255.0f), (unsigned char)lrintf(o.y * 255.0f),
                       (unsigned char)lrintf(o.z * 255.0f), 255);
}

// ---- pass 2: the sweep --------------------------------------------------------------------------
//
// A warp owns 32 x ROWS outputs (8, 4 or 2 rows), one column of ROWS outputs per lane, and takes the
// staged source rows one after another, each in the cheaper of two ways (de_row):
//   by offset  every lane takes the source dx columns from its own, for dx up to the row's largest
//              reach; a step without a disc that reaches is dropped (a warp-wide maximum of the radii);
//   by source  the row's non-empty sources, fewer than those offsets, one after another for all lanes.
// Either way a source's colour and weight parameters are read once for up to ROWS outputs, only the output
// rows within the largest disc at hand are touched, and every output adds its sources in ascending
// column order.
//
// The order of every output's sum is fixed: row-major over the discs that cover it, or, in 32 x 8 tiles
// with few discs of radius >= 2 (9 + their number < (2 rmax + 1)^2), first those of radius 0 and 1 and then
// the larger ones, row-major each.
//
// Weights.  w(d2) = (1 - d2 / (r + 1/2)^2) (2/pi) / r^2 as the FP64 table rounds it, without the table:
// with both coefficients split into a multiple of g = 2^-24 times the leading one's binade and a
// remainder, (hi - d2 * step) is exact in FP32, the remainders' part is below 2^-10 of it, and one
// addition rounds their sum: equal to the table for every radius up to 56 and every offset
// (de_weight_params, checked on the host).  Outside the disc the same expression is negative, so its
// maximum with zero is the coverage test.  Two outputs at a time in packed FP32 arithmetic.
//
// An output takes sources that do not cover it times zero, which is nothing where they are finite.  Sums that come out
// not finite are taken again from the covering sources alone (de_row_covered): looking at the sums costs a
// hundredth of the instructions (3840 x 2160 bins 641 -> 629 us, 960 x 540 at radius 20 329 -> 331).
//
// Bound: instruction issue (67 % of the slots at 23 warps per SM; about 70 instructions per source and
// 8 outputs).  Density estimation of 3840 x 2160 bins at 1000 points per bin: 990 us as one output per
// thread over the box of the tile's largest radius, 598 here; 960 x 540 at radius 20 1,090 us as a gather
// from global memory, 330 here.
constexpr int kTileW = 32, kTileH = 8;     // the tile whose discs set the order of its sums
constexpr int kDeThreads = 256;
constexpr int kCtaW = 2 * kTileW;          // a CTA: 8 warps, two side by side, each 32 x ROWS outputs
constexpr int kBandRows = 24;              // staged source rows at a time where the halo is not staged whole

// per radius: hi, step (exact part), and the remainders' coefficients; all zero for an empty bin
struct DeParams {
    float4 r[kDeMaxSweepR + 1];
};

template <bool WHOLE>
using DeParamsFor = std::conditional_t<WHOLE, DeSmallParams, DeParams>;  // as few parameter bytes per launch as it takes

// the tonemap a DE kernel applies to its own output (TM = true)
struct TmArgs {
    uint32_t ss;
    float gamma, brightness, vibrancy, k2;
    const double* stats;  // [0] = sum of the estimator's output density (k2 <= 0)
    float4* out_f32;      // (w / ss) x (h / ss), may be null
    uchar4* out8;         // may be null
};

typedef unsigned long long f32x2;  // two packed FP32 values
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// the lane's outputs: channel c of outputs 2q and 2q + 1 in v[q][c]
template <int ROWS>
struct DeAcc {
    f32x2 v[ROWS / 2][4];
};
// the rows of a warp seen from one source row: their squared distances, negated, and each pair's nearer one
template <int ROWS>
struct DeRows {
    f32x2 ndy2[ROWS / 2];
    int near2[ROWS / 2];
};
// one source (or each lane's own) at -dx^2 into the outputs: colour, parameters p[0], p[1], and the
// largest squared row distance that matters
template <int ROWS>
__device__ __forceinline__ void de_add(DeAcc<ROWS>& acc, const float4& c, const float4* p, float ndx2, const DeRows<ROWS>& rows,
                                       int left) {
    const float4 pa = p[0], pb = p[1];
    const f32x2 nd = pack2(ndx2, ndx2), step = pack2(pa.z, pa.w), lstep = pack2(pb.z, pb.w);
    const f32x2 t0 = fma2(nd, step, pack2(pa.x, pa.y)), l0 = fma2(nd, lstep, pack2(pb.x, pb.y));
    const f32x2 cr = pack2(c.x, c.x), cg = pack2(c.y, c.y), cb = pack2(c.z, c.z), ca = pack2(c.w, c.w);
#pragma unroll
    for (int q = 0; q < ROWS / 2; q++) {
        if (rows.near2[q] > left) continue;
        const float2 w = unpack2(add2(fma2(rows.ndy2[q], step, t0), fma2(rows.ndy2[q], lstep, l0)));
        const f32x2 wt = pack2(fmaxf(w.x, 0.0f), fmaxf(w.y, 0.0f));
        acc.v[q][0] = fma2(cr, wt, acc.v[q][0]);
        acc.v[q][1] = fma2(cg, wt, acc.v[q][1]);
        acc.v[q][2] = fma2(cb, wt, acc.v[q][2]);
        acc.v[q][3] = fma2(ca, wt, acc.v[q][3]);
    }
}

// every output of the warp finite (0 * x is NaN where x is not)
template <int ROWS>
__device__ __forceinline__ bool de_finite(const DeAcc<ROWS>& acc) {
    f32x2 z = 0;
#pragma unroll
    for (int q = 0; q < ROWS / 2; q++)
#pragma unroll
        for (int c = 0; c < 4; c++) z = fma2(acc.v[q][c], 0, z);
    const float2 f = unpack2(z);
    return __all_sync(0xffffffffu, f.x + f.y == 0.0f) != 0;
}
template <int ROWS>
__device__ __forceinline__ void de_clear(DeAcc<ROWS>& acc) {
#pragma unroll
    for (int q = 0; q < ROWS / 2; q++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc.v[q][c] = 0;
}

// One staged source row into the warp's outputs: s_c, s_r (radius + 1, 0 = empty) point at the row's first
// column of the warp's window (R columns left of its outputs), dy = the row's offset from the warp's
// first output row.  WHICH: kAll radii, kSmall (0 and 1) or kLarge (the others).  s_p: the parameters,
// each value twice.
enum DeWhich { kAll, kSmall, kLarge };
template <DeWhich WHICH>
__device__ __forceinline__ int de_pick(int r) {
    if (WHICH == kSmall) return r > 1 ? -1 : r;
    if (WHICH == kLarge) return r < 2 ? -1 : r;
    return r;
}
template <int ROWS, int CHUNKS, DeWhich WHICH>
__device__ __forceinline__ void de_row(DeAcc<ROWS>& acc, const float4* s_c, const uint8_t* s_r, const float4* s_p, int R, int dy) {
    const int lane = threadIdx.x & 31;
    const int md = dy < 0 ? -dy : (dy > ROWS - 1 ? dy - (ROWS - 1) : 0);  // to the warp's nearest row
    // the discs of the row that reach the warp's rows, 32 columns at a time
    unsigned b[CHUNKS];
    int r[CHUNKS], rr = -1, n = 0;
#pragma unroll
    for (int k = 0; k < CHUNKS; k++) {
        const int x = 32 * k + lane;
        r[k] = x < kTileW + 2 * R ? de_pick<WHICH>((int)s_r[x] - 1) : -1;
        if (r[k] < md) r[k] = -1;
        b[k] = __ballot_sync(0xffffffffu, r[k] >= 0);
        n += __popc(b[k]);
        rr = max(rr, r[k]);
    }
    if (n == 0) return;
    rr = __reduce_max_sync(0xffffffffu, rr);
    const int span = min(rr, (int)sqrtf((float)(rr * rr + rr - md * md)));
    DeRows<ROWS> rows;
#pragma unroll
    for (int q = 0; q < ROWS / 2; q++) {
        const int e0 = dy - 2 * q, e1 = e0 - 1;
        rows.ndy2[q] = pack2(-(float)(e0 * e0), -(float)(e1 * e1));
        rows.near2[q] = min(e0 * e0, e1 * e1);
    }
    if (n <= 2 * span + 1) {
#pragma unroll
        for (int k = 0; k < CHUNKS; k++)
            while (b[k]) {
                const int col = __ffs(b[k]) - 1, x = 32 * k + col;
                b[k] &= b[k] - 1;
                const int rs = __shfl_sync(0xffffffffu, r[k], col);
                const float dx = (float)(lane + R - x);
                de_add(acc, s_c[x], s_p + 2 * (rs + 1), -dx * dx, rows, rs * rs + rs);
            }
        return;
    }
    const int reach = md * md;
    for (int dx = -span; dx <= span; dx++) {
        const int q = de_pick<WHICH>((int)s_r[R + lane + dx] - 1);
        const int m = __reduce_max_sync(0xffffffffu, q);
        const int left = m * m + m - dx * dx;
        if (m < 0 || left < reach) continue;
        de_add(acc, s_c[R + lane + dx], s_p + 2 * (q + 1), -(float)(dx * dx), rows, left);
    }
}

// The same for sources that may not be finite: an output that a disc does not cover takes nothing from it
// (in de_add it takes the colour times zero).  Sums of finite sources are the same bits.
template <int ROWS>
__device__ __forceinline__ void de_row_covered(DeAcc<ROWS>& acc, const float4* s_c, const uint8_t* s_r, const float4* s_p, int R,
                                               int dy, DeWhich which) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int dx = -R; dx <= R; dx++) {
        const int x = R + lane + dx, r = (int)s_r[x] - 1;
        if (r < 0 || (which == kSmall && r > 1) || (which == kLarge && r < 2)) continue;
        const float4 c = s_c[x], pa = s_p[2 * (r + 1)], pb = s_p[2 * (r + 1) + 1];
        const float ndx2 = -(float)(dx * dx);
        const float t0 = fmaf(ndx2, pa.z, pa.x), l0 = fmaf(ndx2, pb.z, pb.x);
#pragma unroll
        for (int q = 0; q < ROWS / 2; q++) {
            float wt[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int e = dy - 2 * q - k;
                const float ndy2 = -(float)(e * e);
                wt[k] = fmaxf(__fadd_rn(fmaf(ndy2, pa.z, t0), fmaf(ndy2, pb.z, l0)), 0.0f);
            }
            const f32x2 w2 = pack2(wt[0], wt[1]);
            const bool lo = wt[0] > 0.0f, hi = wt[1] > 0.0f;
            acc.v[q][0] = fma2(pack2(lo ? c.x : 0.0f, hi ? c.x : 0.0f), w2, acc.v[q][0]);
            acc.v[q][1] = fma2(pack2(lo ? c.y : 0.0f, hi ? c.y : 0.0f), w2, acc.v[q][1]);
            acc.v[q][2] = fma2(pack2(lo ? c.z : 0.0f, hi ? c.z : 0.0f), w2, acc.v[q][2]);
            acc.v[q][3] = fma2(pack2(lo ? c.w : 0.0f, hi ? c.w : 0.0f), w2, acc.v[q][3]);
        }
    }
}

// staged rows [row0, row0 + rows) of the CTA's window, whose origin is (gx0, gy0), to the staging's start.
// The radii of a warp's rows are loaded together and the colours copied asynchronously: radius, then colour,
// then the next bin took some forty memory latencies a CTA (3840 x 2160 bins with discs of radius 0 alone 256
// -> 194 us, at 1000 points per bin 642 -> 598).
__device__ __forceinline__ void de_stage(const float4* __restrict__ in, const uint8_t* __restrict__ rad, int w, int h, int gx0,
                                         int gy0, int pitch, int row0, int rows, float4* s_c, uint8_t* s_r) {
    constexpr int kRows = 8;  // a warp's rows at a time
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t to = umma::smem_u32(s_c);
    for (int x = lane; x < pitch; x += 32) {
        const int gx = gx0 + x;
        const bool column = gx >= 0 && gx < w;
        for (int i0 = warp; i0 < rows; i0 += kRows * warps) {
            int r[kRows];
#pragma unroll
            for (int u = 0; u < kRows; u++) {
                const int i = i0 + u * warps, gy = gy0 + row0 + i;
                r[u] = column && i < rows && gy >= 0 && gy < h ? rad[(size_t)gy * w + gx] : 255;
            }
#pragma unroll
            for (int u = 0; u < kRows; u++) {
                const int i = i0 + u * warps, gy = gy0 + row0 + i;
                if (i >= rows) break;
                // the colour lands by itself; an empty bin's is zero
                umma::cp_async16(to + 16u * (uint32_t)(i * pitch + x), r[u] != 255 ? in + (size_t)gy * w + gx : in, r[u] != 255 ? 16u : 0u);
                s_r[i * pitch + x] = (uint8_t)(r[u] + 1);  // 255 -> 0
            }
        }
    }
    umma::cp_async_commit();
    umma::cp_async_wait<0>();
}

__host__ __device__ constexpr size_t de_smem_bytes(int rows, int R, bool whole) {
    const size_t n = (size_t)(whole ? 4 * rows + 2 * R : kBandRows) * (kCtaW + 2 * R);
    return (size_t)(R + 2) * 32 + n * 16 + ((n + 15) & ~(size_t)15);
}

// WHOLE: the halo staged whole (R <= kDeMaxSmemR), each tile's order chosen as above; else the source
// rows pass through shared memory in bands, every tile row-major.  TM: the outputs stay in shared
// memory (over the staging) and are tonemapped there.
template <bool WHOLE, bool TM, int ROWS>
__global__ void __launch_bounds__(kDeThreads, 3) de_sweep_kernel(const float4* __restrict__ in, const uint8_t* __restrict__ rad,
                                                                 uint32_t w, uint32_t h, int R, const __grid_constant__ DeParamsFor<WHOLE> P,
                                                                 float4* __restrict__ out, const TmArgs tm) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int cta_rows = 4 * ROWS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pitch = kCtaW + 2 * R, all = cta_rows + 2 * R;
    const int held = WHOLE ? all : kBandRows;
    float4* s_p = reinterpret_cast<float4*>(smem);                  // (R + 2) x {hi, hi, step, step}, {lo, lo, lstep, lstep}
    float4* s_c = s_p + 2 * (R + 2);
    uint8_t* s_r = reinterpret_cast<uint8_t*>(s_c + (size_t)held * pitch);
    const int tx0 = blockIdx.x * kCtaW, ty0 = blockIdx.y * cta_rows;
    for (int r = threadIdx.x; r <= R + 1; r += kDeThreads) {  // entry 0: the empty bin
        const float4 p = r ? P.r[r - 1] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        s_p[2 * r] = make_float4(p.x, p.x, p.y, p.y);
        s_p[2 * r + 1] = make_float4(p.z, p.z, p.w, p.w);
    }
    const int x0 = (warp & 1) * kTileW, y0 = (warp >> 1) * ROWS;  // the warp's outputs in the CTA's
    DeAcc<ROWS> acc;
    de_clear(acc);
    if constexpr (WHOLE) {
        // the warps whose outputs lie in one 32 x 8 tile look through its discs together (2 rows per warp, the
        // image of 522 x 290 bins at radius 5: 34.8 -> 33.0 us a call)
        constexpr int kShare = kTileH / ROWS, kTiles = 8 / kShare;
        __shared__ int s_tile[2][kTiles];  // the largest radius, the number of discs of radius >= 2
        if (kShare > 1 && threadIdx.x < 2 * kTiles) (&s_tile[0][0])[threadIdx.x] = 0;
        de_stage(in, rad, (int)w, (int)h, tx0 - R, ty0 - R, pitch, 0, all, s_c, s_r);
        __syncthreads();
        // of the discs that reach the warp's 32 x 8 tile: the largest radius, and the number of those of
        // radius >= 2
        int rmax = 0, big = 0;
        const uint8_t* tr = s_r + (y0 & ~(kTileH - 1)) * pitch + x0;
        for (int i = (warp >> 1) % kShare; i < kTileH + 2 * R; i += kShare) {
            const int dy = i - R, md = dy < 0 ? -dy : (dy > kTileH - 1 ? dy - (kTileH - 1) : 0);
            for (int x = lane; x < kTileW + 2 * R; x += 32) {
                const int r = (int)tr[i * pitch + x] - 1, dx = x - R;
                if (r < 0 || r < md || dx + r < 0 || dx - r > kTileW - 1) continue;
                rmax = max(rmax, r);
                big += r >= 2;
            }
        }
        rmax = __reduce_max_sync(0xffffffffu, rmax);
        big = __reduce_add_sync(0xffffffffu, big);
        if (kShare > 1) {
            const int t = ((warp >> 1) / kShare) * 2 + (warp & 1);
            if (lane == 0) {
                atomicMax(&s_tile[0][t], rmax);
                atomicAdd(&s_tile[1][t], big);
            }
            __syncthreads();
            rmax = s_tile[0][t];
            big = s_tile[1][t];
        }
        const float4* wc = s_c + y0 * pitch + x0;  // the warp's window
        const uint8_t* wr = s_r + y0 * pitch + x0;
        const bool small_first = 9 + big < (2 * rmax + 1) * (2 * rmax + 1);
        if (small_first) {
            for (int i = max(0, R - 1); i < min(ROWS + R + 1, ROWS + 2 * R); i++)
                de_row<ROWS, 2, kSmall>(acc, wc + i * pitch, wr + i * pitch, s_p, R, i - R);
            if (big)
                for (int i = R - rmax; i < ROWS + R + rmax; i++)
                    de_row<ROWS, 2, kLarge>(acc, wc + i * pitch, wr + i * pitch, s_p, R, i - R);
        } else {
            for (int i = R - rmax; i < ROWS + R + rmax; i++)
                de_row<ROWS, 2, kAll>(acc, wc + i * pitch, wr + i * pitch, s_p, R, i - R);
        }
        if (!de_finite(acc)) {  // a source that is not finite
            de_clear(acc);
            for (int part = small_first ? kSmall : kAll; part <= (small_first ? kLarge : kAll); part++)
                for (int i = 0; i < ROWS + 2 * R; i++)
                    de_row_covered(acc, wc + i * pitch, wr + i * pitch, s_p, R, i - R, (DeWhich)part);
        }
        __syncthreads();
    } else {
        int again = 0;  // the second time over the bands: a source that is not finite
        for (int b = 0; b < all; b += kBandRows) {
            const int rows = min(kBandRows, all - b);
            __syncthreads();
            de_stage(in, rad, (int)w, (int)h, tx0 - R, ty0 - R, pitch, b, rows, s_c, s_r);
            __syncthreads();
            // this band's rows within reach of the warp's
            const int first = max(0, y0 - b), last = min(rows, y0 + ROWS + 2 * R - b);
            for (int i = first; i < last; i++) {
                const float4* rc = s_c + i * pitch + x0;
                const uint8_t* rr = s_r + i * pitch + x0;
                const int dy = b + i - y0 - R;
                if (again) de_row_covered(acc, rc, rr, s_p, R, dy, kAll);
                else if (R <= 16) de_row<ROWS, 2, kAll>(acc, rc, rr, s_p, R, dy);
                else if (R <= 32) de_row<ROWS, 3, kAll>(acc, rc, rr, s_p, R, dy);
                else de_row<ROWS, 5, kAll>(acc, rc, rr, s_p, R, dy);
            }
            if (b + kBandRows >= all && !again && __syncthreads_or(!de_finite(acc))) {
                again = 1;
                de_clear(acc);
                b = -kBandRows;
            }
        }
    }
    float4* s_out = s_c;  // TM: the CTA's outputs, over the staging (every warp is past it)
#pragma unroll
    for (int q = 0; q < ROWS / 2; q++) {
        const float2 r = unpack2(acc.v[q][0]), g = unpack2(acc.v[q][1]), b = unpack2(acc.v[q][2]), a = unpack2(acc.v[q][3]);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const float4 o = k ? make_float4(r.y, g.y, b.y, a.y) : make_float4(r.x, g.x, b.x, a.x);
            const int oy = y0 + 2 * q + k, ox = x0 + lane;
            const int gx = tx0 + ox, gy = ty0 + oy;
            if (TM) s_out[oy * kCtaW + ox] = o;
            else if (gx < (int)w && gy < (int)h) out[(size_t)gy * w + gx] = o;
        }
    }
    if constexpr (TM) {
        __syncthreads();
        const uint32_t ss = tm.ss, pw = kCtaW / ss, ph = cta_rows / ss, ow = w / ss, oh = h / ss;
        const float k = tonemap_scale(tm.k2, tm.stats, w, h);
        for (uint32_t p = threadIdx.x; p < pw * ph; p += kDeThreads) {
            const uint32_t px = p % pw, py = p / pw;
            const uint32_t gx = tx0 / ss + px, gy = ty0 / ss + py;
            if (gx >= ow || gy >= oh) continue;
            const float4 o = tonemap_block(s_out + (size_t)py * ss * kCtaW + px * ss, kCtaW, ss, k, tm.gamma, tm.brightness,
                                           tm.vibrancy);
            const size_t oi = (size_t)gy * ow + gx;
            if (tm.out_f32) tm.out_f32[oi] = o;
            if (tm.out8) tm.out8[oi] = to_rgba8(o);
        }
    }
}

constexpr size_t kDeMaxSmem = 112 * 1024;  // two CTAs per SM

template <int ROWS>
static cudaError_t set_de_smem() {
    const void* k[3] = {(const void*)de_sweep_kernel<true, false, ROWS>, (const void*)de_sweep_kernel<true, true, ROWS>,
                        (const void*)de_sweep_kernel<false, false, ROWS>};
    for (const void* f : k) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDeMaxSmem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// the DE kernels' shared-memory limits, set once per device before any launch (also before a
// stream capture that contains DE)
cudaError_t density_prepare() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static bool done[64] = {};
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    e = set_de_smem<8>();
    if (e == cudaSuccess) e = set_de_smem<4>();
    if (e == cudaSuccess) e = set_de_smem<2>();
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    return e;
}

// The weight parameters of every radius up to R (the sweep's comment).  The leading coefficient's
// binade sets the grid of the exact part; the remainders are rounded to FP32.
static void de_weight_params(int R, DeParams& P) {
    P.r[0] = make_float4(1.0f, 4.0f, 0.0f, 0.0f);  // radius 0: weight 1 at the centre
    for (int r = 1; r <= R; r++) {
        const double lead = 0.63661977236 / (double)(r * r), slope = lead / ((r + 0.5) * (r + 0.5));
        int e = 0;
        std::frexp(lead, &e);
        const double g = std::ldexp(1.0, e - 24), hi = std::rint(lead / g) * g, step = std::rint(slope / g) * g;
        P.r[r] = make_float4((float)hi, (float)step, (float)(lead - hi), (float)(slope - step));
    }
}

template <int ROWS>
static cudaError_t launch_de_rows(int R, const DeParams& P, const float4* in, const uint8_t* rad, uint32_t w, uint32_t h,
                                  float4* out, cudaStream_t st, const TmArgs* tm) {
    const bool whole = R <= kDeMaxSmemR;
    DeSmallParams S;
    std::copy(P.r, P.r + kDeMaxSmemR + 1, S.r);
    const dim3 grid((w + kCtaW - 1) / kCtaW, (h + 4 * ROWS - 1) / (4 * ROWS));
    const size_t smem = de_smem_bytes(ROWS, R, whole);  // (a fused CTA's outputs fit in its staging)
    if (tm) de_sweep_kernel<true, true, ROWS><<<grid, kDeThreads, smem, st>>>(in, rad, w, h, R, S, out, *tm);
    else if (whole) de_sweep_kernel<true, false, ROWS><<<grid, kDeThreads, smem, st>>>(in, rad, w, h, R, S, out, TmArgs{});
    else de_sweep_kernel<false, false, ROWS><<<grid, kDeThreads, smem, st>>>(in, rad, w, h, R, P, out, TmArgs{});
    return cudaGetLastError();
}

// R: the launch's largest radius.  More rows per warp read a source once for more outputs, fewer leave
// more warps to hide latency.  Measured, radius 9, 250 points per bin, us at 8 / 4 / 2 rows, density estimation
// alone and with the tonemap on chip: 3840 x 2160 (4,080 CTAs of 8 rows) 640 / 736 / 890 and 694 / 835 / 959;
// 2560 x 1440 (1,800) 342 / 376 / 437 and 370 / 422 / 468; 1920 x 1080 (1,020) 235 / 242 / 273 and 252 / 270 / 293;
// 1600 x 900 (725) 183 / 186 / 208 and 195 / 208 / 221; 1440 x 810 (598) 163 / 167 / 179 and 175 / 183 / 192;
// 1280 x 720 (460) 153 / 144 / 152 and 157 / 161 / 161; 960 x 540 114 / 99 / 108 and 120 / 110 / 115; 512 x 512 (256
// CTAs of 4 rows) 90 / 77 / 77 and 97 / 85 / 81; 640 x 360 (230) 89 / 73 / 65 and 97 / 81 / 67; 320 x 180
// 83 / 63 / 48 and 89 / 69 / 50: 8 rows from 4 CTAs for each of the 152 SMs, 4 from about 1.6.
static cudaError_t launch_de_sweep(int R, const float4* in, const uint8_t* rad, uint32_t w, uint32_t h, float4* out,
                                   cudaStream_t st, const TmArgs* tm = nullptr) {
    cudaError_t e = density_prepare();
    if (e != cudaSuccess) return e;
    DeParams P{};
    de_weight_params(R, P);
    const auto ctas = [&](uint32_t rows) { return (uint64_t)((w + kCtaW - 1) / kCtaW) * ((h + 4 * rows - 1) / (4 * rows)); };
    if (ctas(8) >= 4 * 152) return launch_de_rows<8>(R, P, in, rad, w, h, out, st, tm);
    if (ctas(4) >= 240) return launch_de_rows<4>(R, P, in, rad, w, h, out, st, tm);
    return launch_de_rows<2>(R, P, in, rad, w, h, out, st, tm);
}

// large radii: the gather straight from global memory
__global__ void de_gather_global_kernel(const float4* __restrict__ in, const uint8_t* __restrict__ rad,
                                        uint32_t w, uint32_t h, const float* __restrict__ weights,
                                        const DeTables T, float4* __restrict__ out) {
    const int ox = blockIdx.x * blockDim.x + threadIdx.x, oy = blockIdx.y;
    if (ox >= (int)w) return;
    const int Rm = T.R > T.min_r ? T.R : T.min_r;
    float4 acc = make_float4(0, 0, 0, 0);
    for (int dy = -Rm; dy <= Rm; dy++) {
        const int gy = oy + dy;
        if (gy < 0 || gy >= (int)h) continue;
        for (int dx = -Rm; dx <= Rm; dx++) {
            const int gx = ox + dx;
            if (gx < 0 || gx >= (int)w) continue;
            const size_t gi = (size_t)gy * w + gx;
            const int r = rad[gi];
            if (r == 255) continue;
            const int ax = dx < 0 ? -dx : dx, ay = dy < 0 ? -dy : dy;
            if (ax > r || ay > r) continue;
            float wt;
            if (r == 0) wt = 1.0f;
            else {
                if (4 * (ax * ax + ay * ay) > (2 * r + 1) * (2 * r + 1)) continue;
                wt = weights[T.wbase[r] + ay * (r + 1) + ax];
            }
            const float4 v = in[gi];
            acc.x = fmaf(v.x, wt, acc.x);
            acc.y = fmaf(v.y, wt, acc.y);
            acc.z = fmaf(v.z, wt, acc.z);
            acc.w = fmaf(v.w, wt, acc.w);
        }
    }
    out[(size_t)oy * w + ox] = acc;
}

// FP64 sum and max of the density channel, count of non-empty bins
template <int AHEAD>
__global__ void stats_kernel(const float4* __restrict__ in, size_t n, double* out) {
    // (the maximum and the count in FP32 and 32 bits, the sum alone at this part's low FP64 rate)
    double s = 0.0;
    float top = 0.0f;
    uint32_t count = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += AHEAD * stride) {
        float a[AHEAD];
        load_densities(in, i, stride, n, a);
#pragma unroll
        for (int u = 0; u < AHEAD; u++) {
            s += (double)a[u];
            top = a[u] > top ? a[u] : top;
            count += a[u] > 0.0f ? 1u : 0u;
        }
    }
    double m = (double)top;
    unsigned long long nz = count;
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
        nz += __shfl_down_sync(0xffffffffu, nz, o);
    }
    __shared__ double ss[32], sm[32];
    __shared__ unsigned long long sn[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { ss[wid] = s; sm[wid] = m; sn[wid] = nz; }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        s = lane < nw ? ss[lane] : 0.0;
        m = lane < nw ? sm[lane] : 0.0;
        nz = lane < nw ? sn[lane] : 0ull;
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_down_sync(0xffffffffu, s, o);
            m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
            nz += __shfl_down_sync(0xffffffffu, nz, o);
        }
        if (lane == 0) {
            atomicAdd(out, s);
            // a >= 0: the IEEE bit pattern orders like the value
            atomicMax(reinterpret_cast<unsigned long long*>(out + 1), (unsigned long long)__double_as_longlong(m));
            atomicAdd(reinterpret_cast<unsigned long long*>(out + 2), nz);
        }
    }
}

// tonemap.glsl:18-38 with an ss x ss box filter (tonemap_block), one output pixel per thread
__global__ void tonemap_kernel(const float4* __restrict__ in, uint32_t w, uint32_t h, uint32_t ss, float gamma,
                               float brightness, float vibrancy, float k2, const double* __restrict__ stats,
                               float4* __restrict__ out_f32, uchar4* __restrict__ out8) {
    const uint32_t ow = w / ss, oh = h / ss;
    const uint32_t ox = blockIdx.x * blockDim.x + threadIdx.x, oy = blockIdx.y;
    if (ox >= ow || oy >= oh) return;
    const float k = tonemap_scale(k2, stats, w, h);
    const float4 o = tonemap_block(in + (size_t)oy * ss * w + (size_t)ox * ss, w, ss, k, gamma, brightness, vibrancy);
    const size_t oi = (size_t)oy * ow + ox;
    if (out_f32) out_f32[oi] = o;
    if (out8) out8[oi] = to_rgba8(o);
}

// The tonemap with flam3's spatial filter in place of the ss x ss box (no counterpart in the
// reference, which ignores flam3's filter and filter_shape, flame.cpp:166-176): output pixel
// (ox, oy) is the weighted sum, by the separable taps c[i] c[j], of the log-scaled bins of the
// fwidth x fwidth window starting at (ox ss - pad, oy ss - pad), pad = (fwidth - ss) / 2, then
// tonemap_finish.  A CTA stages the log-scaled bins of its tile's windows once in shared memory, sums each of
// their rows along x once per output column, then the rows of each output pixel: 6 + 6 rows' worth of
// shared-memory reads per pixel at ss = 2 and 6 taps instead of 36.  A row's bins are stored by their column
// modulo ss (up to 8), so that a warp's neighbouring pixels read neighbouring 16 bytes.  3840 x 2160 bins to 1920 x
// 1080: 139 -> 106 us (25 us at the copy bandwidth; bound by the instructions of every bin's log scale).
struct FilterArgs {
    int fwidth, pad;
    int tw, th;        // output pixels per CTA tile (tw a power of two)
    float taps[kMaxFilterTaps];
};
struct FilterTile {
    int rw, rh, mod, cols;  // bins of the tile's windows; columns of one residue modulo mod
    __host__ __device__ FilterTile(const FilterArgs& F, int ss)
        : rw(F.tw * ss + F.fwidth - ss), rh(F.th * ss + F.fwidth - ss), mod(ss <= 8 ? ss : 1), cols((rw + mod - 1) / mod) {}
    __host__ __device__ size_t bytes(const FilterArgs& F) const { return ((size_t)rh * mod * cols + (size_t)rh * F.tw) * 16; }
};
constexpr size_t kFilterSmem = 200 * 1024;

__global__ void __launch_bounds__(256) tonemap_filter_kernel(const float4* __restrict__ in, uint32_t w, uint32_t h,
                                                             uint32_t ss_, float gamma, float brightness,
                                                             float vibrancy, float k2, const double* __restrict__ stats,
                                                             const __grid_constant__ FilterArgs F,
                                                             float4* __restrict__ out_f32, uchar4* __restrict__ out8) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int ss = (int)ss_;
    const FilterTile t(F, ss);
    float4* s_l = reinterpret_cast<float4*>(smem);      // [row][column % mod][column / mod]
    float4* s_r = s_l + (size_t)t.rh * t.mod * t.cols;  // [row][output column]
    const int ox0 = blockIdx.x * F.tw, oy0 = blockIdx.y * F.th;
    const int gx0 = ox0 * ss - F.pad, gy0 = oy0 * ss - F.pad;
    const float k = tonemap_scale(k2, stats, w, h);
    constexpr int kLoads = 3;  // rows of a warp at a time: one after another they take as many latencies more
    for (int x = threadIdx.x & 31; x < t.rw; x += 32) {
        const int gx = gx0 + x, col = x / t.mod;
        const bool in_x = gx >= 0 && gx < (int)w;
        float4* dst = s_l + (x - col * t.mod) * t.cols + col;
        for (int y0 = threadIdx.x >> 5; y0 < t.rh; y0 += 8 * kLoads) {
            float4 c[kLoads];
#pragma unroll
            for (int u = 0; u < kLoads; u++) {
                const int y = y0 + 8 * u, gy = gy0 + y;
                c[u] = in_x && y < t.rh && gy >= 0 && gy < (int)h ? in[(size_t)gy * w + gx] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < kLoads; u++) {
                if (y0 + 8 * u >= t.rh) break;
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (c[u].w > 0.0f) {
                    const float ls = tonemap_log_scale(c[u].w, k, brightness);
                    v = make_float4(c[u].x * ls, c[u].y * ls, c[u].z * ls, c[u].w * ls);
                }
                dst[(y0 + 8 * u) * t.mod * t.cols] = v;
            }
        }
    }
    __syncthreads();
    // tw divides 256: a thread keeps its column
    const int px = (int)threadIdx.x & (F.tw - 1), step = 256 / F.tw;
    const float4* column = s_l + (t.mod == ss ? px : px * ss);
    for (int y = (int)threadIdx.x / F.tw; y < t.rh; y += step) {
        float4 r = make_float4(0, 0, 0, 0);
        const float4* at = column + (size_t)y * t.mod * t.cols;
        for (int i = 0; i < F.fwidth; at++)  // one bin of each residue after the other, then the next column
            for (int res = 0; res < t.mod && i < F.fwidth; res++, i++) {
                const float4 v = at[res * t.cols];
                const float c = F.taps[i];
                r.x = fmaf(v.x, c, r.x);
                r.y = fmaf(v.y, c, r.y);
                r.z = fmaf(v.z, c, r.z);
                r.w = fmaf(v.w, c, r.w);
            }
        s_r[y * F.tw + px] = r;
    }
    __syncthreads();
    const uint32_t ow = w / ss_, oh = h / ss_;
    for (int py = (int)threadIdx.x / F.tw; py < F.th; py += step) {
        const uint32_t ox = ox0 + px, oy = oy0 + py;
        if (ox >= ow || oy >= oh) continue;
        float4 acc = make_float4(0, 0, 0, 0);
        for (int j = 0; j < F.fwidth; j++) {
            const float4 r = s_r[(py * ss + j) * F.tw + px];
            const float c = F.taps[j];
            acc.x = fmaf(r.x, c, acc.x);
            acc.y = fmaf(r.y, c, acc.y);
            acc.z = fmaf(r.z, c, acc.z);
            acc.w = fmaf(r.w, c, acc.w);
        }
        const float4 o = tonemap_finish(acc.x, acc.y, acc.z, acc.w, gamma, vibrancy);
        const size_t oi = (size_t)oy * ow + ox;
        if (out_f32) out_f32[oi] = o;
        if (out8) out8[oi] = to_rgba8(o);
    }
}

// flam3's filter functions and their supports: Gaussian exp(-2x^2) sqrt(2/pi) on [-1.5, 1.5],
// box on [-0.5, 0.5], triangle 1 - |x| and the cubic Hermite 2|x|^3 - 3x^2 + 1 on [-1, 1]
static double filter_support(int shape) { return shape == RF_FILTER_BOX ? 0.5 : (shape == RF_FILTER_GAUSSIAN ? 1.5 : 1.0); }
static double filter_value(int shape, double x) {
    const double t = std::fabs(x);
    switch (shape) {
        case RF_FILTER_GAUSSIAN: return std::exp(-2.0 * x * x) * std::sqrt(2.0 / 3.14159265358979323846);
        case RF_FILTER_BOX: return t <= 0.5 ? 1.0 : 0.0;
        case RF_FILTER_TRIANGLE: return t < 1.0 ? 1.0 - t : 0.0;
        case RF_FILTER_HERMITE: return t < 1.0 ? (2.0 * t - 3.0) * t * t + 1.0 : 0.0;
        default: return 0.0;
    }
}

// The taps: the window spans fw = 2 * support * ss * radius bins, rounded up to an integer width
// of the parity of ss (so it centres on the output pixel's ss x ss block), sampled at each
// cell's centre with the coordinate stretched so the window covers the support, normalised in
// FP64.  Returns fwidth, or -1 beyond kMaxFilterTaps.
int filter_taps(uint32_t ss, float radius, int shape, float* taps) {
    const double support = filter_support(shape);
    const double fw = 2.0 * support * (double)ss * (double)radius;
    int fwidth = (int)fw + 1;
    if ((fwidth ^ (int)ss) & 1) fwidth++;
    if (fwidth > kMaxFilterTaps) return -1;
    const double adjust = fw > 0.0 ? support * (double)fwidth / fw : 1.0;
    double t[kMaxFilterTaps], sum = 0.0;
    for (int i = 0; i < fwidth; i++) {
        t[i] = filter_value(shape, ((2.0 * i + 1.0) / (double)fwidth - 1.0) * adjust);
        sum += t[i];
    }
    for (int i = 0; i < fwidth; i++) taps[i] = (float)(t[i] / sum);
    return fwidth;
}

cudaError_t launch_tonemap_filter(const float4* in, uint32_t w, uint32_t h, uint32_t ss, float radius, int shape,
                                  float gamma, float brightness, float vibrancy, float k2, const double* stats,
                                  float4* out_f32, uchar4* out8, cudaStream_t st) {
    FilterArgs F{};
    F.fwidth = filter_taps(ss, radius, shape, F.taps);
    if (F.fwidth < 0) return cudaErrorInvalidValue;
    F.pad = (F.fwidth - (int)ss) / 2;
    // the largest tile whose staged windows and row sums fit in 64 KB of shared memory (three CTAs an SM), else
    // in all of it
    static const int tiles[][2] = {{32, 8}, {16, 8}, {8, 8}, {8, 4}, {4, 4}, {2, 2}, {1, 1}};
    size_t smem = 0;
    for (const size_t limit : {(size_t)64 * 1024, kFilterSmem}) {
        for (const auto& t : tiles) {
            F.tw = t[0];
            F.th = t[1];
            smem = FilterTile(F, (int)ss).bytes(F);
            if (smem <= limit) break;
        }
        if (smem <= limit) break;
    }
    if (smem > kFilterSmem) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(tonemap_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFilterSmem);
    if (e != cudaSuccess) return e;
    const uint32_t ow = w / ss, oh = h / ss;
    const dim3 grid((ow + F.tw - 1) / F.tw, (oh + F.th - 1) / F.th);
    tonemap_filter_kernel<<<grid, 256, smem, st>>>(in, w, h, ss, gamma, brightness, vibrancy, k2, stats, F, out_f32,
                                                   out8);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// the radius thresholds alone
static void de_thresholds(int R, int min_r, float curve, DeTables& T) {
    T = DeTables{};
    T.R = R;
    T.min_r = min_r;
    T.mode = (curve > 0.0f) ? 0 : (curve < 0.0f ? 1 : 2);
    for (int k = 1; k <= R; k++) {
        // int(R / a^curve) >= k  <=>  a^curve <= R / k
        const double t = std::pow((double)R / (double)k, 1.0 / (double)curve);
        float f = (float)t;
        if (T.mode == 0 && (double)f > t) f = std::nextafter(f, -INFINITY);  // a <= f  <=>  a <= t
        if (T.mode == 1 && (double)f < t) f = std::nextafter(f, INFINITY);   // a >= f  <=>  a >= t
        T.thr[k - 1] = f;
    }
}

static void de_tables(int R, int min_r, float curve, DeTables& T, std::vector<float>& wts) {
    de_thresholds(R, min_r, curve, T);
    wts.clear();
    const int rmax = R > min_r ? R : min_r;
    for (int r = 0; r <= rmax && r <= 100; r++) {
        T.wbase[r] = (int)wts.size();
        const double nf = 0.63661977236 / (double)(r > 0 ? r * r : 1);
        const double den = (r + 0.5) * (r + 0.5);
        for (int ay = 0; ay <= r; ay++)
            for (int ax = 0; ax <= r; ax++) {
                const int d2 = ax * ax + ay * ay;
                wts.push_back(r == 0 ? 1.0f : (float)((1.0 - (double)d2 / den) * nf));
            }
        // the whole disc: the table's weights of every (dx, dy) with 4 (dx^2 + dy^2) <= (2r + 1)^2
        double s = 0.0;
        for (int dy = -r; dy <= r; dy++)
            for (int dx = -r; dx <= r; dx++) {
                const int ax = dx < 0 ? -dx : dx, ay = dy < 0 ? -dy : dy;
                if (r == 0) s += 1.0;
                else if (4 * (ax * ax + ay * ay) <= (2 * r + 1) * (2 * r + 1))
                    s += (double)wts[T.wbase[r] + ay * (r + 1) + ax];
            }
        T.wsum[r] = s;
    }
}

static cudaError_t launch_density_passes(const float4* in, uint32_t w, uint32_t h, const DeTables& T, float4* out,
                                         uint8_t* rad, const float* dw, cudaStream_t st);

cudaError_t launch_density(const float4* in, uint32_t w, uint32_t h, int R, int min_r, float curve, float4* out,
                           cudaStream_t st) {
    DeTables T;
    std::vector<float> wts;
    const bool sweep = !density_reads_weights(R, min_r);
    if (sweep) de_thresholds(R, min_r, curve, T);
    else de_tables(R, min_r, curve, T, wts);
    uint8_t* rad = nullptr;
    float* dw = nullptr;
    cudaError_t e = scratch_alloc(&rad, (size_t)w * h, st);
    if (e != cudaSuccess) return e;
    if (!sweep) {
        e = scratch_alloc(&dw, wts.size(), st);
        if (e != cudaSuccess) { cudaFreeAsync(rad, st); return e; }
        cudaMemcpyAsync(dw, wts.data(), wts.size() * sizeof(float), cudaMemcpyHostToDevice, st);
    }
    e = launch_density_passes(in, w, h, T, out, rad, dw, st);
    cudaFreeAsync(rad, st);
    if (dw) cudaFreeAsync(dw, st);
    return e;
}

bool density_reads_weights(int R, int min_r) { return std::max(R, min_r) > kDeMaxSweepR; }

size_t density_weight_count(int R, int min_r) {
    const int rmax = R > min_r ? R : min_r;
    size_t n = 0;
    for (int r = 0; r <= rmax && r <= 100; r++) n += (size_t)(r + 1) * (r + 1);
    return n;
}

static cudaError_t launch_density_passes(const float4* in, uint32_t w, uint32_t h, const DeTables& T, float4* out,
                                         uint8_t* rad, const float* dw, cudaStream_t st) {
    const size_t n = (size_t)w * h;
    launch_radius(in, n, T, rad, st);
    const int rmax = T.R > T.min_r ? T.R : T.min_r;
    if (rmax <= kDeMaxSweepR) return launch_de_sweep(rmax, in, rad, w, h, out, st);
    de_gather_global_kernel<<<dim3((w + 127) / 128, h), 128, 0, st>>>(in, rad, w, h, dw, T, out);
    return cudaGetLastError();
}

bool density_tonemap_fused(int R, int min_r, uint32_t ss) {
    const int rmax = R > min_r ? R : min_r;
    return rmax <= kDeMaxSmemR && ss >= 1 && kTileW % ss == 0 && kTileH % ss == 0;
}

// The image tail of a frame (main.cpp:490-535: the density-estimation raster pass, then the
// tonemap pass) in two passes: pass 1 finds every bin's radius and, for an automatic k2, the FP64
// density sum of the estimator's output (de_radius_sum_kernel); pass 2 estimates each 32 x 8 tile
// in shared memory and tonemaps it there, so the estimator's FP32 output never reaches DRAM.
// Where that does not apply (density_tonemap_fused false: ss does not divide the tile, or radii
// beyond the shared-memory path) the estimator writes `de_scratch`, then the statistics and
// tonemap passes run on it.  rad: a byte per bin; dw: the weight table (density_weights) where
// density_reads_weights, else unused; stats: 3 doubles.
cudaError_t launch_density_tonemap(const float4* in, uint32_t w, uint32_t h, int R, int min_r, float curve,
                                   uint32_t ss, float gamma, float brightness, float vibrancy, float k2,
                                   float4* out_f32, uchar4* out8, uint8_t* rad, const float* dw, double* stats,
                                   float4* de_scratch, cudaStream_t st) {
    DeTables T;
    std::vector<float> wts;
    const bool need_sum = !(k2 > 0.0f), fused = density_tonemap_fused(R, min_r, ss);
    if ((fused && need_sum) || density_reads_weights(R, min_r)) de_tables(R, min_r, curve, T, wts);
    else de_thresholds(R, min_r, curve, T);
    cudaError_t e;
    if (!fused) {
        if (!de_scratch) return cudaErrorInvalidValue;
        e = launch_density_passes(in, w, h, T, de_scratch, rad, dw, st);
        if (e == cudaSuccess && need_sum) e = launch_stats(de_scratch, w, h, stats, st);
        if (e == cudaSuccess)
            e = launch_tonemap(de_scratch, w, h, ss, gamma, brightness, vibrancy, k2, need_sum ? stats : nullptr,
                               out_f32, out8, st);
        return e;
    }
    if (need_sum) {
        e = cudaMemsetAsync(stats, 0, 3 * sizeof(double), st);
        if (e != cudaSuccess) return e;
        DeParams P{};
        DeSmallParams S;
        de_weight_params(kDeMaxSmemR, P);
        std::copy(P.r, P.r + kDeMaxSmemR + 1, S.r);
        de_radius_sum_kernel<<<1024, 256, 0, st>>>(in, w, h, T, S, rad, stats);
    } else {
        launch_radius(in, (size_t)w * h, T, rad, st);
    }
    const TmArgs tm{ss, gamma, brightness, vibrancy, k2, need_sum ? stats : nullptr, out_f32, out8};
    return launch_de_sweep(R > min_r ? R : min_r, in, rad, w, h, nullptr, st, &tm);
}

void density_weights(int R, int min_r, std::vector<float>& wts) {
    DeTables T;
    de_tables(R, min_r, 1.0f, T, wts);
}

cudaError_t launch_density_resident(const float4* in, uint32_t w, uint32_t h, int R, int min_r, float curve,
                                    float4* out, uint8_t* rad, const float* dw, cudaStream_t st) {
    DeTables T;
    std::vector<float> wts;
    if (density_reads_weights(R, min_r)) de_tables(R, min_r, curve, T, wts);
    else de_thresholds(R, min_r, curve, T);
    return launch_density_passes(in, w, h, T, out, rad, dw, st);
}

cudaError_t launch_stats(const float4* in, uint32_t w, uint32_t h, double* out3, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out3, 0, 3 * sizeof(double), st);
    if (e != cudaSuccess) return e;
    const size_t n = (size_t)w * h;
    if (n >= kAheadBins) stats_kernel<4><<<1024, 256, 0, st>>>(in, n, out3);
    else stats_kernel<1><<<1024, 256, 0, st>>>(in, n, out3);
    return cudaGetLastError();
}

// out2 = (sum h, sum h^2) of a hit-count histogram, FP64; out2 must start at zero
__global__ void hit_moments_kernel(const uint32_t* __restrict__ hits, size_t n, double* out2) {
    double s = 0.0, q = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = (double)hits[i];
        s += v;
        q += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        q += __shfl_down_sync(0xffffffffu, q, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out2, s);
        atomicAdd(out2 + 1, q);
    }
}

cudaError_t launch_hit_moments(const uint32_t* hits, uint32_t w, uint32_t h, double* out2, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out2, 0, 2 * sizeof(double), st);
    if (e != cudaSuccess) return e;
    hit_moments_kernel<<<256, 256, 0, st>>>(hits, (size_t)w * h, out2);
    return cudaGetLastError();
}

cudaError_t launch_tonemap(const float4* in, uint32_t w, uint32_t h, uint32_t ss, float gamma, float brightness,
                           float vibrancy, float k2, const double* stats, float4* out_f32, uchar4* out8,
                           cudaStream_t st) {
    const uint32_t ow = w / ss, oh = h / ss;
    tonemap_kernel<<<dim3((ow + 127) / 128, oh), 128, 0, st>>>(in, w, h, ss, gamma, brightness, vibrancy, k2, stats,
                                                               out_f32, out8);
    return cudaGetLastError();
}

}  // namespace rfk
