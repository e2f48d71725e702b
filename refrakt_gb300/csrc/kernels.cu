// Chaos-game kernels for sm_103a: the interpreted chaos kernel (its body, the walker shuffle
// and the reference's RNG draw order are in chaos_body.cuh), RNG seeding, the walker-shuffle
// table, temporal-sample animation and the single-step probe.
#include <cuda_runtime.h>

#include <algorithm>

#include "chaos_body.cuh"
#include "kernels.h"

namespace rfk {

template <int THREADS, int SPT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) chaos_kernel(const ChaosArgs A) {
    chaos_body<THREADS, SPT, InterpEval>(A);
}

// Interleaved bin records (32 bytes: float4 RGBA, uint32 count, pad) added into the caller's
// planes, then cleared for the next call.
__global__ void merge_records_kernel(float4* __restrict__ rec, size_t n, float4* __restrict__ bins,
                                     uint32_t* __restrict__ hits) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = rec[2 * i];
        const uint32_t c = reinterpret_cast<const uint32_t*>(rec + 2 * i + 1)[0];
        if (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f) {
            float4 b = bins[i];
            b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
            bins[i] = b;
            rec[2 * i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        if (c) {
            if (hits) hits[i] += c;
            rec[2 * i + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
}

cudaError_t launch_merge_records(float4* rec, size_t n, float4* bins, uint32_t* hits, cudaStream_t st) {
    merge_records_kernel<<<152 * 16, 256, 0, st>>>(rec, n, bins, hits);
    return cudaGetLastError();
}

// One step of adding the point lists (chaos_args.h, splat 4) to the planes: range `range`'s lists into scratch
// planes that stay in L2, and range - 1's scratch planes (the other set) into the caller's, cleared.  The
// first half is bound by the SMs' requests to L2 (a reduction or two per point), the second by DRAM (the
// planes read and written once), so they run side by side, in interleaved CTAs of one launch.  80 M points
// of the space-filling genome on 8192 x 8192 bins: lists written by the chaos kernel in 0.76 ms, added in
// 33 steps of 20 to 48 us (of which 335 us are the reductions, 156 us reading the lists, 430 us the planes,
// 130 us launches), 1.84 ms in all; interleaved records written at random and merged took 2.9 + 0.8 ms.
// Ranges of 2^20 bins 1.95 ms; 256 threads, 4 CTAs per SM (spills), half the merging CTAs 1.87 to 1.94.
//
// Where a range's lists hold fewer than 2^24 points (range_count_kernel), a point of opacity 1 takes one
// reduction: the alpha sum of such points is their exact count.  The others go to a second set with a count
// plane.  In a fuller range every point takes its colour's reduction and its count's (80 M points on 8192 x 4608
// bins: 2.4 instead of 1.65 ms).
struct RangeArgs {
    const uint2* list;
    const uint32_t* list_n;
    uint32_t cap, ranges, range_bits, ctas, range, nb;
    const float4* palette;
    RangeScratch set[2];
    RangeState* state;  // per range
    float4* bins;
    uint32_t* hits;
};
constexpr uint32_t kRangeThreads = 512, kMergeCtas = 1024;

// a CTA per range: whether its lists hold fewer than 2^24 points
__global__ void __launch_bounds__(256) range_count_kernel(const uint32_t* __restrict__ list_n, uint32_t ctas, uint32_t ranges,
                                                          uint32_t cap, RangeState* state) {
    __shared__ unsigned long long s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    unsigned long long in = 0;
    for (uint32_t c = threadIdx.x; c < ctas; c += 256) in += min(list_n[(size_t)c * ranges + blockIdx.x], cap);
    atomicAdd(&s_sum, in);
    __syncthreads();
    if (threadIdx.x == 0) state[blockIdx.x] = RangeState{s_sum < (1u << 24) ? 1u : 0u, 0u};
}

template <bool UNIT>
__device__ __forceinline__ void range_add(const RangeArgs& R, uint32_t cta, float4* s_pal) {
    const size_t at = (size_t)cta * R.ranges + R.range;
    const uint32_t n = min(R.list_n[at], R.cap);
    if (n == 0) return;
    const uint2* list = R.list + at * R.cap;
    const RangeScratch& S = R.set[R.range & 1];
    if (threadIdx.x < 256) s_pal[threadIdx.x] = R.palette[threadIdx.x];
    __syncthreads();
    constexpr int U = 4;  // entries in flight per thread
    for (uint32_t i0 = 0; i0 < n; i0 += kRangeThreads * U) {
        uint2 e[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + kRangeThreads * u + threadIdx.x;
            e[u] = i < n ? __ldcs(list + i) : make_uint2(kNoBin, 0u);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t bin = e[u].x == kNoBin ? kNoBin : e[u].x & 0xffffffu;
            const float op = __uint_as_float(e[u].y);
            const float4 c = s_pal[e[u].x >> 24];
            const float4 v = make_float4(c.x, c.y, c.z, op);
            if (UNIT) {
                const bool other = bin != kNoBin && op != 1.0f;
                splat_adaptive(BinTarget{S.rgba, nullptr, 0u, 0u}, other ? kNoBin : bin, v);
                if (__any_sync(0xffffffffu, other)) {
                    splat_adaptive(BinTarget{S.rgba2, S.count, 0u, 0u}, other ? bin : kNoBin, v);
                    if (other) R.state[R.range].mixed = 1u;
                }
            } else {
                splat_adaptive(BinTarget{S.rgba, S.count, 0u, 0u}, bin, v);
            }
        }
    }
}

template <bool UNIT>
__device__ __forceinline__ void range_merge(const RangeArgs& R, uint32_t cta) {
    const uint32_t r = R.range - 1, first = r << R.range_bits, n = min(R.nb - first, 1u << R.range_bits);
    const RangeScratch& S = R.set[r & 1];
    const bool mixed = UNIT && R.state[r].mixed != 0;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    constexpr uint32_t kStep = kMergeCtas * kRangeThreads;
    constexpr int U = 2;
    for (uint32_t i0 = cta * kRangeThreads + threadIdx.x; i0 < n; i0 += kStep * U) {
        float4 v[U], b[U];
        uint32_t c[U], h[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + kStep * u;
            v[u] = zero;
            c[u] = 0u;
            if (i >= n) continue;
            if (UNIT) {
                v[u] = S.rgba[i];
                c[u] = (uint32_t)v[u].w;
                if (v[u].w != 0.0f) S.rgba[i] = zero;
                if (mixed) {
                    if (const uint32_t m = S.count[i]) {
                        const float4 w = S.rgba2[i];
                        v[u] = make_float4(v[u].x + w.x, v[u].y + w.y, v[u].z + w.z, v[u].w + w.w);
                        c[u] += m;
                        S.rgba2[i] = zero;
                        S.count[i] = 0u;
                    }
                }
            } else {
                c[u] = S.count[i];
                if (c[u]) {
                    v[u] = S.rgba[i];
                    S.rgba[i] = zero;
                    S.count[i] = 0u;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c[u]) {
                b[u] = __ldcs(R.bins + first + i0 + kStep * u);
                h[u] = __ldcs(R.hits + first + i0 + kStep * u);
            }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c[u]) {
                __stcs(R.bins + first + i0 + kStep * u,
                       make_float4(b[u].x + v[u].x, b[u].y + v[u].y, b[u].z + v[u].z, b[u].w + v[u].w));
                __stcs(R.hits + first + i0 + kStep * u, h[u] + c[u]);
            }
    }
}

__global__ void __launch_bounds__(kRangeThreads, 3) range_step_kernel(const __grid_constant__ RangeArgs R) {
    __shared__ float4 s_pal[256];
    const uint32_t adds = R.range < R.ranges ? R.ctas : 0u, merges = R.range > 0 ? kMergeCtas : 0u;
    const uint32_t both = 2 * min(adds, merges);
    const bool add = blockIdx.x < both ? (blockIdx.x & 1u) == 0u : adds > merges;
    const uint32_t cta = blockIdx.x < both ? blockIdx.x >> 1 : blockIdx.x - both / 2;
    const bool unit = R.state[add ? R.range : R.range - 1].unit != 0;
    if (add) {
        if (unit) range_add<true>(R, cta, s_pal);
        else range_add<false>(R, cta, s_pal);
    } else {
        if (unit) range_merge<true>(R, cta);
        else range_merge<false>(R, cta);
    }
}

cudaError_t load_draw_kernels() {
    cudaFuncAttributes f;
    for (const void* k : {(const void*)range_count_kernel, (const void*)range_step_kernel, (const void*)merge_records_kernel})
        if (const cudaError_t e = cudaFuncGetAttributes(&f, k)) return e;
    return cudaSuccess;
}

cudaError_t launch_ranges(const ChaosArgs& a, uint32_t ctas, const RangeScratch set[2], RangeState* state, cudaStream_t st) {
    RangeArgs R{a.list, a.list_n, a.list_cap, a.ranges, a.range_bits, ctas, 0, a.W * a.H, a.palette, {set[0], set[1]}, state, a.bins, a.hits};
    range_count_kernel<<<a.ranges, 256, 0, st>>>(a.list_n, ctas, a.ranges, a.list_cap, state);
    cudaError_t e = cudaGetLastError();
    for (; R.range <= a.ranges && e == cudaSuccess; R.range++) {
        const uint32_t grid = (R.range < a.ranges ? ctas : 0u) + (R.range > 0 ? kMergeCtas : 0u);
        range_step_kernel<<<grid, kRangeThreads, 0, st>>>(R);
        e = cudaGetLastError();
    }
    return e;
}

// src/flame.cpp:138-141 — slot i seeded with warmup_ctx(i + seed * N)
__global__ void init_rng_kernel(uint4* rng, uint64_t n, uint64_t seed) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Jsf s = jsf_seed((uint32_t)(i + seed * n));
    rng[i] = make_uint4(s.a, s.b, s.c, s.d);
}

// the walker-shuffle table: `count` keyed permutations of [0, n), one entry per thread
__global__ void shuffle_table_kernel(uint16_t* out, uint32_t n, uint32_t count, uint64_t seed) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)n * count) return;
    const uint32_t k = (uint32_t)(i / n), j = (uint32_t)(i - (uint64_t)k * n);
    out[i] = (uint16_t)feistel(j, n, derive_key(seed, k, 0, TAG_TABLE));
}

// The pipelined exchange's table (chaos_body.cuh, PIPE): with P = n/S slots per phase, the last
// phase's destinations [n-P, n) take the first P of a keyed order of [P, n) — never a walker of
// the previous pass's first phase, whose slots a fast thread may already overwrite — and the first
// phase's destinations [0, P) the first P not yet taken of a keyed order of [0, n-P) — never a
// walker of the previous pass's last phase, which a slow thread may still be computing; the middle
// destinations take the rest in a keyed order of [0, n).  One warp per permutation: the lanes walk
// each keyed order 32 entries at a time and a ballot ranks the free ones, so the result is the
// sequential scan's.  The taken-slot bitmap is in shared memory (n / 32 words per warp).
// n <= kMaxPipeSlots, S >= 3 (then enough sources stay free for the first phase).
constexpr uint32_t kMaxPipeSlots = 4096;
constexpr int kPipeTableWarps = 8;  // permutations per CTA
__global__ void __launch_bounds__(32 * kPipeTableWarps)
    shuffle_table_pipe_kernel(uint16_t* out, uint32_t n, uint32_t count, uint64_t seed, uint32_t phases) {
    __shared__ uint32_t s_taken[kPipeTableWarps][kMaxPipeSlots / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x * kPipeTableWarps + w;
    if (k >= count) return;  // whole warps leave together
    uint32_t* taken = s_taken[w];
    for (uint32_t i = lane; i < n / 32; i += 32) taken[i] = 0;
    __syncwarp();
    const uint32_t P = n / phases;
    uint16_t* o = out + (size_t)k * n;
    const uint64_t k3 = derive_key(seed, k, 3, TAG_TABLE), k1 = derive_key(seed, k, 1, TAG_TABLE),
                   k2 = derive_key(seed, k, 2, TAG_TABLE);
    for (uint32_t d = lane; d < P; d += 32) {
        const uint32_t src = P + feistel(d, n - P, k3);
        o[n - P + d] = (uint16_t)src;
        atomicOr(&taken[src >> 5], 1u << (src & 31));
    }
    __syncwarp();
    // the untaken entries of a keyed order of [0, len), in order, to destinations [d0, d1)
    auto scan = [&](uint32_t len, uint64_t key, uint32_t d0, uint32_t d1) {
        uint32_t d = d0;
        for (uint32_t base = 0; base < len && d < d1; base += 32) {
            const uint32_t i = base + lane;
            const uint32_t src = i < len ? feistel(i, len, key) : 0u;
            const bool free = i < len && !((taken[src >> 5] >> (src & 31)) & 1u);
            const uint32_t ballot = __ballot_sync(0xffffffffu, free);
            const uint32_t rank = __popc(ballot & ((1u << lane) - 1u));
            if (free && d + rank < d1) {
                o[d + rank] = (uint16_t)src;
                atomicOr(&taken[src >> 5], 1u << (src & 31));
            }
            d = min(d + (uint32_t)__popc(ballot), d1);
            __syncwarp();
        }
    };
    scan(n - P, k1, 0, P);
    scan(n, k2, P, n - P);
}

// animate.tpl.glsl:18-96 — one program copy per temporal sample, each xform's linear part
// rotated by 0.31415926535 * dt * rotation_frequency, dt = (t - T/2) / (T/2) * tss_width.
__global__ void animate_kernel(const uint32_t* base, uint32_t words, uint32_t T, float tss_width,
                               uint32_t* out, uint32_t stride) {
    const uint32_t t = blockIdx.x;
    uint32_t* dst = out + (size_t)t * stride;
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = base[i];
    __syncthreads();
    if (T < 2 || threadIdx.x != 0) return;  // T = 1: the template divides 0 by 0; no rotation
    const int half = (int)(T / 2);
    const float dt = (float)((int)t - half) / (float)half * tss_width;
    const uint32_t nx = base[H_NX];
    for (uint32_t k = 0; k <= nx; k++) {
        const uint32_t off = (k < nx) ? base[H_XOFF + k] : base[H_FINAL];
        if (off == 0) continue;
        float* a = reinterpret_cast<float*>(dst + off + X_AFF);
        const float ang = 0.31415926535f * dt * __uint_as_float(base[off + X_ROTF]);
        float sn, cs;
        sincosf(ang, &sn, &cs);
        const float a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3];
        a[0] = a0 * cs + a2 * sn;
        a[1] = a1 * cs + a3 * sn;
        a[2] = a2 * cs - a0 * sn;
        a[3] = a3 * cs - a1 * sn;
    }
}

// single dispatch() per point, for parity tests
__global__ void probe_kernel(const uint32_t* prog, int xform, uint32_t n, const float* in, uint32_t* rng,
                             int first_run, float* out) {
    __shared__ uint32_t s_prog[kProgMaxWords];
    for (uint32_t k = threadIdx.x; k < prog[H_WORDS]; k += blockDim.x) s_prog[k] = prog[k];
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t off = (xform < 0) ? s_prog[H_FINAL] : s_prog[H_XOFF + xform];
    Jsf s{rng[4 * i], rng[4 * i + 1], rng[4 * i + 2], rng[4 * i + 3]};
    const XformOut o = eval_xform((uint32_t)__cvta_generic_to_shared(s_prog + off), in[3 * i], in[3 * i + 1],
                                  in[3 * i + 2], first_run != 0, s);
    out[4 * i] = o.x; out[4 * i + 1] = o.y; out[4 * i + 2] = o.c; out[4 * i + 3] = o.op;
    rng[4 * i] = o.rng.a; rng[4 * i + 1] = o.rng.b; rng[4 * i + 2] = o.rng.c; rng[4 * i + 3] = o.rng.d;
}

// ---------------------------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------------------------
size_t chaos_smem(int slots, uint32_t prog_words, uint32_t steps, uint32_t tile_bins, int pipe, uint32_t ranges) {
    return chaos_smem_bytes(slots, prog_words, steps, tile_bins, pipe, ranges);
}

template <int THREADS, int SPT>
static cudaError_t launch_chaos_t(const ChaosArgs& a, uint32_t grid, cudaStream_t st) {
    const size_t smem = chaos_smem_bytes(THREADS * SPT, a.prog_words, a.steps,
                                         a.splat == 3 && a.draw ? a.tile_w * a.tile_h : 0u, 0,
                                         a.splat == 4 && a.draw ? a.ranges : 0u);
    auto kern = chaos_kernel<THREADS, SPT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

bool chaos_shape_supported(int threads, int slots) {
    switch (threads * 8 + slots / threads) {
    case 256 * 8 + 1: case 512 * 8 + 1: case 512 * 8 + 2: case 512 * 8 + 4:
    case 1024 * 8 + 1: case 1024 * 8 + 2: case 1024 * 8 + 4: return slots % threads == 0;
    default: return false;
    }
}

cudaError_t launch_chaos(int threads, int slots, const ChaosArgs& a, uint32_t grid, cudaStream_t st) {
    if (!chaos_shape_supported(threads, slots)) return cudaErrorInvalidValue;
    switch (threads * 8 + slots / threads) {
    case 256 * 8 + 1: return launch_chaos_t<256, 1>(a, grid, st);
    case 512 * 8 + 1: return launch_chaos_t<512, 1>(a, grid, st);
    case 512 * 8 + 2: return launch_chaos_t<512, 2>(a, grid, st);
    case 512 * 8 + 4: return launch_chaos_t<512, 4>(a, grid, st);
    case 1024 * 8 + 1: return launch_chaos_t<1024, 1>(a, grid, st);
    case 1024 * 8 + 2: return launch_chaos_t<1024, 2>(a, grid, st);
    case 1024 * 8 + 4: return launch_chaos_t<1024, 4>(a, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

// the chaos kernel with a cluster CTA's slots (the same shared memory as a specialised one)
static const void* cluster_probe(int local) {
    return local == 256    ? (const void*)chaos_kernel<256, 1>
           : local == 512  ? (const void*)chaos_kernel<512, 1>
           : local == 1024 ? (const void*)chaos_kernel<1024, 1>
                           : (const void*)chaos_kernel<1024, 2>;
}

int chaos_cluster(int slots, uint64_t domains, uint32_t prog_words, uint32_t steps) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    for (int k = 8; k >= 2; k /= 2) {
        const int local = slots / k;  // slots of a CTA, on up to 1024 threads
        if (local < kGroup || domains * (uint64_t)k > (uint64_t)sms) continue;
        const size_t smem = chaos_smem_bytes(local, prog_words, steps);
        const void* f = cluster_probe(local);
        cudaLaunchConfig_t c{};
        c.gridDim = dim3((unsigned)(domains * k));
        c.blockDim = dim3(local < 1024 ? local : 1024);
        c.dynamicSmemBytes = smem;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = k;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        c.attrs = &at;
        c.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&n, f, &c) == cudaSuccess && (uint64_t)n >= domains)
            return k;
        cudaGetLastError();
    }
    return 1;
}

cudaError_t launch_init_rng(uint4* rng, uint64_t n, uint64_t seed, cudaStream_t st) {
    const uint32_t b = 256;
    init_rng_kernel<<<(unsigned)((n + b - 1) / b), b, 0, st>>>(rng, n, seed);
    return cudaGetLastError();
}

cudaError_t launch_shuffle_table(uint16_t* out, uint32_t n, uint32_t count, uint64_t seed, cudaStream_t st,
                                 uint32_t phases) {
    const uint64_t total = (uint64_t)n * count;
    const uint32_t b = 256;
    if (phases >= 3) {
        if (n > kMaxPipeSlots || n % phases) return cudaErrorInvalidValue;
        shuffle_table_pipe_kernel<<<(count + kPipeTableWarps - 1) / kPipeTableWarps, 32 * kPipeTableWarps, 0, st>>>(
            out, n, count, seed, phases);
        return cudaGetLastError();
    }
    shuffle_table_kernel<<<(unsigned)((total + b - 1) / b), b, 0, st>>>(out, n, count, seed);
    return cudaGetLastError();
}

cudaError_t launch_animate(const uint32_t* base, uint32_t words, uint32_t T, float tss, uint32_t* out,
                           uint32_t stride, cudaStream_t st) {
    animate_kernel<<<T, 128, 0, st>>>(base, words, T, tss, out, stride);
    return cudaGetLastError();
}

cudaError_t launch_probe(const uint32_t* prog, int xform, uint32_t n, const float* in, uint32_t* rng, int first_run,
                         float* out, cudaStream_t st) {
    const uint32_t b = 128;
    probe_kernel<<<(n + b - 1) / b, b, 0, st>>>(prog, xform, n, in, rng, first_run, out);
    return cudaGetLastError();
}

}  // namespace rfk
