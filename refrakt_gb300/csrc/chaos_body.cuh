// The chaos game of one CTA (the body of chaos_kernel, kernels.cu, and of the genome-specialised
// kernels compiled at run time, specialize.cpp), parameterised by the xform evaluator:
// `Eval::apply<FINAL>(prog, word, x, y, c, op, first_run, rng)` applies the xform of an xform_word.
// InterpEval interprets the compiled genome program (variations.cuh); a specialised evaluator is
// generated per genome structure (specialize.cpp).
//
// The reference runs one GLSL invocation per walker per pass and ping-pongs every walker
// through memory between passes (shaders/flame.glsl:41-90, src/flame.cpp:228-330).  Here one
// CTA owns a block of walker slots (the mixing domain) for L consecutive passes: the genome is
// staged once in shared memory, the slots' walkers and JSF32 states stay in shared memory, and
// between passes the walkers are permuted among the CTA's slots through a double-buffered
// shared-memory exchange (the walker shuffle).  At each launch boundary every walker is gathered
// from HBM through a keyed permutation of its temporal sample, so walkers also mix across CTAs.
//
// Per slot and pass the order of RNG draws is the reference's: the first slot of each 256-slot
// group draws the group's xform id (flame.glsl:51-53), then the first-pass jitter (:64), the
// variations in codegen order, the first-pass colour (variation_table.cpp:242) and, when
// drawing, the final xform (flame.cpp:23).
#pragma once

#include "chaos_args.h"
#include "splat.cuh"
#include "variations.cuh"

namespace rfk {

// A group's drawn xform as the slots read it: id | (its block's word offset) << 8.
__device__ __forceinline__ uint32_t xform_word(const uint32_t* prog, int xi) {
    return (uint32_t)xi | (prog[H_XOFF + xi] << 8);
}

struct InterpEval {
    static constexpr bool kFinal = true;
    template <bool FINAL>
    static __device__ __forceinline__ void apply(const uint32_t* prog, uint32_t word, float& x, float& y, float& c,
                                                 float& op, bool first_run, Jsf& rng) {
        const uint32_t blk = (uint32_t)__cvta_generic_to_shared(prog) + 4u * (word >> 8);
        const XformOut o = eval_xform(blk, x, y, c, first_run, rng);
        x = o.x; y = o.y; c = o.c; op = o.op;
        rng = o.rng;
    }
};

// The final xform on a drawn copy of the walker; op becomes the point's opacity.
template <class Eval>
__device__ __forceinline__ void final_xform(const uint32_t* prog, uint32_t final_off, float& x, float& y, float& c,
                                            float& op, Jsf& rng) {
    float o;
    Eval::template apply<true>(prog, final_off << 8, x, y, c, o, false, rng);
    op = o * op;
}

// The slot a thread serves in phase k of a pass: phase k covers slots [k * THREADS, (k + 1) *
// THREADS), and warps are permuted per phase (warp w serves warp w ^ k's 32 slots), so the 256-slot
// groups' first slots fall to SPT * THREADS / 256 different warps, one per warp: the group xform
// draws at the start of a pass run in parallel instead of SPT after another.
template <int THREADS>
__device__ __forceinline__ uint32_t phase_slot(int k, int tid) {
    return (uint32_t)(k * THREADS + (tid ^ (32 * k)));
}
// the phase in which thread tid serves a group's first slot, or -1
template <int THREADS, int SPT>
__device__ __forceinline__ int draw_phase(int tid) {
    const int k = (tid % kGroup) >> 5;
    return ((tid & 31) == 0 && k < SPT) ? k : -1;
}

// Shared memory of a chaos CTA (dynamic, in this order):
//   program words (prog_words), palette float4[256], walker exchange float4 [2][SLOTS],
//   JSF32 states uint4[SLOTS], group xform ids int[2][SLOTS/256], per-pass permutation ids
//   uint32[steps], (8-byte aligned) the pipelined exchange's two mbarriers; with the tile splat
//   (16-byte aligned) the tile's float4 RGBA sums and uint32 counts; with the list splat (16-byte
//   aligned) a count per bin range
__host__ __device__ inline size_t chaos_smem_bytes(int slots, uint32_t prog_words, uint32_t steps,
                                                   uint32_t tile_bins = 0, int pipe = 0, uint32_t ranges = 0) {
    size_t b = ((size_t)prog_words * 4 + 15) & ~(size_t)15;
    b += 256 * 16;
    b += (size_t)2 * slots * 16;
    b += (size_t)slots * 16;
    b += (size_t)2 * (slots / kGroup) * 4;
    b += (size_t)steps * 4;
    if (pipe) b = ((b + 7) & ~(size_t)7) + 16;
    if (tile_bins) b = ((b + 15) & ~(size_t)15) + (size_t)tile_bins * 20;
    if (ranges) b = ((b + 15) & ~(size_t)15) + (size_t)ranges * 4;
    return b;
}

// The pipelined walker exchange's two CTA-wide mbarriers: [0] completes when every thread has
// finished the first SPT-1 phases of a pass, [1] when every thread has finished the pass.
__device__ __forceinline__ uint32_t xbar_addr(const uint64_t* b) { return (uint32_t)__cvta_generic_to_shared(b); }
__device__ __forceinline__ void xbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(xbar_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void xbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(xbar_addr(b)) : "memory");
}
// waits (bounded) for the completion of the barrier's phase of the given parity: 2^16 tries, each
// suspending the thread for at most 16 us (the suspend-time hint), so about a second at most;
// false when the wait ran out
__device__ __forceinline__ bool xbar_wait(uint64_t* b, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 16); i++) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(xbar_addr(b)), "r"(parity), "r"(16384u)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The cluster exchange: a mixing domain spread over the CTAs of a thread-block cluster, each with its
// share of the slots in its own shared memory.  A pass's walkers are read from the CTA that holds them
// (distributed shared memory); one cluster barrier per pass replaces the CTA's.  (Not the .aligned forms: they
// follow code in which lanes part -- the evaluator's branches, the walker reset, the group's draw -- and those forms
// are undefined unless the warp has met again.  The 65,536 walkers of the CLUSTER comment below: no difference.)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ float4 cluster_load(const float4* local, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}

// One CTA of THREADS threads owns SLOTS = THREADS * SPT walker slots — the walker shuffle's mixing
// domain — for the launch's passes.  Every slot's walker and JSF32 state live in shared memory;
// each thread serves SPT slots per pass (phase_slot(k, tid), in SPT different 256-slot groups, so
// a warp's work per pass averages over SPT xforms).  64 registers per thread:
// 1024 threads x 1, 512 x 2 or 256 x 4 CTAs per SM.
// SPLAT >= 0 fixes the splat strategy at compile time (0 global, 1 warp-aggregated, 2 adaptive),
// so the hot loop carries only that one; -1 dispatches on A.splat.  RESET >= 0 likewise fixes
// the walker reset of flame.glsl:68 (reset_bad_walker); -1 reads A.reset.
//
// PIPE = 1 (SPT >= 3) replaces the pass barrier by the pipelined exchange.  The shuffle table's
// permutations (shuffle_table_pipe_kernel) send the first phase's slots no walker of the previous
// pass's last phase and the last phase's slots no walker of its first phase.  So a warp starts the
// next pass as soon as every warp has finished the first SPT-1 phases of this one (mbarrier 0:
// the first phase's sources are written, and the first phase's slots — which it overwrites — are
// no longer read), and waits for the whole previous pass (mbarrier 1) only before its second
// phase: the slowest warps' last phase overlaps the others' next pass, with the walkers still
// double-buffered.  A group's xform for pass s + 1 is drawn right after its first slot's pass-s
// evaluation (the same point of that slot's RNG stream) into the other xform-id buffer.
//
// CLUSTER = K > 1 spreads a mixing domain over the K CTAs of a cluster (SLOTS = its slots / K), for
// simulations whose domains are fewer than the SMs: with one CTA per domain the others idle.  The
// arrival on the pass's cluster barrier comes after the last walker's store and the group's xform draw (as
// PIPE draws it: the next pass reads both behind the barrier), the wait before the next pass's first
// read, so the splat alone passes under it.  What is left is one warp's chain per pass: 65,536 walkers of the three-xform genome in 2048-slot domains take
// 3.9 us per pass on 32 CTAs and 2.7 us on 128 (16.6 -> 24.0 Gpoints/s), in 4096-slot ones 6.3 us on 16
// and 4.4 us on 128.
template <int THREADS, int SPT, class Eval, int SPLAT = -1, int RESET = -1, int PIPE = 0, int CLUSTER = 1>
__device__ __forceinline__ void chaos_body(const ChaosArgs& A) {
    static_assert(!PIPE || SPT >= 3, "the pipelined exchange needs three phases");
    static_assert(!PIPE || CLUSTER == 1, "one exchange or the other");
    constexpr uint32_t SLOTS = (uint32_t)THREADS * SPT;       // of this CTA
    constexpr uint32_t DOMAIN_SLOTS = SLOTS * CLUSTER;        // of the mixing domain
    constexpr int G = SLOTS / kGroup;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_prog = reinterpret_cast<uint32_t*>(smem);
    float4* s_pal = reinterpret_cast<float4*>(smem + (((size_t)A.prog_words * 4 + 15) & ~(size_t)15));
    float4* s_w = s_pal + 256;
    uint4* s_rng = reinterpret_cast<uint4*>(s_w + 2 * SLOTS);
    uint32_t* s_xid = reinterpret_cast<uint32_t*>(s_rng + SLOTS);
    uint32_t* s_perm = reinterpret_cast<uint32_t*>(s_xid + 2 * G);
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(((unsigned long long)(s_perm + A.steps) + 7) & ~7ull);
    // the tile splat's shared-memory histogram (splat 3)
    const bool tiled = SPLAT == 3 || (SPLAT < 0 && A.splat == 3);
    const uint32_t tile_bins = tiled && A.draw ? A.tile_w * A.tile_h : 0u;
    TileTarget tt{nullptr, nullptr};
    if (tile_bins) {
        tt.rgba = reinterpret_cast<float4*>(
            smem + ((chaos_smem_bytes(SLOTS, A.prog_words, A.steps, 0, PIPE) + 15) & ~(size_t)15));
        tt.count = reinterpret_cast<uint32_t*>(tt.rgba + tile_bins);
    }

    const bool listed = SPLAT == 4 || (SPLAT < 0 && A.splat == 4);
    const uint32_t ranges = listed && A.draw ? A.ranges : 0u;
    uint32_t* s_list = reinterpret_cast<uint32_t*>(smem + ((chaos_smem_bytes(SLOTS, A.prog_words, A.steps, 0, PIPE) + 15) & ~(size_t)15));

    const int tid = threadIdx.x;
    for (uint32_t i = tid; i < ranges; i += THREADS) s_list[i] = 0u;
    for (uint32_t i = tid; i < tile_bins; i += THREADS) {
        tt.rgba[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        tt.count[i] = 0u;
    }
    const uint32_t chunk = blockIdx.x / CLUSTER;  // mixing domain
    const uint32_t rank = blockIdx.x % CLUSTER;   // of this CTA in it
    const uint32_t ts = chunk / A.chunks_per_ts;
    const uint32_t slot0 = rank * SLOTS;          // first slot within the mixing domain
    const uint32_t gid0 = (chunk - ts * A.chunks_per_ts) * DOMAIN_SLOTS + slot0;  // and within the temporal sample
    const size_t ts_base = (size_t)ts * A.ppts;

    if (PIPE && tid == 0) {
        xbar_init(s_bar + 0, THREADS);
        xbar_init(s_bar + 1, THREADS);
    }
    const uint32_t* prog = A.progs + (size_t)ts * A.prog_stride;
    for (uint32_t i = tid; i < A.prog_words; i += THREADS) s_prog[i] = prog[i];
    if (A.draw)
        for (int i = tid; i < 256; i += THREADS) s_pal[i] = A.palette[i];
    for (uint32_t s = tid; s < A.steps; s += THREADS)
        s_perm[s] = (uint32_t)(derive_key(A.seed, (uint64_t)A.pass0 + s, chunk, TAG_LOCAL) % A.table_size);

    // JSF32 states, and every walker gathered through a keyed permutation of its temporal
    // sample (pass 0 of a warmup reads the start points instead, flame.glsl:58-61)
    const uint64_t gkey = derive_key(A.seed, A.pass0, ts, TAG_GLOBAL);
    for (int k = 0; k < SPT; k++) {
        const uint32_t ls = phase_slot<THREADS>(k, tid);
        s_rng[ls] = A.rng[ts_base + gid0 + ls];
        const uint32_t src = feistel(gid0 + ls, A.ppts, gkey);
        float4 w;
        if (A.first_run) {
            sample_point(src, A.ppts, w.x, w.y);
            w.z = 0.0f;
            w.w = 0.0f;
        } else {
            w = A.walk_in[ts_base + src];
        }
        s_w[ls] = w;
    }

    const uint32_t foff = s_prog[H_FINAL];
    const bool has_final = A.draw && foff != 0;
    const int dphase = draw_phase<THREADS, SPT>(tid);
    const float W = (float)A.W, H = (float)A.H;
    const bool reset = RESET >= 0 ? RESET != 0 : A.reset != 0;
    uint32_t drawn = 0, emitted = 0;
    // flame.glsl:51-53: the first slot of each 256-slot group draws the group's xform for pass s
    // from its own RNG stream (the pipelined and cluster exchanges draw inside the pass loop instead)
    auto draw_group_xform = [&](uint32_t s, uint32_t ls, Jsf& rng) {
        const int xi = select_xform(s_prog, randf(rng));
        s_xid[(s & 1) * G + ls / kGroup] = xform_word(s_prog, xi);
        if (A.trace && A.pass0 + s < A.trace_passes)
            A.trace[(size_t)(A.pass0 + s) * A.n_groups + (ts_base + gid0 + ls) / kGroup] = (uint8_t)xi;
    };
    if ((PIPE || CLUSTER > 1) && dphase >= 0) {
        const uint32_t ls = phase_slot<THREADS>(dphase, tid);
        const uint4 r4 = s_rng[ls];
        Jsf rng{r4.x, r4.y, r4.z, r4.w};
        draw_group_xform(0, ls, rng);
        s_rng[ls] = make_uint4(rng.a, rng.b, rng.c, rng.d);
    }
    __syncthreads();
    if (CLUSTER > 1) cluster_arrive();
    // PIPE: false after a wait ran out — the thread counts it (the host reports RF_ERR_TIMEOUT)
    // and waits no more, so the launch still ends
    bool synced = true;
    constexpr bool kAhead = CLUSTER > 1 && SPT == 1;
    uint32_t ahead[SPT];  // this pass's sources
    if (kAhead)
        for (int k = 0; k < SPT; k++) ahead[k] = slot0 + phase_slot<THREADS>(k, tid);

    for (uint32_t s = 0; s < A.steps; s++) {
        const int buf = s & 1;
        // this pass's sources in the exchange buffer (identity on the gather pass)
        uint32_t src[SPT];
#pragma unroll
        for (int k = 0; k < SPT; k++) {
            if (kAhead) src[k] = ahead[k];
            else src[k] = (s == 0) ? slot0 + phase_slot<THREADS>(k, tid)
                                   : (uint32_t)A.table[(size_t)s_perm[s] * DOMAIN_SLOTS + slot0 + phase_slot<THREADS>(k, tid)];
        }
        if (CLUSTER > 1) {
            cluster_wait();
            // the next pass's sources, a pass ahead: with a few warps per SM their L2 latency is not hidden
#pragma unroll
            for (int k = 0; k < SPT; k++)
                if (kAhead && s + 1 < A.steps) ahead[k] = A.table[(size_t)s_perm[s + 1] * DOMAIN_SLOTS + slot0 + phase_slot<THREADS>(k, tid)];
        } else if (!PIPE) {
            if (dphase >= 0) {
                const uint32_t ls = phase_slot<THREADS>(dphase, tid);
                const uint4 r4 = s_rng[ls];
                Jsf rng{r4.x, r4.y, r4.z, r4.w};
                draw_group_xform(s, ls, rng);
                s_rng[ls] = make_uint4(rng.a, rng.b, rng.c, rng.d);
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int k = 0; k < SPT; k++) {
            const uint32_t ls = phase_slot<THREADS>(k, tid);
            uint32_t j = src[0];
#pragma unroll
            for (int q = 1; q < SPT; q++)
                if (q == k) j = src[q];
            // PIPE: the first phase reads walkers of the previous pass's first SPT-1 phases, the
            // others any of its walkers
            if (PIPE && synced && s > 0 && k < 2 && !xbar_wait(s_bar + k, (s - 1) & 1)) {
                synced = false;
                atomicAdd(A.counters + 3, 1ull);
            }
            const float4 v = CLUSTER > 1 ? cluster_load(s_w + buf * SLOTS + j % SLOTS, j / SLOTS) : s_w[buf * SLOTS + j];
            float x = v.x, y = v.y, c = v.z;
            const uint4 r4 = s_rng[ls];
            Jsf rng{r4.x, r4.y, r4.z, r4.w};
            const uint32_t xw = s_xid[buf * G + ls / kGroup];
            const bool first = A.first_run && s == 0;
            if (first) {  // flame.glsl:64: xy += randf() * .1 * PI * 2.0 * sincos(sqrt(randf()))
                const float u1 = randf(rng);
                const float u2 = randf(rng);
                const float amp = __fmul_rn(__fmul_rn(__fmul_rn(u1, 0.1f), kPI), 2.0f);
                float sn, cs;
                jitter_sincos(sqrtf(u2), sn, cs);
                x = __fadd_rn(x, __fmul_rn(amp, sn));
                y = __fadd_rn(y, __fmul_rn(amp, cs));
            }
            // the xform: the walker's next state; then (when drawing) the final xform on the copy that is drawn
            float op = 0.0f;
            Eval::template apply<false>(s_prog, xw, x, y, c, op, first, rng);
            if (reset) reset_bad_walker(x, y, op, rng);  // flame.glsl:68, before pos_out
            s_w[(buf ^ 1) * SLOTS + ls] = make_float4(x, y, c, 0.0f);
            if (Eval::kFinal && has_final) final_xform<Eval>(s_prog, foff, x, y, c, op, rng);
            // the group's xform for the next pass, at the point of the slot's stream where the
            // pass-barrier form draws it
            if ((PIPE || CLUSTER > 1) && k == dphase && s + 1 < A.steps) draw_group_xform(s + 1, ls, rng);
            s_rng[ls] = make_uint4(rng.a, rng.b, rng.c, rng.d);
            if (PIPE && k >= SPT - 2) xbar_arrive(s_bar + (k - (SPT - 2)));
            if (CLUSTER > 1 && k == SPT - 1) cluster_arrive();
            if (A.draw) {
                if (op > 0.0f) emitted++;
                const float px = fmaf(A.ss[0], x, fmaf(A.ss[2], y, A.ss[4]));
                const float py = fmaf(A.ss[1], x, fmaf(A.ss[3], y, A.ss[5]));
                uint32_t bin = kNoBin, local = kNoBin, pi = 0;
                float4 val = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (px >= 0.0f && py >= 0.0f && px < W && py < H && op > 0.0f) {
                    const uint32_t bx = (uint32_t)px, by = (uint32_t)py;
                    const uint32_t row = A.H - 1 - by;  // flame.glsl:84 row flip; W*H < 2^32 - 1
                    bin = row * A.W + bx;
                    if (tile_bins && bx - A.tile_x0 < A.tile_w && row - A.tile_y0 < A.tile_h)
                        local = (row - A.tile_y0) * A.tile_w + (bx - A.tile_x0);
                    pi = palette_index(c);
                    if (SPLAT != 4) {
                        const float4 col = s_pal[pi];
                        val = make_float4(col.x, col.y, col.z, op);
                    }
                    drawn++;
                }
                const BinTarget t{A.bins, A.hits, A.rgba_shift, A.count_shift};
                if constexpr (SPLAT == 0) {
                    splat_global(t, bin, val);
                } else if constexpr (SPLAT == 1) {
                    splat_warp(t, bin, val);
                } else if constexpr (SPLAT == 2) {
                    splat_adaptive(t, bin, val);
                } else if constexpr (SPLAT == 3) {
                    splat_tile(t, tt, bin, local, val);
                } else if constexpr (SPLAT == 4) {
                    splat_list(A, t, s_list, s_pal, bin, pi, op);
                } else {
                    if (A.splat == 1) splat_warp(t, bin, val);
                    else if (A.splat == 2) splat_adaptive(t, bin, val);
                    else if (A.splat == 3) splat_tile(t, tt, bin, local, val);
                    else if (A.splat == 4) splat_list(A, t, s_list, s_pal, bin, pi, op);
                    else splat_global(t, bin, val);
                }
            }
        }
    }
    if (CLUSTER > 1) cluster_wait();  // no CTA leaves while another reads its walkers
    // the tile's non-empty bins into the histogram, once per launch
    if (tile_bins) {
        __syncthreads();
        const BinTarget t{A.bins, A.hits, A.rgba_shift, A.count_shift};
        for (uint32_t i = tid; i < tile_bins; i += THREADS) {
            const uint32_t n = tt.count[i];
            if (!n) continue;
            const uint32_t row = A.tile_y0 + i / A.tile_w, col = A.tile_x0 + i % A.tile_w;
            const float4 v = tt.rgba[i];
            red_add_f32x4(t.at_rgba(row * A.W + col), v.x, v.y, v.z, v.w);
            if (t.count) red_add_u32x1(t.at_count(row * A.W + col), n);
        }
    }
    if (ranges) {
        __syncthreads();
        for (uint32_t i = tid; i < ranges; i += THREADS) A.list_n[blockIdx.x * ranges + i] = s_list[i];
    }
    // each slot's final walker and state were written by the thread that owns the slot
    const int out_buf = A.steps & 1;
    for (int k = 0; k < SPT; k++) {
        const uint32_t ls = phase_slot<THREADS>(k, tid);
        A.walk_out[ts_base + gid0 + ls] = s_w[out_buf * SLOTS + ls];
        A.rng[ts_base + gid0 + ls] = s_rng[ls];
    }

    if (A.draw) {
        const uint32_t d = __reduce_add_sync(0xffffffffu, drawn);
        const uint32_t e = __reduce_add_sync(0xffffffffu, emitted);
        if ((tid & 31) == 0) {
            atomicAdd(A.counters + 0, (unsigned long long)d);
            atomicAdd(A.counters + 1, (unsigned long long)e);
        }
    }
    if (tid == 0) atomicAdd(A.counters + 2, (unsigned long long)SLOTS * A.steps);
}

}  // namespace rfk
