// Which way a drawing call takes -- the planes, interleaved records, or point lists -- and what it holds on the device,
// without a GPU: the simulation's host code over a fake CUDA runtime whose stream runs when it is synchronised, and
// fake launches that record their arguments and leave what the kernels would.
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <cstdio>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <string>

#include "../../refrakt_gb300/csrc/api.cpp"

// ---- fake runtime: one stream, a queue ----
static std::deque<std::function<void()>> g_queue;
static std::map<void*, size_t> g_live;   // device allocations
static std::map<void*, size_t> g_event;  // operations queued before the event's last record
static size_t g_queued = 0, g_run = 0, g_peak = 0, g_device = (size_t)280 << 30;
static const void* g_fail_memset = nullptr;  // the next clear of this address fails
static size_t live() {
    size_t n = 0;
    for (auto& a : g_live) n += a.second;
    return n;
}
static void enqueue(std::function<void()> f) { g_queue.push_back(std::move(f)); g_queued++; }
static void run_stream(size_t most = ~(size_t)0) {
    for (; most && !g_queue.empty(); most--) {
        auto f = std::move(g_queue.front());
        g_queue.pop_front();
        f();
        g_run++;
    }
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    if (live() + n > g_device) return cudaErrorMemoryAllocation;
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    g_live[*p] = n;
    g_peak = std::max(g_peak, live());
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    run_stream();
    if (p) { munmap(p, g_live.at(p)); g_live.erase(p); }
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = g_device - live(); *t = g_device; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { run_stream(); memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (k == cudaMemcpyDeviceToHost) enqueue([=] { memcpy(d, s, n); });
    else { run_stream(); memcpy(d, s, n); }
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (p == g_fail_memset) { g_fail_memset = nullptr; return cudaErrorInvalidValue; }
    if (n < (1u << 20)) enqueue([=] { memset(p, v, n); });  // (large ones are fresh and zero)
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "a CUDA error"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { run_stream(); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { g_event.erase(e); free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { g_event[(void*)e] = g_queued; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return g_event[(void*)e] <= g_run ? cudaSuccess : cudaErrorNotReady; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.0f; return cudaSuccess; }
}

// ---- fake launches ----
static rfk::ChaosArgs g_last;  // the last drawing launch
static unsigned long long g_hottest = 1, g_points = 1u << 20, g_over = 0;  // what a launch's lists hold
namespace rfk {
size_t chaos_smem(int slots, uint32_t words, uint32_t steps, uint32_t tile, int, uint32_t) { return words * 4 + 4096 + (size_t)slots * 48 + steps * 4 + tile * 20; }
int chaos_cluster(int, uint64_t, uint32_t, uint32_t) { return 1; }
bool chaos_shape_supported(int, int) { return true; }
cudaError_t launch_chaos(int, int, const ChaosArgs& a, uint32_t, cudaStream_t) { if (a.draw) g_last = a; return cudaSuccess; }
cudaError_t launch_spec(const void*, int, int, const ChaosArgs& a, uint32_t, size_t, cudaStream_t) { if (a.draw) g_last = a; return cudaSuccess; }
cudaError_t launch_merge_records(float4*, size_t, float4*, uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_init_rng(uint4*, uint64_t, uint64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_shuffle_table(uint16_t*, uint32_t, uint32_t, uint64_t, cudaStream_t, uint32_t) { return cudaSuccess; }
cudaError_t launch_animate(const uint32_t*, uint32_t, uint32_t, float, uint32_t*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_probe(const uint32_t*, int, uint32_t, const float*, uint32_t*, int, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_density(const float4*, uint32_t, uint32_t, int, int, float, float4*, cudaStream_t) { return cudaSuccess; }
bool density_reads_weights(int, int) { return false; }
void density_weights(int, int, std::vector<float>&) {}
bool density_tonemap_fused(int, int, uint32_t) { return true; }
cudaError_t launch_stats(const float4*, uint32_t, uint32_t, double*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_tonemap(const float4*, uint32_t, uint32_t, uint32_t, float, float, float, float, const double*, float4*, uchar4*, cudaStream_t) { return cudaSuccess; }
int filter_taps(uint32_t, float, int, float*) { return 1; }
cudaError_t launch_tonemap_filter(const float4*, uint32_t, uint32_t, uint32_t, float, int, float, float, float, float, const double*, float4*, uchar4*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_density_tonemap(const float4*, uint32_t, uint32_t, int, int, float, uint32_t, float, float, float, float, float4*, uchar4*, uint8_t*, const float*, double*, float4*, cudaStream_t) { return cudaSuccess; }
cudaError_t scratch_alloc(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t scratch_trim() { return cudaSuccess; }
int spec_kernel(const std::vector<uint32_t>&, int, int, int, const void**, SpecKind, int, int, int, int) { return RF_ERR_UNSUPPORTED; }
std::string spec_source(const std::vector<uint32_t>&, int, int, SpecKind, int, int, int, int) { return ""; }
int spec_compile(const std::string&, std::vector<char>&) { return RF_ERR_UNSUPPORTED; }
bool spec_available(std::string*) { return false; }
cudaError_t launch_ranges(const ChaosArgs&, uint32_t, const RangeScratch[2], RangeState*, unsigned long long* stats, cudaStream_t) {
    const unsigned long long h = g_hottest, n = g_points, o = g_over;
    if (stats) enqueue([=] {
        stats[0] = std::max(stats[0], h);
        stats[1] += n;
        stats[2] += o;
    });
    return cudaSuccess;
}
}  // namespace rfk

#define CHECK(x) do { if (!(x)) { printf("line %d: %s (%s)\n", __LINE__, #x, rf_last_error()); return 1; } } while (0)
enum Route { kPlanes, kRecords, kLists };
static Route route() { return g_last.splat == 4 ? kLists : g_last.rgba_shift ? kRecords : kPlanes; }

struct Scene {
    rf_compiler* c = nullptr;
    rf_flame* f = nullptr;
    rf_sim* s = nullptr;
    float4* bins = nullptr;
    uint32_t* hits = nullptr;
    Scene(uint64_t walkers, uint32_t slots) {
        rf_compiler_create(nullptr, &c);
        const rf_synth_desc sd{RF_SYNTH_SPACEFILL, 0, 3, 0, 0, 8192, 8192};
        rf_flame_synthesize(&sd, c, &f);
        rf_sim_desc d{};
        d.walkers = walkers;
        d.cta_slots = slots;
        d.specialize = -1;
        rf_sim_create(&d, &s);
        cudaMalloc((void**)&bins, ((size_t)1 << 27) * 16);
        cudaMalloc((void**)&hits, ((size_t)1 << 27) * 4);
        rf_warmup(s, f, 3, 0.0f);
    }
    int draw(uint32_t w, uint32_t h, uint32_t passes = 16) { return rf_draw_to_bins(s, f, (float*)bins, hits, w, h, passes, nullptr); }
    ~Scene() {
        rf_sim_destroy(s);
        rf_flame_free(f);
        rf_compiler_destroy(c);
        cudaFree(bins);
        cudaFree(hits);
    }
};

// a call that fails before its launches leaves nothing behind for the next
static int failed_call() {
    Scene t(155648, 1024);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);
    g_fail_memset = t.s->counters + 4;
    CHECK(t.draw(8191, 8192) != RF_OK && !g_fail_memset);
    CHECK(rf_set_bin_layout(t.s, RF_BINS_DIRECT) == RF_OK);
    CHECK(t.draw(640, 360) == RF_OK && route() == kPlanes && g_last.ranges == 0);
    CHECK(rf_set_bin_layout(t.s, RF_BINS_AUTO) == RF_OK);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists && g_last.ranges == 18);
    return 0;
}

// records from the second call on where the call's own points have a hot bin or full lists, and only there: what
// the caller's count plane holds from elsewhere does not matter
static int own_points() {
    for (int k = 0; k < 6; k++) {
        Scene t(155648, 1024);
        const uint32_t passes = k == 4 || k == 5 ? 1024 : 16;  // 1024: four launches
        g_hottest = k == 1 ? 1024 : k == 4 ? 1023 : k == 5 ? 1024 : 1;
        g_over = k == 2 ? 155648 * 16 / 8 + 1 : k == 3 ? 155648 * 16 / 8 : 0;
        memset(t.hits, 0, 1 << 20);
        t.hits[77] = k == 0 ? 4000000000u : 0u;  // another program's points
        CHECK(t.draw(8192, 8192, passes) == RF_OK && route() == kLists);
        cudaStreamSynchronize(nullptr);
        CHECK(t.draw(8192, 8192, passes) == RF_OK && route() == (k == 1 || k == 2 || k == 5 ? kRecords : kLists));
    }
    return 0;
}

// a verdict is one grid's and one view's, and is not taken before its statistics have arrived
static int own_view() {
    Scene t(155648, 1024);
    g_over = 0;
    g_hottest = 1 << 19;
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);  // nothing has arrived
    cudaStreamSynchronize(nullptr);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kRecords);
    // another grid, asked for and drawn before the stream gets anywhere: the first grid's figures are not its own
    g_hottest = 1;
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    cudaStreamSynchronize(nullptr);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    // a view with a hot bin, after one without
    const float center[2] = {0.1f, 0.2f};
    g_hottest = 1 << 19;
    CHECK(rf_flame_set_view(t.f, center, 5000.0f, 0.0f) == RF_OK);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    cudaStreamSynchronize(nullptr);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kRecords);
    // and one without, after one with: the hot view's copy lands while the new view's is behind it
    CHECK(rf_flame_set_view(t.f, center, 4000.0f, 0.0f) == RF_OK);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);  // hot, not arrived
    g_hottest = 1;
    CHECK(rf_flame_set_view(t.f, center, 3000.0f, 0.0f) == RF_OK);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    run_stream(g_queue.size() - 1);  // all but the new view's copy
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    cudaStreamSynchronize(nullptr);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists);
    return 0;
}

// the lists take what the records would or an eighth of the free memory, and nothing when records take over
static int memory() {
    const size_t gb = (size_t)1 << 30, records = (size_t)32 << 26;
    g_over = 0;
    g_hottest = 1;
    for (size_t free : {3 * gb, 8 * gb, 30 * gb, 200 * gb}) {
        g_device = (size_t)280 << 30;
        Scene t(622592, 4096);
        const size_t held = live();
        g_device = held + free;
        for (int k = 0; k < 4; k++) {  // 159 M points a launch: 5.1e9 bytes of lists at four times an even spread, 1.6 at 1.25
            CHECK(t.draw(8192, 8192, 512) == RF_OK && route() == kLists);
            CHECK(live() - held <= std::max(free / 8, records));
        }
        CHECK(free < 200 * gb || live() - held > (size_t)5100000000);
    }
    g_device = (size_t)280 << 30;
    Scene t(155648, 1024);
    const size_t before = live();
    for (int turn = 0; turn < 7; turn++) {
        const float center[2] = {0.01f * turn, 0.0f};
        CHECK(rf_flame_set_view(t.f, center, 4000.0f, 0.0f) == RF_OK);
        g_hottest = 1 << 19;
        CHECK(t.draw(8192, 8192) == RF_OK);
        CHECK(route() == (turn < 4 ? kLists : kRecords));  // views that turn and turn again stay with records
        cudaStreamSynchronize(nullptr);
        CHECK(t.draw(8192, 8192) == RF_OK && route() == kRecords);
        CHECK(live() == before + records);
    }
    CHECK(rf_flame_set_xform_value(t.f, 0, "color", 0.7f) == RF_OK && rf_warmup(t.s, t.f, 3, 0.0f) == RF_OK);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);  // another genome
    return 0;
}

int main(int argc, char** argv) {
    const std::string name = argc > 1 ? argv[1] : "";
    const int rc = name == "failed_call" ? failed_call() : name == "own_points" ? own_points() : name == "own_view" ? own_view() : name == "memory" ? memory() : 2;
    if (rc == 0) printf("OK\n");
    return rc;
}
