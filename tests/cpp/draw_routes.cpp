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
static std::map<void*, std::pair<size_t, float>> g_event;  // operations queued before its last record, device time then
static float g_clock = 0, g_lists_ms = 1, g_records_ms = 2;  // device time; what a launch takes with lists and with records
static bool g_capturing = false, g_fail_launch = false;
static size_t g_queued = 0, g_run = 0, g_peak = 0, g_device = (size_t)280 << 30;
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
    if (g_capturing) return cudaErrorStreamCaptureUnsupported;
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
    if (n < (1u << 20)) enqueue([=] { memset(p, v, n); });  // (large ones are fresh and zero)
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "a CUDA error"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { run_stream(); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { g_event.erase(e); free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { g_event[(void*)e] = {g_queued, g_clock}; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return g_event[(void*)e].first <= g_run ? cudaSuccess : cudaErrorNotReady; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t a, cudaEvent_t b) { *t = g_event[(void*)b].second - g_event[(void*)a].second; return cudaSuccess; }
}

// ---- fake launches ----
static rfk::ChaosArgs g_last;  // the last drawing launch
static cudaError_t launched(const rfk::ChaosArgs& a) {
    if (!a.draw) return cudaSuccess;
    if (g_fail_launch) { g_fail_launch = false; return cudaErrorLaunchOutOfResources; }
    g_last = a;
    g_clock += a.splat == 4 ? g_lists_ms : g_records_ms;
    enqueue([] {});
    return cudaSuccess;
}
namespace rfk {
size_t chaos_smem(int slots, uint32_t words, uint32_t steps, uint32_t tile, int, uint32_t) { return words * 4 + 4096 + (size_t)slots * 48 + steps * 4 + tile * 20; }
int chaos_cluster(int, uint64_t, uint32_t, uint32_t) { return 1; }
bool chaos_shape_supported(int, int) { return true; }
cudaError_t launch_chaos(int, int, const ChaosArgs& a, uint32_t, cudaStream_t) { return launched(a); }
cudaError_t launch_spec(const void*, int, int, const ChaosArgs& a, uint32_t, size_t, cudaStream_t) { return launched(a); }
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
cudaError_t launch_ranges(const ChaosArgs&, uint32_t, const RangeScratch[2], RangeState*, cudaStream_t) { return cudaSuccess; }
cudaError_t load_draw_kernels() { return cudaSuccess; }
}  // namespace rfk

#define CHECK(x) do { if (!(x)) { printf("line %d: %s (route %d, %zu bytes; %s)\n", __LINE__, #x, g_last.splat == 4 ? 2 : g_last.rgba_shift != 0, live(), rf_last_error()); return 1; } } while (0)
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

// a call that fails leaves nothing behind for the next
static int failed_call() {
    Scene t(155648, 1024);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);
    g_fail_launch = true;
    CHECK(t.draw(8191, 8192) != RF_OK && !g_fail_launch);
    CHECK(rf_set_bin_layout(t.s, RF_BINS_DIRECT) == RF_OK);
    CHECK(t.draw(640, 360) == RF_OK && route() == kPlanes && g_last.ranges == 0);
    CHECK(rf_set_bin_layout(t.s, RF_BINS_AUTO) == RF_OK);
    CHECK(t.draw(8192, 4608) == RF_OK && route() == kLists && g_last.ranges == 18);
    return 0;
}

// one call of each form, lists first where a launch has few points per bin, then the faster form; the choice waits for
// the second call's end and for a call of the first one's length
static int faster_form() {
    for (int k = 0; k < 4; k++) {
        const bool lists_win = k & 1, many = k & 2;
        g_lists_ms = lists_win ? 1 : 3;
        Scene t(many ? 2490368 : 155648, many ? 4096 : 1024);
        const uint32_t passes = many ? 64 : 16;  // 159 M points a launch on 67 M bins, or 2.5 M
        const Route first = many ? kRecords : kLists, second = many ? kLists : kRecords;
        CHECK(t.draw(8192, 8192, passes) == RF_OK && route() == first);
        CHECK(t.draw(8192, 8192, passes / 2) == RF_OK && route() == first);  // timed in its place: the lengths differ
        CHECK(t.draw(8192, 8192, passes / 2) == RF_OK && route() == second);
        CHECK(t.draw(8192, 8192, passes / 2) == RF_OK && route() == first);  // the second has not finished
        cudaStreamSynchronize(nullptr);
        for (int n = 0; n < 3; n++) CHECK(t.draw(8192, 8192, passes) == RF_OK && route() == (lists_win ? kLists : kRecords));
        // small grids and a layout that is asked for have no choice
        CHECK(t.draw(4096, 4096) == RF_OK && route() == kRecords);
        CHECK(t.draw(640, 360) == RF_OK && route() == kPlanes);
        CHECK(rf_set_bin_layout(t.s, RF_BINS_INTERLEAVED) == RF_OK && t.draw(8192, 8192) == RF_OK && route() == kRecords);
    }
    return 0;
}

// a choice is one genome's, grid's and view's: another's calls are timed afresh, after 16 calls at most
static int own_view() {
    Scene t(155648, 1024);
    const auto settle = [&](uint32_t h) {  // two timed calls and the choice
        for (int n = 0; n < 2; n++) if (t.draw(8192, h)) return kPlanes;
        cudaStreamSynchronize(nullptr);
        return t.draw(8192, h) ? kPlanes : route();
    };
    g_lists_ms = 1;
    CHECK(settle(8192) == kLists);
    g_lists_ms = 3;
    for (int n = 0; n < 13; n++) CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);
    const float center[2] = {0.1f, 0.2f};
    CHECK(rf_flame_set_view(t.f, center, 5000.0f, 0.0f) == RF_OK);
    for (int n = 0; n < 2; n++) CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);  // the old choice stands
    CHECK(settle(8192) == kRecords);
    for (int n = 0; n < 20; n++) CHECK(t.draw(8192, 8192) == RF_OK && route() == kRecords);
    g_lists_ms = 1;
    CHECK(settle(4608) == kLists);  // another grid
    for (int n = 0; n < 20; n++) CHECK(t.draw(8192, 4608) == RF_OK);
    g_lists_ms = 3;
    CHECK(rf_flame_set_xform_value(t.f, 0, "color", 0.7f) == RF_OK && rf_warmup(t.s, t.f, 3, 0.0f) == RF_OK);
    CHECK(settle(4608) == kRecords);  // another genome
    // a new view with every call: one form throughout, nothing is allocated in turn
    const size_t held = live();
    for (int n = 0; n < 40; n++) {
        CHECK(rf_flame_set_view(t.f, center, 4000.0f + n, 0.0f) == RF_OK);
        CHECK(t.draw(8192, 4608) == RF_OK && route() == kRecords && live() == held);
    }
    return 0;
}

// the lists take what the records would or an eighth of the free memory, the chosen form's memory comes in the place of
// the other's, and a form without memory leaves the call to the other
static int memory() {
    const size_t gb = (size_t)1 << 30, records = (size_t)32 << 26;
    g_lists_ms = 1;
    for (size_t free : {3 * gb, 8 * gb, 30 * gb, 200 * gb}) {
        g_device = (size_t)280 << 30;
        Scene t(622592, 4096);
        const size_t held = live();
        g_device = held + free;
        for (int k = 0; k < 4; k++) {  // 80 M points a launch: 2.5e9 bytes of lists at four times an even spread, 0.8 at 1.25
            g_peak = 0;
            CHECK(t.draw(8192, 8192, 128) == RF_OK && route() == (k == 1 ? kRecords : kLists));
            CHECK(live() - held <= std::max(free / 8, records) && g_peak <= held + std::max(free / 8, records));
            cudaStreamSynchronize(nullptr);
        }
        CHECK(free < 30 * gb || live() - held > (size_t)2500000000);
    }
    g_lists_ms = 3;
    for (size_t free : {16 * gb, gb, gb / 8}) {  // records do not fit in 1 GB; lists of 2.5 M points take 0.2 GB
        g_device = (size_t)280 << 30;
        Scene t(155648, 1024);
        const size_t held = live();
        g_device = held + free;
        for (int k = 0; k < 4; k++) {
            const int rc = t.draw(8192, 8192);
            if (free == gb / 8) CHECK(rc == RF_ERR_CUDA);
            else CHECK(rc == RF_OK && route() == (free == gb || k == 0 ? kLists : kRecords));
            cudaStreamSynchronize(nullptr);
        }
        if (free == 16 * gb) CHECK(live() == held + records);
    }
    g_device = (size_t)280 << 30;
    return 0;
}

// a captured call allocates and frees nothing, and what its graph holds stays
static int captured() {
    g_lists_ms = 1;
    Scene t(155648, 1024);
    const auto graph = [&](uint32_t h) { g_capturing = true; const int rc = t.draw(8192, h); g_capturing = false; return rc; };
    CHECK(graph(8192) == RF_OK && route() == kPlanes);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists);
    CHECK(graph(8192) == RF_OK && route() == kPlanes);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kRecords);
    CHECK(graph(4608) == RF_OK && route() == kRecords);
    float4* const rec = t.s->rec;
    cudaStreamSynchronize(nullptr);
    CHECK(t.draw(8192, 8192) == RF_OK && route() == kLists && t.s->rec == rec && g_live.count(rec));
    CHECK(graph(8192) == RF_OK && route() == kRecords);
    return 0;
}

int main(int argc, char** argv) {
    const std::string name = argc > 1 ? argv[1] : "";
    const int rc = name == "failed_call" ? failed_call() : name == "faster_form" ? faster_form() : name == "own_view" ? own_view() : name == "memory" ? memory() : name == "captured" ? captured() : 2;
    if (rc == 0) printf("OK\n");
    return rc;
}
