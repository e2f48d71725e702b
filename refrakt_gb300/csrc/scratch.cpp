// Stream-ordered scratch of the image passes, from one memory pool per device.
//
// The device's default pool gives its free memory back at every synchronisation (release threshold
// 0, and the pool is the process's: not this library's to change), so a frame loop that waits for
// each image pays for mapping its scratch again in every call: density_tonemap of 640 x 360 bins took
// 243 us after a synchronisation and 84 us without one.  This pool keeps up to kScratchKeep bytes --
// the radius plane of a 67-million-bin grid -- and gives them back when a simulation, batch or denoiser
// is destroyed, or at rf_release_scratch.  Pools order their memory by stream, so calls on several streams and threads share it
// safely.  During stream capture the allocation becomes a node of the graph, as before, from the
// default pool.
#include "scratch.h"

#include <mutex>

namespace rfk {

namespace {

constexpr size_t kScratchKeep = (size_t)64 << 20;
constexpr int kMaxDevices = 64;

std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};

// the current device's pool, null where it cannot be made
cudaMemPool_t pool(bool create) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_pool[dev] && create) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) == cudaSuccess) {
            unsigned long long keep = kScratchKeep;
            cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
            g_pool[dev] = p;
        } else {
            cudaGetLastError();
        }
    }
    return g_pool[dev];
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
    cudaMemPool_t mp = capturing ? nullptr : pool(true);
    return mp ? cudaMallocFromPoolAsync(p, bytes, mp, st) : cudaMallocAsync(p, bytes, st);
}

cudaError_t scratch_trim() {
    cudaMemPool_t mp = pool(false);
    return mp ? cudaMemPoolTrimTo(mp, 0) : cudaSuccess;
}

}  // namespace rfk
