// Per-device pool behind StreamScratch.
#include "scratch.cuh"

#include <mutex>

namespace omb {

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
int g_holders[kMaxDevices] = {};
}  // namespace

void scratch_hold(int device) {
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> lock(g_mutex);
    ++g_holders[device];
    if (g_pool[device]) return;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    unsigned long long kept = kScratchKept;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept);
    g_pool[device] = pool;
}

void scratch_drop(int device) {
    if (device < 0 || device >= kMaxDevices) return;
    std::lock_guard<std::mutex> lock(g_mutex);
    // (the pool object itself stays: it holds nothing after the trim)
    if (--g_holders[device] == 0 && g_pool[device]) cudaMemPoolTrimTo(g_pool[device], 0);
}

StreamScratch::StreamScratch(size_t bytes, cudaStream_t st) : stream(st) {
    int device = 0;
    if (bytes == 0) return;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (capture != cudaStreamCaptureStatusNone) return;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return;
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        pool = g_pool[device];
    }
    if (pool && cudaMallocFromPoolAsync(&p, bytes, pool, st) != cudaSuccess) {
        cudaGetLastError();
        p = nullptr;
    }
}

StreamScratch::~StreamScratch() {
    if (p) cudaFreeAsync(p, stream);
}

}  // namespace omb
