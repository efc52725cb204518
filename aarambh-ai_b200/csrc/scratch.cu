// Device memory that a call needs only until its kernels have run, from one stream-ordered pool per device.
#include <mutex>

#include "common.cuh"

namespace ab2 {

// What stays in a pool between calls; the rest goes back to the device at the next synchronisation.
constexpr unsigned long long SCRATCH_KEPT_BYTES = 160ull << 20;

static std::mutex g_pool_mutex;
static cudaMemPool_t g_pool[64] = {nullptr};

static cudaError_t pool_of(int dev, cudaMemPool_t *out) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaError_t e = cudaMemPoolCreate(&g_pool[dev], &props);
        if (e != cudaSuccess) { g_pool[dev] = nullptr; return e; }
        unsigned long long kept = SCRATCH_KEPT_BYTES;
        cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &kept);
    }
    *out = g_pool[dev];
    return cudaSuccess;
}

thread_local const RecordedScratch *g_recorded_scratch = nullptr;

// For hosts that keep the device's memory to themselves: no lease is larger.
bool scratch_allowed(size_t bytes) {
    static const char *most = getenv("AB2_SCRATCH_MAX_BYTES");
    return !most || bytes <= strtoull(most, nullptr, 10);
}

int scratch_prepare() {
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    cudaMemPool_t pool;
    if (pool_of(dev, &pool) != cudaSuccess) cudaGetLastError();  // leases will be refused
    return AB2_OK;
}

bool ScratchLease::take(size_t bytes) {
    if (!scratch_allowed(bytes)) return false;
    if (g_recorded_scratch) {
        if (bytes > g_recorded_scratch->bytes) return false;
        ptr = g_recorded_scratch->ptr;
        return true;
    }
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= 64)) return false;
    if (e == cudaSuccess) e = pool_of(dev, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&ptr, bytes, pool, stream);
    if (e == cudaSuccess) return pooled = true;
    ptr = nullptr;
    cudaGetLastError();
    return false;
}

ScratchLease::~ScratchLease() {
    if (pooled) cudaFreeAsync(ptr, stream);
}

}  // namespace ab2
