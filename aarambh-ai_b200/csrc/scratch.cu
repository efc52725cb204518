// Device memory that a call needs only until its kernels have run, from one stream-ordered pool per device.
#include <mutex>

#include "common.cuh"

namespace ab2 {

// What stays in a pool between calls; the rest goes back to the device at the next synchronisation.
constexpr unsigned long long SCRATCH_KEPT_BYTES = 160ull << 20;

static std::mutex g_pool_mutex;
static cudaMemPool_t g_pool[64] = {nullptr};

int ScratchLease::take(size_t bytes) {
    int dev = 0;
    AB2_CUDA(cudaGetDevice(&dev));
    AB2_REQUIRE(dev >= 0 && dev < 64, AB2_ERR_BAD_ARG, "device index %d out of range", dev);
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        if (!g_pool[dev]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.handleTypes = cudaMemHandleTypeNone;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            AB2_CUDA(cudaMemPoolCreate(&g_pool[dev], &props));
            unsigned long long kept = SCRATCH_KEPT_BYTES;
            AB2_CUDA(cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &kept));
        }
    }
    AB2_CUDA(cudaMallocFromPoolAsync(&ptr, bytes, g_pool[dev], stream));
    return AB2_OK;
}

ScratchLease::~ScratchLease() {
    if (ptr) cudaFreeAsync(ptr, stream);
}

}  // namespace ab2
