#include "mem.h"

#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace mask {

namespace {

std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};

int pool_of_current_device(cudaMemPool_t* out) {
    int dev = -1;
    MASK_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(MASK_ERR_NO_DEVICE, "device ordinal outside the supported range");
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (g_pool[dev] == nullptr) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        MASK_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = kDevicePoolKeep;
        MASK_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pool[dev] = pool;
    }
    *out = g_pool[dev];
    return MASK_OK;
}

struct HostBuf {
    void* p;
    size_t size;
};
// never destroyed: a plan may be released while the process's static objects are already going away
std::mutex& host_mu() { static std::mutex* m = new std::mutex; return *m; }
std::vector<HostBuf>& host_free() { static auto* v = new std::vector<HostBuf>; return *v; }
size_t g_host_kept = 0;

}  // namespace

int device_alloc(void** p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    cudaMemPool_t pool = nullptr;
    int rc = pool_of_current_device(&pool);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 16), pool, st));
    return MASK_OK;
}

void device_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

int HostStage::get(size_t bytes) {
    {
        std::lock_guard<std::mutex> lock(host_mu());
        auto& v = host_free();
        int best = -1;
        for (int i = 0; i < (int)v.size(); i++)
            if (v[i].size >= bytes && (best < 0 || v[i].size < v[best].size)) best = i;
        if (best >= 0) {
            p_ = v[best].p;
            size_ = v[best].size;
            g_host_kept -= size_;
            v.erase(v.begin() + best);
            return MASK_OK;
        }
    }
    size_t size = 4096;
    while (size < bytes) size *= 2;
    MASK_CUDA_TRY(cudaHostAlloc(&p_, size, cudaHostAllocPortable));
    size_ = size;
    return MASK_OK;
}

HostStage::~HostStage() {
    if (!p_) return;
    {
        std::lock_guard<std::mutex> lock(host_mu());
        if (g_host_kept + size_ <= kHostCacheKeep) {
            const int rc = without_exceptions([&] { host_free().push_back({p_, size_}); return MASK_OK; });
            if (rc == MASK_OK) {
                g_host_kept += size_;
                return;
            }
        }
    }
    cudaFreeHost(p_);
}

}  // namespace mask
