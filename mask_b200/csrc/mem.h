// Memory that outlives a call: a stream-ordered device pool for the plans' tables and for scratch, and a
// small cache of pinned host buffers for copies that the host waits for.
//
// cudaMalloc and cudaFree cost 10 to 300 us each and cudaFree waits for the whole device; building one plan
// made more than a dozen of each.  The device pool keeps at most kDevicePoolKeep bytes when nothing uses
// them (the driver gives back what is above at the next synchronisation), the host cache at most
// kHostCacheKeep.  Both may be used from any thread and stream.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace mask {

constexpr size_t kDevicePoolKeep = (size_t)128 << 20;   // per device
constexpr size_t kHostCacheKeep = (size_t)16 << 20;

// From / to the current device's pool, in stream order.
int device_alloc(void** p, size_t bytes, cudaStream_t st);
void device_free(void* p, cudaStream_t st);

// Device scratch of one call, freed in stream order when the frame ends.
struct DevScratch {
    void* p = nullptr;
    cudaStream_t st = nullptr;
    DevScratch() = default;
    DevScratch(const DevScratch&) = delete;
    DevScratch& operator=(const DevScratch&) = delete;
    ~DevScratch() { release(); }
    void release() {
        if (p) device_free(p, st);
        p = nullptr;
    }
    int alloc(size_t bytes, cudaStream_t stream) {
        st = stream;
        return device_alloc(&p, bytes, stream);
    }
    template <typename T> T* as(size_t byte_offset = 0) const { return reinterpret_cast<T*>(static_cast<char*>(p) + byte_offset); }
};

// A pinned host buffer held while in scope.  The holder synchronises before it lets go of the buffer.
class HostStage {
public:
    HostStage() = default;
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    ~HostStage();
    int get(size_t bytes);
    template <typename T> T* as() const { return static_cast<T*>(p_); }

private:
    void* p_ = nullptr;
    size_t size_ = 0;
};

}  // namespace mask
