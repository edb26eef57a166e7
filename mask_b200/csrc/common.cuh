// Shared helpers of the mask_b200 library: status reporting and small device utilities.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <new>

#include "mask_b200.h"

namespace mask {

// Per-thread message for the last failure, returned by mask_last_error().
void set_error(const char* fmt, ...);

inline int fail(int status, const char* what) {
    set_error("%s", what);
    return status;
}

// Runs the part of an entry point that allocates host memory: nothing may be thrown through the C ABI.
template <typename Body>
int without_exceptions(Body body) noexcept {
    try {
        return body();
    } catch (const std::bad_alloc&) {
        return fail(MASK_ERR_OUT_OF_MEMORY, "out of host memory");
    } catch (...) {
        return fail(MASK_ERR_INVALID_ARGUMENT, "unexpected exception");
    }
}

#define MASK_CUDA_TRY(expr)                                                              \
    do {                                                                                 \
        cudaError_t e_ = (expr);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            mask::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_),      \
                            __FILE__, __LINE__);                                         \
            return MASK_ERR_CUDA;                                                        \
        }                                                                                \
    } while (0)

#define MASK_REQUIRE(cond, msg)                                      \
    do {                                                             \
        if (!(cond)) return mask::fail(MASK_ERR_INVALID_ARGUMENT, msg); \
    } while (0)

constexpr int kWinRows = 16;   // rows per window
constexpr int kTileCols = 8;   // condensed columns per tile
constexpr int kTileElems = 128;

// Windows of M >= 1 rows; M + 15 need not fit int32.
__host__ __device__ inline int32_t window_count(int32_t M) { return (M - 1) / kWinRows + 1; }

inline unsigned blocks_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// Number of the thread, and of the warp, in the grid.  A warp per row passes 2^32 threads at 2^27 rows.
__device__ __forceinline__ int64_t grid_thread() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t grid_warp() { return grid_thread() >> 5; }

// Swizzle<2,2,3> over a row-major 16x8 tile (SR-BCRS value layout).
__host__ __device__ inline int sw223(int i) { return i ^ (((i >> 5) & 3) << 2); }
// Swizzle<1,2,3> over the same tile (ME-TCF COO index).
__host__ __device__ inline int sw123(int i) { return i ^ (((i >> 5) & 1) << 2); }

constexpr int kMaxDevices = 64;

inline int sm_count() {
    static std::atomic<int> known[kMaxDevices];   // asked for once per device
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev >= 0 && dev < kMaxDevices && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        return 148;
    if (dev >= 0 && dev < kMaxDevices) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Opts a kernel in to `bytes` of dynamic shared memory and the largest carveout, once per device.  `done` is the
// caller's, one bit per device and kernel (setting an attribute again does no harm).
inline int opt_in_shared_memory(const void* kernel, int bytes, std::atomic<uint64_t>& done) {
    int dev = 0;
    MASK_CUDA_TRY(cudaGetDevice(&dev));
    const uint64_t bit = dev >= 0 && dev < 64 ? (uint64_t)1 << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return MASK_OK;
    MASK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    MASK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    done.fetch_or(bit, std::memory_order_release);
    return MASK_OK;
}

}  // namespace mask
