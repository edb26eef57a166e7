// Device-wide exclusive scan over functors.
#pragma once

#include "common.cuh"

namespace mask {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanChunk = kScanThreads * kScanItems;
constexpr int kSmallItems = 4;
constexpr int kSmallScan = 2 * 1024 * kSmallItems;   // one block takes 4 us per 4096 items, two launches 8 us
constexpr int kDirectSpine = 4096;                   // chunks whose sums every block of the last pass adds up itself

// Words of int64 that device_scan needs at `spine` for n items.
inline size_t scan_spine_words(int64_t n) { return (size_t)((n + kScanChunk - 1) / kScanChunk + 1); }

// ---- device-wide scan (reduce chunks, with many of them scan their sums in one block, apply) --------------------
// In: functor giving the value at index i (int32 or int64; sums are 64-bit, so two counts can share a value).  Out:
// functor receiving (i, exclusive, value).
template <typename In>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(In in, int64_t n, int64_t* spine) {
    __shared__ int64_t warp_sum[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk;
    int64_t s = 0;
    for (int i = threadIdx.x; i < kScanChunk; i += kScanThreads) {
        const int64_t idx = base + i;
        if (idx < n) s += in(idx);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int i = 0; i < kScanThreads / 32; i++) t += warp_sum[i];
        spine[blockIdx.x] = t;
    }
}

// One block: exclusive scan of spine[0..nchunks) in place.
static __global__ void __launch_bounds__(1024) scan_spine_kernel(int64_t* spine, int64_t nchunks) {
    __shared__ int64_t warp_tot[32];
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t base = 0; base < nchunks; base += 1024) {
        const int64_t idx = base + threadIdx.x;
        const int64_t v = idx < nchunks ? spine[idx] : 0;
        int64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int64_t w = warp_tot[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_tot[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const int64_t before = carry + (wid > 0 ? warp_tot[wid - 1] : 0);
        if (idx < nchunks) spine[idx] = before + x - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_tot[31];
        __syncthreads();
    }
}

template <typename In, typename Out>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(In in, Out out, int64_t n, const int64_t* spine, bool scanned) {
    __shared__ int64_t warp_tot[kScanThreads / 32], warp_ahead[kScanThreads / 32];
    int64_t ahead = 0;   // of the chunks before this one
    if (!scanned)
        for (int i = threadIdx.x; i < blockIdx.x; i += kScanThreads) ahead += spine[i];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanItems;
    decltype(in((int64_t)0)) v[kScanItems];
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = (base + i < n) ? in(base + i) : 0;
        s += v[i];
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t x = s;
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    for (int o = 16; o > 0; o >>= 1) ahead += __shfl_xor_sync(0xffffffffu, ahead, o);
    if (lane == 31) {
        warp_tot[wid] = x;
        warp_ahead[wid] = ahead;
    }
    __syncthreads();
    int64_t before = x - s + (scanned ? spine[blockIdx.x] : 0);
    for (int i = 0; i < kScanThreads / 32; i++) before += warp_ahead[i] + (i < wid ? warp_tot[i] : 0);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out(base + i, before, v[i]);
        before += v[i];
    }
}

// The whole scan in one block, for counts that three launches would take longer for.
template <typename In, typename Out>
__global__ void __launch_bounds__(1024) scan_small_kernel(In in, Out out, int64_t n) {
    __shared__ int64_t warp_tot[32];
    int64_t carry = 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t c = 0; c < n; c += 1024 * kSmallItems) {
        const int64_t base = c + (int64_t)threadIdx.x * kSmallItems;
        decltype(in((int64_t)0)) v[kSmallItems];
        int64_t s = 0;
#pragma unroll
        for (int i = 0; i < kSmallItems; i++) {
            v[i] = (base + i < n) ? in(base + i) : 0;
            s += v[i];
        }
        int64_t x = s;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[wid] = x;
        __syncthreads();
        int64_t before = carry + x - s;
        for (int i = 0; i < 32; i++) {
            const int64_t t = warp_tot[i];
            if (i < wid) before += t;
            carry += t;
        }
#pragma unroll
        for (int i = 0; i < kSmallItems; i++) {
            if (base + i < n) out(base + i, before, v[i]);
            before += v[i];
        }
        __syncthreads();
    }
}

template <typename In, typename Out>
static int device_scan(In in, Out out, int64_t n, int64_t* spine, cudaStream_t st) {
    if (n <= kSmallScan) {
        scan_small_kernel<<<1, 1024, 0, st>>>(in, out, n);
        MASK_CUDA_TRY(cudaGetLastError());
        return MASK_OK;
    }
    const int64_t chunks = (n + kScanChunk - 1) / kScanChunk;
    scan_reduce_kernel<<<(unsigned)chunks, kScanThreads, 0, st>>>(in, n, spine);
    MASK_CUDA_TRY(cudaGetLastError());
    const bool scanned = chunks > kDirectSpine;
    if (scanned) {
        scan_spine_kernel<<<1, 1024, 0, st>>>(spine, chunks);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    scan_apply_kernel<<<(unsigned)chunks, kScanThreads, 0, st>>>(in, out, n, spine, scanned);
    MASK_CUDA_TRY(cudaGetLastError());
    return MASK_OK;
}

}  // namespace mask
