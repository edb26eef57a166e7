// Sorting and ranking of small integer keys: a register sort for one warp, a bitmap with prefix counts for one
// block.  Used by the format builder (columns of a window) and the row reorders (neighbours of a node).
#pragma once

#include <climits>
#include <cstdint>

#include <cuda_runtime.h>

namespace mask {

template <typename Key>
__device__ __forceinline__ void order2(Key& a, Key& b) {
    const Key lo = a < b ? a : b, hi = a < b ? b : a;
    a = lo;
    b = hi;
}

// Ascending bitonic sort of 32 E keys held by a warp, key j in register j % E of lane j / E.  Runs that a
// bitonic network wants descending are sorted ascending with their bits flipped.
template <int E, typename Key>
__device__ __forceinline__ void warp_sort(Key (&key)[E], int lane) {
    Key flip = (lane & 1) ? ~(Key)0 : (Key)0;
#pragma unroll
    for (int i = 0; i < E; i++) key[i] ^= flip;
#pragma unroll
    for (int k = 2; k <= E; k <<= 1)
#pragma unroll
        for (int s = k >> 1; s > 0; s >>= 1)
#pragma unroll
            for (int i = 0; i < E; i++)
                if ((i ^ s) > i) {
                    if ((i & k) == 0 || k == E) order2(key[i], key[i ^ s]);
                    else order2(key[i ^ s], key[i]);
                }
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1) {
        const Key want = (lane & k & 31) ? ~(Key)0 : (Key)0;
        const Key turn = flip ^ want;
        flip = want;
#pragma unroll
        for (int i = 0; i < E; i++) key[i] ^= turn;
#pragma unroll 1
        for (int s = k >> 1; s > 0; s >>= 1) {
            const bool low = (lane & s) == 0;
#pragma unroll
            for (int i = 0; i < E; i++) {
                const Key o = __shfl_xor_sync(0xffffffffu, key[i], s);
                key[i] = ((o < key[i]) == low) ? o : key[i];
            }
        }
#pragma unroll
        for (int s = E >> 1; s > 0; s >>= 1)
#pragma unroll
            for (int i = 0; i < E; i++)
                if ((i ^ s) > i) order2(key[i], key[i ^ s]);
    }
}

// The least of the values that the THREADS threads of a block hand in, to all of them (INT_MAX: none).  `word`: one per
// warp; nobody may still read or write them.
template <int THREADS>
__device__ __forceinline__ int block_least(int x, int* word) {
    const int lane = threadIdx.x & 31;
    x = __reduce_min_sync(0xffffffffu, x);
    if (lane == 0) word[threadIdx.x >> 5] = x;
    __syncthreads();
    return __reduce_min_sync(0xffffffffu, lane < THREADS / 32 ? word[lane] : INT_MAX);
}

constexpr int kMarkMax = 1 << 20;   // most keys a MarkSet holds
constexpr int mark_set_bytes(int keys) { return keys / 8 + keys / 64; }   // bitmap, then `before`

// A bitmap of columns (or other small numbers) in shared memory and what ranks them: 16-bit counts of the marks before every four words
// (128 columns) within their run of 128 words (4096 columns), and the marks before every run.
struct MarkSet {
    uint32_t* bits;
    uint16_t* before;
    int* run_before;
    int n_runs;
    __device__ __forceinline__ void mark(int d) const { atomicOr(bits + (d >> 5), 1u << (d & 31)); }
    // For a whole warp whose keys mostly ascend with the lane (d < 0: none): lanes that share a word mark together,
    // which in a dense set would be up to 32 atomics on one address.  (__match_any_sync finds the lanes as well,
    // but took longer than the conflicts it saves.)
    __device__ __forceinline__ void mark_ascending(int d) const {
        const int lane = threadIdx.x & 31, word = d >> 5;
        uint32_t b = d >= 0 ? 1u << (d & 31) : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_down_sync(0xffffffffu, word, o);
            const uint32_t x = __shfl_down_sync(0xffffffffu, b, o);
            if (w == word) b |= x;   // lanes behind the last one return their own
        }
        const int left = __shfl_up_sync(0xffffffffu, word, 1);
        if (d >= 0 && (lane == 0 || left != word)) atomicOr(bits + word, b);
    }
    __device__ __forceinline__ void unmark(int d) { bits[d >> 5] = 0; }
    __device__ __forceinline__ int rank(int d) const {
        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(bits)[d >> 7];
        const unsigned long long below = (1ull << (d & 63)) - 1ull;
        return run_before[d >> 12] + before[d >> 7] + (d & 64 ? __popcll(v.x) + __popcll(v.y & below) : __popcll(v.x & below));
    }
    // Counts the marks of the whole set (returned to every thread) and prepares rank(); called by all THREADS threads.
    template <int THREADS>
    __device__ __forceinline__ int count(int* warp_sum) {
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        __syncthreads();
        for (int r = warp; r < n_runs; r += THREADS / 32) {   // four words a lane
            const uint4 v = reinterpret_cast<const uint4*>(bits)[r * 32 + lane];
            const int c = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            int x = c;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            before[r * 32 + lane] = (uint16_t)(x - c);
            if (lane == 31) run_before[r] = x;
        }
        __syncthreads();
        const int mine = tid < n_runs ? run_before[tid] : 0;
        int x = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        int ahead = 0, all = 0;
#pragma unroll
        for (int i = 0; i < (kMarkMax / 4096 < THREADS ? kMarkMax / 4096 : THREADS) / 32; i++) {
            const int v = warp_sum[i];
            all += v;
            if (i < warp) ahead += v;
        }
        if (tid < n_runs) run_before[tid] = ahead + x - mine;
        __syncthreads();
        return all;
    }
};

}  // namespace mask
