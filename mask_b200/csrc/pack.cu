// Device format builder: CSR -> SR-BCRS 16x8 / ME-TCF / MCO, bit-identical to the reference host packers.
//
// The reference condenses the columns of every 16-row window with a per-thread byte mask over
// all K columns plus std::sort, then places every entry with a binary search
// (examples/src_fp32/sr_bcrs/testbed/main_16x8.cu:209-318).  Here:
//
//   1. condense    every entry gets its condensed position (the rank of its column among the distinct
//                  columns of its window), every window its number of distinct columns.  The entries of a
//                  window are contiguous in the CSR.  Windows of up to 1024 entries: one warp sorts them in
//                  registers (bitonic network over 1..32 keys a lane, key = column << 10 | entry) and
//                  numbers the distinct ones.  Larger windows: one block marks the columns in a bitmap in
//                  shared memory, 2^19 columns at a time, and ranks every entry by a prefix popcount, which
//                  costs the same whatever the row lengths.  Rows that are not strictly ascending or columns
//                  outside [0, K) raise an error flag.
//   2. tiles       ceil(distinct / 8) per window, exclusive scan -> val_soff, total T; the scan also notes
//                  the window in which every 64th tile lies.
//   3. fill        one warp per 16 to 64 consecutive tiles composes them 8 at a time in shared memory (a row of
//                  the window is walked from the entry where the tiles begin; positions ascend along a row)
//                  and writes whole tiles, so a value array of 512 bytes a tile is written once, coalesced,
//                  and never read.  ME-TCF and MCO count the entries per tile the same way first (16 x 4-bit row
//                  histogram, 128-bit mask), scan the run lengths and place the entries.
//
// Measured on a power-law graph with 2^20 nodes (17.1 M entries, 1.97 M tiles; one read of the CSR and one
// write of the packed arrays is 0.2 ms at copy speed): condense 0.13 ms and, overlapping, 0.09 and 0.12 for large windows, scan 0.01,
// SR-BCRS fill 0.32; a binary
// search of every entry in its 15 sibling rows, two more scans and a scatter into cleared tiles took 2.3 ms.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "condense.cuh"
#include "mem.h"
#include "scan.cuh"
#include "launch.cuh"

namespace mask {

constexpr int kFillTiles = 64;   // most tiles a warp of the fill writes, not counting the rest of a small window
constexpr int kFillThreads = 128;

struct PackScratch {
    int32_t* pos;           // nnz: condensed position of every entry
    int32_t* cols;          // nnz: distinct columns of a window in ascending order, from the window's first entry on
    int32_t* rows;          // 16 W + 1: rowptr, rows behind the last one empty
    int32_t* distinct;      // W: distinct columns per window
    int32_t* big_list;      // windows of condense_big_kernel
    int32_t* hub_list;      // windows of condense_hub_kernel
    int32_t* first_window;  // per kFillTiles tiles (at most nnz tiles)
    int64_t* spine;         // per scan chunk
    int32_t* status;        // [0] error flags, [4], [5] lengths of the lists
    size_t bytes;
};

static inline size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

static PackScratch carve(void* base, int32_t M, int64_t nnz) {
    PackScratch s{};
    char* p = static_cast<char*>(base);
    size_t off = 0;
    const size_t n = (size_t)std::max<int64_t>(nnz, 1), W = (size_t)window_count(M);
    auto take = [&](size_t bytes) { char* r = p ? p + off : nullptr; off += align_up(bytes); return r; };
    s.pos = reinterpret_cast<int32_t*>(take(n * 4));
    s.cols = reinterpret_cast<int32_t*>(take(n * 4));
    s.rows = reinterpret_cast<int32_t*>(take((W * kWinRows + 1) * 4));
    s.distinct = reinterpret_cast<int32_t*>(take(W * 4));
    s.big_list = reinterpret_cast<int32_t*>(take((n / 1024 + 1) * 4));
    s.hub_list = reinterpret_cast<int32_t*>(take((n / 8192 + 1) * 4));
    s.first_window = reinterpret_cast<int32_t*>(take((n / kFillTiles + 1) * 4));
    const size_t chunks = (std::max<size_t>(n, (size_t)M + 1) + kScanChunk - 1) / kScanChunk + 1;
    s.spine = reinterpret_cast<int64_t*>(take(chunks * 8));
    s.status = reinterpret_cast<int32_t*>(take(64));
    s.bytes = std::max(off, 16 * n);   // hosts have sized it by 16 bytes an entry
    return s;
}

// ---- condensed positions ---------------------------------------------------------------------
constexpr int kSortMax = 1024;                    // largest window a warp sorts in registers
constexpr int kSortIdxBits = 10;
constexpr int kHubMin = 8192;                     // larger windows are shared by the blocks of a cluster
constexpr int kBigThreads = 512;
constexpr int kBigKeep = kHubMin / kBigThreads;
constexpr int kHubThreads = 512;
constexpr int kHubKeep = 8;                       // entries a thread of them keeps in registers
static_assert(kHubThreads == 32 * kWinRows, "a warp for each row");
constexpr int kBigBits = 1 << 19;                 // columns marked at a time: two blocks per SM
constexpr int kHubBlocks = 8;
constexpr int kHubBits = 1 << 19;                 // columns marked at a time by one block of a cluster: two blocks per SM
constexpr int kHubBitsWide = 1 << 20;             // the same where eight of these cover K and eight of those do not: one block per SM
static_assert(kHubBitsWide <= kMarkMax, "");

// One window of n <= 32 E entries: sorts (column, entry), numbers the distinct columns, writes every entry's
// number to pos and the distinct columns to cols; returns how many there are.
template <int E, typename Key>
__device__ __forceinline__ int condense_warp(const int32_t* __restrict__ col, int n, int lane, uint16_t* __restrict__ slot_pos,
                                             int32_t* __restrict__ pos, int32_t* __restrict__ cols) {
    Key key[E];
#pragma unroll
    for (int i = 0; i < E; i++) {
        const int e = i * 32 + lane;   // any order will do
        key[i] = e < n ? ((Key)(uint32_t)__ldg(col + e) << kSortIdxBits) | (Key)e : ~(Key)0;
    }
    warp_sort<E, Key>(key, lane);
    Key before = __shfl_up_sync(0xffffffffu, key[E - 1], 1);
    int cnt = 0;
    uint32_t first = 0;   // bit i: key i starts a new column
#pragma unroll
    for (int i = 0; i < E; i++) {
        const bool f = lane * E + i < n && ((lane == 0 && i == 0) || (key[i] >> kSortIdxBits) != (before >> kSortIdxBits));
        before = key[i];
        first |= (f ? 1u : 0u) << i;
        cnt += f;
    }
    int x = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    int at = x - cnt - 1;
#pragma unroll
    for (int i = 0; i < E; i++) {
        at += (first >> i) & 1u;
        if (lane * E + i < n) slot_pos[(uint32_t)key[i] & (kSortMax - 1)] = (uint16_t)at;
    }
    __syncwarp();
    for (int e = lane; e < n; e += 32) {
        const int q = slot_pos[e];
        pos[e] = q;
        if (q < n) cols[q] = __ldg(col + e);   // entries of one column write the same word
    }
    return __shfl_sync(0xffffffffu, x, 31);
}

// Is column c of entry e acceptable: inside [0, K), and above its left neighbour unless e begins a row?
__device__ __forceinline__ int entry_faults(const int32_t* __restrict__ colind, int e, int c, int32_t K, bool row_start) {
    int bad = (c < 0 || c >= K) ? 2 : 0;
    if (!row_start && __ldg(colind + e - 1) >= c) bad |= 1;
    return bad;
}

// Which of the 32 entries from e on begin a row, for a whole warp; bound: where row `lane` of the window begins (lanes 0..15).
// (Comparing every entry with all 16 cost condense_big_kernel 139 us where this and no work behind a window's end cost 123.)
__device__ __forceinline__ uint32_t row_starts(int bound, int e) {
    const uint32_t at = (uint32_t)(bound - e);
    return __reduce_or_sync(0xffffffffu, (threadIdx.x & 31) < kWinRows && at < 32u ? 1u << at : 0u);
}

// One warp, which is a block, per window; windows above kSortMax entries go to the list of the bitmap kernel.  What bounds it is the
// latency of a warp's loads and of its sort, so as many warps as registers allow (power-law graph with 2^20 nodes: four warps a
// block, 20 of 96 registers an SM, 148 us; 24 single ones of 80 registers 135, 28 of 72 128; the 64-bit keys of more than 2^22
// columns would spill).
template <typename Key>
__global__ void __launch_bounds__(32, sizeof(Key) == 4 ? 28 : 12) condense_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind,
                                                       int32_t M, int32_t K, int32_t W, int32_t* __restrict__ pos,
                                                       int32_t* __restrict__ cols, int32_t* __restrict__ rows,
                                                       int32_t* __restrict__ distinct, int32_t* __restrict__ big_list,
                                                       int32_t* __restrict__ hub_list, int32_t* __restrict__ status) {
    __shared__ uint16_t slot_pos[kSortMax];
    const int lane = threadIdx.x, w = blockIdx.x;
    if (w >= W) return;
    const int r0 = w * kWinRows;
    const int bound = __ldg(rowptr + r0 + min(min(lane, kWinRows), M - r0));   // lane i: where row i of the window begins
    const int base = __shfl_sync(0xffffffffu, bound, 0), n = __shfl_sync(0xffffffffu, bound, kWinRows) - base;
    if (lane <= kWinRows) (rows + r0)[lane] = bound;   // entry 16 is the next window's entry 0
    if (n > kSortMax) {
        if (lane == 0) {
            if (n > kHubMin) hub_list[atomicAdd(status + 5, 1)] = w;
            else big_list[atomicAdd(status + 4, 1)] = w;
        }
        return;
    }
    int bad = 0;
    for (int j = 0; j < n; j += 32) {
        const int e = base + j + lane;
        const uint32_t starts = row_starts(bound, base + j);
        if (j + lane < n) bad |= entry_faults(colind, e, __ldg(colind + e), K, starts >> lane & 1u);
    }
    if (bad) atomicOr(status, bad);
    int d = 0;
    if (n > 512) d = condense_warp<32, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    else if (n > 256) d = condense_warp<16, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    else if (n > 128) d = condense_warp<8, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    else if (n > 64) d = condense_warp<4, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    else if (n > 32) d = condense_warp<2, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    else if (n > 0) d = condense_warp<1, Key>(colind + base, n, lane, slot_pos, pos + base, cols + base);
    if (lane == 0) distinct[w] = d;
}

// Windows of kSortMax + 1 to kHubMin entries, dealt to the blocks round-robin: the entries stay in registers,
// kBigBits columns are marked, counted, ranked and unmarked at a time, each time from the smallest column that is
// left: columns up to 2^31 - 2 are 4096 such ranges, most of them without an entry of the window.
__global__ void __launch_bounds__(kBigThreads, 2) condense_big_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind,
                                                                   int32_t M, int32_t K, int32_t* __restrict__ pos,
                                                                   int32_t* __restrict__ cols, int32_t* __restrict__ distinct,
                                                                   const int32_t* __restrict__ big_list, int32_t* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int run_before[kBigBits / 4096];
    __shared__ int bound[kWinRows + 1];
    __shared__ int warp_sum[32];
    const int tid = threadIdx.x;
    const int n_big = status[4];
    MarkSet marks{reinterpret_cast<uint32_t*>(smem), reinterpret_cast<uint16_t*>(smem + kBigBits / 8), run_before,
                  (min(K, kBigBits) + 4095) / 4096};
    for (int i = tid; i < marks.n_runs * 128; i += kBigThreads) marks.bits[i] = 0;
    for (int b = blockIdx.x; b < n_big; b += gridDim.x) {
        const int w = big_list[b];
        __syncthreads();
        if (tid <= kWinRows) bound[tid] = (rowptr + w * kWinRows)[min(tid, M - w * kWinRows)];
        __syncthreads();
        const int e0 = bound[0], n = bound[kWinRows] - e0;
        const int mine = bound[tid & (kWinRows - 1)];
        int total = 0, bad = 0;
        int c[kBigKeep];
#pragma unroll
        for (int i = 0; i < kBigKeep; i++) {
            const int j = i * kBigThreads + tid;
            c[i] = j < n ? __ldg(colind + e0 + j) : -1;
        }
#pragma unroll
        for (int i = 0; i < kBigKeep; i++) {
            if (i * kBigThreads >= n) break;
            const int e = e0 + i * kBigThreads + tid;
            const uint32_t starts = row_starts(mine, e - (tid & 31));
            if (e - e0 < n) bad |= entry_faults(colind, e, c[i], K, starts >> (tid & 31) & 1u);
            if (c[i] >= K) c[i] = -1;
        }
        // the smallest column from `from` on, INT_MAX if there is none
        auto least_from = [&](int from) {
            int x = INT_MAX;
#pragma unroll
            for (int i = 0; i < kBigKeep; i++)
                if (c[i] >= from) x = min(x, c[i]);
            return block_least<kBigThreads>(x, warp_sum);
        };
        const bool few = K <= 4 * kBigBits;   // looking for the next column costs about what an empty range does
        for (int c0 = few ? 0 : least_from(0); c0 < K;) {
            const int span = min(kBigBits, K - c0);
#pragma unroll
            for (int i = 0; i < kBigKeep; i++) {
                if (i * kBigThreads >= n) break;
                if (c[i] >= c0 && c[i] - c0 < span) marks.mark(c[i] - c0);
            }
            const int all = marks.count<kBigThreads>(warp_sum);
#pragma unroll
            for (int i = 0; i < kBigKeep; i++) {
                if (i * kBigThreads >= n) break;
                if (c[i] >= c0 && c[i] - c0 < span) {
                    const int q = total + marks.rank(c[i] - c0);
                    pos[e0 + i * kBigThreads + tid] = q;
                    cols[e0 + q] = c[i];
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kBigKeep; i++) {
                if (i * kBigThreads >= n) break;
                if (c[i] >= c0 && c[i] - c0 < span) marks.unmark(c[i] - c0);
            }
            total += all;
            __syncthreads();
            if (span == K - c0) break;
            c0 = few ? c0 + span : least_from(c0 + span);
        }
        if (bad) atomicOr(status, bad);
        if (tid == 0) distinct[w] = total;
    }
    wait_for_previous_kernel();   // the hub windows' kernel, if any, has ended when this one has
}

// Windows of more than kHubMin entries, dealt to clusters of kHubBlocks blocks.  Every block takes a range of
// columns -- cut at the eighths of the window's longest row, so that the ranges hold about as many entries each, but no wider than
// a block's marks where eight of those cover K -- which is a run of entries in each of the 16 rows, found by a 32-way search; the blocks
// exchange their counts through distributed shared memory and rank what they marked themselves.  A range wider than the marks is taken
// in parts (marked once to count, once more to rank), each from the smallest column that is left.  Up to kHubKeep entries a thread
// are read once and kept.  A window takes 12 us, most of it waiting, whether a block has one entry a thread or five, so what
// counts is how many clusters run at a time: with marks for 2^20 columns a block filled an SM, and ten clusters of 8 found
// room (137 such windows of a power-law graph with 2^20 nodes: 165 us, with two blocks an SM 81 to 102; with marks for 2^18 most
// ranges are taken in parts: 255).  With one block per window the 150 000 entries of the largest took 0.3 ms.
// Where eight marks of 2^19 columns do not cover K, parts cost more than the second block is worth.  Condensing in all, ranges at the
// eighths alone and 2^19 columns always / as here: power-law graphs of 2^20 nodes 369 / 374 us, 2^21 1600 / 1020, 2^22 4560 / 3030, 2^23
// 13 800 / 10 200, 2^22 and twice the degree 12 000 / 6020; 200 windows of 12 000 / 30 000 / 100 000 entries spread over 2^20 columns
// 122 / 130, 197 / 182, 502 / 505; over 2^22 262 / 140, 456 / 193, 1197 / 540; over 2^23 367 / 249, 652 / 341, 1675 / 977.  Beyond that there
// are parts either way, and two blocks an SM get through them sooner: 12 000 / 100 000 entries over 2^24 columns 570 / 2630 us, with marks for 2^20 773 /
// 3300; over 2^26 1740 / 8360 and 2200 / 9160.
__global__ void __cluster_dims__(kHubBlocks, 1, 1) __launch_bounds__(kHubThreads, 2)
condense_hub_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind, int32_t M, int32_t K, int32_t span,
                    int32_t* __restrict__ pos, int32_t* __restrict__ cols, int32_t* __restrict__ distinct,
                    const int32_t* __restrict__ hub_list, int32_t* __restrict__ status) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int run_before[kHubBitsWide / 4096];
    __shared__ int bound[kWinRows + 1];
    __shared__ int cut[2][kWinRows];           // first entry of the row in this block's columns, first behind them
    __shared__ int first[kWinRows + 1];        // list index of the row's first entry
    __shared__ int warp_sum[32];
    __shared__ int range_marks[2][kHubBlocks]; // two windows: a block may be one ahead of another
    let_next_kernel_start();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int me = (int)cluster.block_rank();
    const int n_hub = status[5], n_clusters = gridDim.x / kHubBlocks;
    MarkSet marks{reinterpret_cast<uint32_t*>(smem), reinterpret_cast<uint16_t*>(smem + span / 8), run_before, span / 4096};
    for (int i = tid; i < span / 128; i += kHubThreads) reinterpret_cast<uint4*>(marks.bits)[i] = make_uint4(0u, 0u, 0u, 0u);
    int turn = 0;
    for (int b = blockIdx.x / kHubBlocks; b < n_hub; b += n_clusters, turn ^= 1) {
        const int w = hub_list[b];
        __syncthreads();
        if (tid <= kWinRows) bound[tid] = (rowptr + w * kWinRows)[min(tid, M - w * kWinRows)];
        __syncthreads();
        const int e0 = bound[0], n = bound[kWinRows] - e0;
        int bad = 0;
        const int row_begin = bound[lane & (kWinRows - 1)];
#pragma unroll 4
        for (uint32_t j0 = me * kHubThreads + warp * 32; j0 < (uint32_t)n; j0 += kHubBlocks * kHubThreads) {
            const int e = e0 + (int)j0 + lane;
            const uint32_t starts = row_starts(row_begin, e0 + (int)j0);
            if (j0 + lane < (uint32_t)n) bad |= entry_faults(colind, e, __ldg(colind + e), K, starts >> lane & 1u);
        }
        if (bad) atomicOr(status, bad);
        int longest = 0;
        for (int r = 1; r < kWinRows; r++)
            if (bound[r + 1] - bound[r] > bound[longest + 1] - bound[longest]) longest = r;
        const int at = bound[longest], len = bound[longest + 1] - at;   // len >= 512: the window has more than 8192 entries
        const bool cover = K <= kHubBlocks * span;   // then no range is wider than a span
        int eighth[kHubBlocks];
#pragma unroll
        for (int i = 1; i <= kHubBlocks; i++) eighth[i - 1] = i == kHubBlocks ? K : min(K, __ldg(colind + at + (int)((int64_t)len * i / kHubBlocks)));
        int c_lo = 0, c_hi = 0;
#pragma unroll
        for (int i = 1, c = 0; i <= kHubBlocks; i++) {
            if (i == me + 1) c_lo = c;
            c = max(c, cover ? max(K - (kHubBlocks - i) * span, min(eighth[i - 1], c + span)) : eighth[i - 1]);
            if (i == me + 1) c_hi = c;
        }
        {   // a row for each warp, both ends at once
            int p[2] = {bound[warp], bound[warp]}, left[2] = {bound[warp + 1] - p[0], bound[warp + 1] - p[0]};
            while (left[0] > 0 || left[1] > 0) {
                int stride[2], probe[2];
                bool below[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    stride[h] = (left[h] + 31) >> 5;
                    probe[h] = min((lane + 1) * stride[h], left[h]);
                    below[h] = left[h] > 0 && __ldg(colind + p[h] + probe[h] - 1) < (h ? c_hi : c_lo);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int hits = __popc(__ballot_sync(0xffffffffu, below[h]));   // the probes that hit come first
                    const int step = hits == 32 ? left[h] : min(hits * stride[h], left[h]);
                    p[h] += step;
                    left[h] = hits == 32 ? 0 : max(0, min(stride[h] - 1, left[h] - step));
                }
            }
            if (lane < 2) cut[lane][warp] = p[lane];
        }
        __syncthreads();
        if (tid == 0) {
            int x = 0;
            for (int r = 0; r < kWinRows; r++) {
                first[r] = x;
                x += max(cut[1][r] - cut[0][r], 0);
            }
            first[kWinRows] = x;
        }
        __syncthreads();
        const int m = first[kWinRows];
        auto entry = [&](int i) {   // entry of list index i
            int r = 0;
#pragma unroll
            for (int half = kWinRows / 2; half > 0; half >>= 1)
                if (first[r + half] <= i) r += half;
            return cut[0][r] + i - first[r];
        };
        // columns of [c0, c0 + part); others only occur in the list when rows are not ascending, which is an error anyway
        auto mark_part = [&](int c0, int part) {
            marks.n_runs = (part + 4095) / 4096;
            for (int i0 = 0; i0 < m; i0 += 4 * kHubThreads) {
                int c[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int i = i0 + k * kHubThreads + tid;
                    c[k] = i < m ? __ldg(colind + entry(i)) : -1;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) marks.mark_ascending(c[k] >= c0 && c[k] - c0 < part ? c[k] - c0 : -1);
            }
        };
        const bool whole = c_hi - c_lo <= span;
        // returns where the next part begins: the smallest column behind this one, c_hi or more if there is none
        auto unmark_part = [&](int c0, int part) {
            int behind = INT_MAX;
            __syncthreads();
            if (whole) {   // every word that can be marked
                for (int i = tid; i < marks.n_runs * 32; i += kHubThreads) reinterpret_cast<uint4*>(marks.bits)[i] = make_uint4(0u, 0u, 0u, 0u);
            } else {
#pragma unroll 4
                for (int i = tid; i < m; i += kHubThreads) {
                    const int c = __ldg(colind + entry(i));
                    if (c < c0) continue;
                    if (c - c0 < part) marks.unmark(c - c0);
                    else behind = min(behind, c);
                }
            }
            __syncthreads();
            return whole ? c_hi : block_least<kHubThreads>(behind, warp_sum);
        };
        // Few entries, in one part: read once and kept.
        const bool kept = whole && m <= kHubKeep * kHubThreads;
        int ke[kHubKeep], kc[kHubKeep];
        int mine = 0;
        if (kept) {
#pragma unroll
            for (int k = 0; k < kHubKeep; k++) {
                const int i = k * kHubThreads + tid;
                ke[k] = i < m ? entry(i) : -1;
            }
#pragma unroll
            for (int k = 0; k < kHubKeep; k++) {
                kc[k] = ke[k] >= 0 ? __ldg(colind + ke[k]) : -1;
                if (kc[k] < c_lo || kc[k] >= c_hi) ke[k] = -1;
            }
            marks.n_runs = (c_hi - c_lo + 4095) / 4096;
#pragma unroll
            for (int k = 0; k < kHubKeep; k++)
                if (k * kHubThreads < m) marks.mark_ascending(ke[k] >= 0 ? kc[k] - c_lo : -1);
            mine = marks.count<kHubThreads>(warp_sum);
        }
        for (int c0 = kept ? c_hi : c_lo; c0 < c_hi;) {
            const int part = min(span, c_hi - c0);
            mark_part(c0, part);
            mine += marks.count<kHubThreads>(warp_sum);
            c0 = whole ? c_hi : unmark_part(c0, part);
        }
        if (tid < kHubBlocks) cluster.map_shared_rank(range_marks[turn], tid)[me] = mine;
        cluster.sync();
        int ahead = 0, total = 0;
        for (int i = 0; i < kHubBlocks; i++) {
            const int v = range_marks[turn][i];
            total += v;
            if (i < me) ahead += v;
        }
        if (kept) {
#pragma unroll
            for (int k = 0; k < kHubKeep; k++)
                if (ke[k] >= 0) {
                    const int q = ahead + marks.rank(kc[k] - c_lo);
                    pos[ke[k]] = q;
                    cols[e0 + q] = kc[k];
                }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kHubKeep; k++)
                if (ke[k] >= 0) marks.unmark(kc[k] - c_lo);
            __syncthreads();
        }
        for (int c0 = kept ? c_hi : c_lo; c0 < c_hi;) {
            const int part = min(span, c_hi - c0);
            int here = mine;
            if (!whole) {
                mark_part(c0, part);
                here = marks.count<kHubThreads>(warp_sum);
            }
            for (int i0 = 0; i0 < m; i0 += 4 * kHubThreads) {
                int e[4], c[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int i = i0 + k * kHubThreads + tid;
                    e[k] = i < m ? entry(i) : -1;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) c[k] = e[k] >= 0 ? __ldg(colind + e[k]) : -1;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (c[k] >= c0 && c[k] - c0 < part) {
                        const int q = ahead + marks.rank(c[k] - c0);
                        pos[e[k]] = q;
                        cols[e0 + q] = c[k];
                    }
            }
            c0 = unmark_part(c0, part);
            ahead += here;
        }
        if (me == 0 && tid == 0) distinct[w] = total;
    }
    cluster.sync();   // nobody leaves while another block may still write its counts here
}

// What a host waits for: pinned memory that the last kernel writes itself, a copy's 6 us cheaper than a copy.
struct HostWords {
    int64_t total;
    int32_t status;
};

// tiles per window, and their exclusive scan
struct WindowTilesIn {
    const int32_t* distinct;
    int32_t W;
    __device__ int32_t operator()(int64_t w) const { return w < W ? (distinct[w] + kTileCols - 1) / kTileCols : 0; }
};
// first_window[c]: the window that holds tile c * kFillTiles
struct SoffOut {
    int32_t* soff;
    int32_t* first_window;
    int32_t W;
    const int32_t* status;
    HostWords* host;
    __device__ void operator()(int64_t w, int64_t before, int32_t tiles) const {
        soff[w] = (int32_t)before;
        if (w == W) {
            host->total = before;
            host->status = *status;
        }
        for (int64_t c = (before + kFillTiles - 1) / kFillTiles; c * kFillTiles < before + tiles; c++) first_window[c] = (int32_t)w;
    }
};

// ---- fill ------------------------------------------------------------------------------------
// nibble r of a tile's row word: stored entries of window row r in the tile (at most 8)
__device__ __forceinline__ int nibble_sum(unsigned long long x) {
    x = (x & 0x0f0f0f0f0f0f0f0full) + ((x >> 4) & 0x0f0f0f0f0f0f0f0full);
    return (int)((x * 0x0101010101010101ull) >> 56);
}

enum FillMode { kFillSrbcrs, kCountMetcf, kFillMetcf, kMaskMco, kFillMco };

struct FillArgs {
    const int32_t* rows;
    const int32_t* cols;
    const int32_t* distinct;
    const float* values;       // NULL: every entry is 1.0 (ME-TCF, MCO)
    const int32_t* pos;
    const int32_t* soff;
    const int32_t* first_window;
    int32_t W;
    int64_t T;
    int32_t chunk;             // tiles per warp: 16, 32 or 64
    int32_t skip_zero;         // MCO: entries with value 0 are not stored
    int32_t* sidx;
    float* block_val;          // SR-BCRS
    int32_t whole_vectors;     // block_val is 16-byte aligned
    int32_t* edge_to_col;
    int32_t* edge_to_row;
    unsigned long long* tile_rows;   // ME-TCF: entries per row of a tile, 16 nibbles
    unsigned long long* masks;       // MCO
    const int32_t* off;        // ME-TCF: [begin, end) per tile; MCO: begin per tile
    int32_t* coo_idx;
    float* out_val;
};

// The window that holds tile t, for a whole warp: the last one from w on that begins at or before t (window w does, the
// end of the last one does not).  32 windows are looked at in a step, then every 32nd, and so on, so that a run of
// windows without tiles costs a step for each factor of 32 in its length.
__device__ __forceinline__ int window_of_tile(const int32_t* __restrict__ soff, int32_t W, int w, int64_t t) {
    const int lane = threadIdx.x & 31;
    for (int stride = 1;;) {
        const int at = (int)min((int64_t)w + (int64_t)(lane + 1) * stride, (int64_t)W);
        const int hits = __popc(__ballot_sync(0xffffffffu, __ldg(soff + at) <= t));   // the probes that hit come first
        w += hits * stride;
        if (hits == 32) stride *= 32;
        else if (stride == 1) return w;
        else stride /= 32;
    }
}

// 32-bit halves of the words that hold a tile's row counts (16 nibbles) and its mask (128 bits)
__device__ __forceinline__ void count_entry(uint32_t* words, int tile, int row) {
    atomicAdd(words + 2 * tile + (row >> 3), 1u << (4 * (row & 7)));
}
__device__ __forceinline__ void mark_entry(uint32_t* words, int tile, int phys) {
    atomicOr(words + 4 * tile + (phys >> 5), 1u << (phys & 31));
}

// One warp per `chunk` consecutive tiles, kSub at a time, composed in shared memory; nothing waits for another
// warp.  The entries of a row that fall into the tiles are consecutive (positions ascend along a row): a few lanes
// take each of the 16 rows, eight entries of it per turn, until one lies behind the tiles; a few rows that go on are
// then taken by all lanes, one after the other.  A window that fits into a chunk is written by the warp in whose chunk
// it begins, so that only larger ones cost a search for where a chunk begins in each row.  What bounds it is the chain
// rows -> positions and values -> tile of every step, which 40 warps an SM cover.  Blocks of 128 threads that composed
// 32 tiles together took, against this: 396 us, now 323 (SR-BCRS, 2^20 nodes, 1.97 M tiles); 97 us, now 15 (47 000 nodes);
// ME-TCF of 30 000 nodes 144 us in two passes, now 31.
template <int MODE>
__global__ void __launch_bounds__(kFillThreads, 10) fill_kernel(const FillArgs p) {
    constexpr bool kIds = MODE == kFillSrbcrs || MODE == kFillMetcf || MODE == kFillMco;
    constexpr bool kMco = MODE == kMaskMco || MODE == kFillMco;
    constexpr int kWarps = kFillThreads / 32;
    // lanes of a row, rows at once; entries of a lane: eight of a row per turn.  A load touches as many lines as rows:
    // with sixteen L1 is what bounds the SR-BCRS fill, with four the turns cost too many instructions.
    constexpr int kLanes = MODE == kFillSrbcrs ? 4 : 2, kAtOnce = 32 / kLanes, kSets = kWinRows / kAtOnce, kPer = 8 / kLanes;
    constexpr unsigned kGroup = (1u << kLanes) - 1;
    constexpr int kSub = MODE == kFillSrbcrs ? 8 : 32, kWords = kMco ? 2 * kSub : kSub;
    __shared__ __align__(16) float tiles[MODE == kFillSrbcrs ? kWarps * kSub * kTileElems : 4];
    __shared__ unsigned long long word_store[MODE == kFillSrbcrs ? 1 : kWarps * kWords];
    __shared__ int32_t begin_store[MODE == kFillMetcf || MODE == kFillMco ? kWarps * kSub : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / kLanes, l = lane % kLanes, group = g * kLanes;
    float* const tile = tiles + (MODE == kFillSrbcrs ? warp * kSub * kTileElems : 0);
    unsigned long long* const words = word_store + (MODE == kFillSrbcrs ? 0 : warp * kWords);
    uint32_t* const half_words = reinterpret_cast<uint32_t*>(words);
    int32_t* const begin = begin_store + (MODE == kFillMetcf || MODE == kFillMco ? warp * kSub : 0);

    const int64_t chunk_begin = ((int64_t)blockIdx.x * kWarps + warp) * p.chunk;
    if (chunk_begin >= p.T) return;
    auto locate = [&](int64_t t) { return window_of_tile(p.soff, p.W, p.first_window[t / kFillTiles], t); };
    int w = locate(chunk_begin);
    int64_t s0 = p.soff[w], s1 = p.soff[w + 1], t = chunk_begin, chunk_end = min(p.T, chunk_begin + p.chunk);
    if (t > s0 && s1 - s0 <= p.chunk) t = s1;
    if (chunk_end < p.T) {
        const int last = locate(chunk_end);
        const int64_t b0 = p.soff[last], b1 = p.soff[last + 1];
        if (b0 < chunk_end && b1 - b0 <= p.chunk) chunk_end = b1;
    }
    if (t >= chunk_end) return;
    if (s1 <= t) {
        w = window_of_tile(p.soff, p.W, w, t);
        s0 = t;
        s1 = p.soff[w + 1];
    }
    if (MODE == kFillSrbcrs) {
        for (int i = lane; i < kSub * kTileElems / 4; i += 32) reinterpret_cast<float4*>(tile)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
    }
    // entry ee of window row rr (whose first is row_beg), at position q, in tiles from position p0 on
    auto place = [&](int rr, int row_beg, int ee, int q, float v, int p0) {
        const int lt = (q - p0) >> 3, cc = q & 7;
        if (MODE == kFillSrbcrs) {
            tile[lt * kTileElems + sw223(rr * kTileCols + cc)] = v;
            if (p.edge_to_col) p.edge_to_col[ee] = q;
            if (p.edge_to_row) p.edge_to_row[ee] = w * kWinRows + rr;
        } else if (MODE == kCountMetcf) {
            count_entry(half_words, lt, rr);
        } else if (MODE == kFillMetcf) {   // entries of earlier rows, then earlier entries of this row
            int at = begin[lt] + (rr == 0 ? 0 : nibble_sum(words[lt] & ((1ull << (4 * rr)) - 1ull)));
            for (int j = ee - 1; j >= row_beg && (__ldg(p.pos + j) >> 3) == (q >> 3); j--) at++;
            p.coo_idx[at] = sw123(rr * kTileCols + cc);
            p.out_val[at] = v;
        } else if (!(p.skip_zero && v == 0.0f)) {
            const int phys = sw123(rr * kTileCols + cc), upper = phys >> 6;
            if (MODE == kMaskMco) {
                mark_entry(half_words, lt, phys);
            } else {   // values in ascending bit order: the slot is the number of bits below
                const int below = __popcll(words[2 * lt + upper] & ((1ull << (phys & 63)) - 1ull));
                p.out_val[begin[lt] + below + (upper ? __popcll(words[2 * lt]) : 0)] = v;
            }
        }
    };
    for (;;) {
        int beg[kSets], e[kSets], end[kSets];
#pragma unroll
        for (int k = 0; k < kSets; k++) {
            e[k] = beg[k] = __ldg(p.rows + w * kWinRows + kAtOnce * k + g);
            end[k] = __ldg(p.rows + w * kWinRows + kAtOnce * k + g + 1);
        }
        const int base = kIds || t > s0 ? __ldg(p.rows + w * kWinRows) : 0, n_cols = kIds ? __ldg(p.distinct + w) : 0;
        const int64_t te = min(s1, chunk_end);
        const int64_t next_s1 = te < chunk_end ? p.soff[w + 2] : 0;
        if (t > s0) {   // the chunk begins inside this window: first entry of every row at or after tile t
            // `first` columns come before it, all of them in the row but for those that only other rows have
            const int first = (int)(t - s0) * kTileCols, all = __ldg(p.rows + w * kWinRows + kWinRows) - base;
#pragma unroll
            for (int k = 0; k < kSets; k++) {
                int at = min(end[k], beg[k] + max(0, first - (all - (end[k] - beg[k]))));
                for (int left = min(end[k], beg[k] + first) - at; __any_sync(0xffffffffu, left > 0);) {   // kLanes + 1 parts
                    const int stride = left / (kLanes + 1) + 1, probe = (l + 1) * stride;
                    const bool below = left > 0 && probe <= left && __ldg(p.pos + at + probe - 1) < first;
                    const int hits = __popc((__ballot_sync(0xffffffffu, below) >> group) & kGroup);   // the probes that hit come first
                    at += hits * stride;
                    left = min(hits == kLanes ? left : stride - 1, left - hits * stride);
                }
                e[k] = at;
            }
        }
        for (int64_t c = t; c < te; c += kSub) {
            const int nt = (int)min((int64_t)kSub, te - c);
            const int p0 = (int)(c - s0) * kTileCols, limit = p0 + nt * kTileCols;
            if (MODE == kCountMetcf) {
                words[lane] = 0ull;
            } else if (MODE == kMaskMco) {
                words[lane] = words[lane + 32] = 0ull;
            } else if (MODE == kFillMetcf) {
                if (lane < nt) { words[lane] = p.tile_rows[c + lane]; begin[lane] = p.off[2 * (c + lane)]; }
            } else if (MODE == kFillMco) {
                for (int i = lane; i < 2 * nt; i += 32) words[i] = p.masks[2 * c + i];
                if (lane < nt) begin[lane] = p.off[c + lane];
            }
            if (kIds) {   // tail slots of a window repeat its last column, or are 0 (ME-TCF)
                for (int i = lane; i < nt * kTileCols; i += 32) {
                    const int q = p0 + i;
                    p.sidx[c * kTileCols + i] = (MODE == kFillMetcf && q >= n_cols) ? 0 : __ldg(p.cols + base + min(q, n_cols - 1));
                }
            }
            if (MODE != kFillSrbcrs) __syncwarp();
            unsigned open = (1u << kSets) - 1;   // this lane's rows that may have more
            for (int turn = 1;; turn++) {
                int q[kSets][kPer];
                float v[kSets][kPer];
#pragma unroll
                for (int k = 0; k < kSets; k++)
#pragma unroll
                    for (int j = 0; j < kPer; j++) {
                        const int i = e[k] + l + kLanes * j;
                        const bool have = (open >> k & 1) && i < end[k];
                        q[k][j] = have ? __ldg(p.pos + i) : 0x7fffffff;
                        v[k][j] = p.values && have ? __ldg(p.values + i) : 1.0f;
                    }
                int rows_open = 0;
#pragma unroll
                for (int k = 0; k < kSets; k++) {
                    int n = 0;
#pragma unroll
                    for (int j = 0; j < kPer; j++) {
                        const bool in = q[k][j] < limit;
                        if (in) place(kAtOnce * k + g, beg[k], e[k] + l + kLanes * j, q[k][j], v[k][j], p0);
                        n += __popc((__ballot_sync(0xffffffffu, in) >> group) & kGroup);
                    }
                    e[k] += n;
                    if (n < kLanes * kPer) open &= ~(1u << k);
                    rows_open += __popc(__ballot_sync(0xffffffffu, n == kLanes * kPer)) / kLanes;
                }
                if (rows_open == 0) break;
                if (rows_open > turn) continue;
                // few rows that go on and on: all lanes on one after the other
#pragma unroll
                for (int k = 0; k < kSets; k++) {
                    for (unsigned left = __ballot_sync(0xffffffffu, (open >> k & 1) && l == 0); left != 0; left &= left - 1) {
                        const int from = __ffs(left) - 1, row_beg = __shfl_sync(0xffffffffu, beg[k], from), row_end = __shfl_sync(0xffffffffu, end[k], from);
                        int at = __shfl_sync(0xffffffffu, e[k], from), taken;
                        do {
                            int q2[2];
                            float v2[2];
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                const int i = at + lane + 32 * j;
                                q2[j] = i < row_end ? __ldg(p.pos + i) : 0x7fffffff;
                                v2[j] = p.values && i < row_end ? __ldg(p.values + i) : 1.0f;
                            }
                            taken = 0;
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                if (q2[j] < limit) place(kAtOnce * k + from / kLanes, row_beg, at + lane + 32 * j, q2[j], v2[j], p0);
                                taken += __popc(__ballot_sync(0xffffffffu, q2[j] < limit));
                            }
                            at += taken;
                        } while (taken == 64);
                        if (group == from) e[k] = at;
                    }
                }
                break;
            }
            __syncwarp();
            if (MODE == kFillSrbcrs) {   // and clear what was read for the next tiles
                float4* out = reinterpret_cast<float4*>(p.block_val + c * kTileElems);
#pragma unroll
                for (int i = 0; i < kSub; i++) {
                    if (i >= nt) break;
                    float4* from = reinterpret_cast<float4*>(tile) + i * 32 + lane;
                    const float4 v = *from;
                    if (p.whole_vectors) {
                        out[i * 32 + lane] = v;
                    } else {
                        float* at = p.block_val + (c + i) * kTileElems + 4 * lane;
                        at[0] = v.x; at[1] = v.y; at[2] = v.z; at[3] = v.w;
                    }
                    *from = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else if (MODE == kCountMetcf) {
                if (lane < nt) p.tile_rows[c + lane] = words[lane];
            } else if (MODE == kMaskMco) {
                for (int i = lane; i < 2 * nt; i += 32) p.masks[2 * c + i] = words[i];
            } else if (lane < nt) {   // the padding at the end of the tile's run
                const int cnt = MODE == kFillMetcf ? nibble_sum(words[lane]) : __popcll(words[2 * lane]) + __popcll(words[2 * lane + 1]);
                const int pad = MODE == kFillMetcf ? (cnt + 7) & ~7 : (cnt + 3) & ~3;
                for (int i = cnt; i < pad; i++) {
                    if (MODE == kFillMetcf) p.coo_idx[begin[lane] + i] = 0;
                    p.out_val[begin[lane] + i] = 0.f;
                }
            }
            __syncwarp();
        }
        t = te;
        if (t == chunk_end) return;
        w++;   // on to the next window with tiles
        s0 = s1;
        s1 = next_s1;
        if (s1 == s0) {
            w = window_of_tile(p.soff, p.W, w, t);
            s1 = p.soff[w + 1];
        }
    }
}

__global__ void block_partition_kernel(const int32_t* __restrict__ val_soff, int32_t W, int32_t* __restrict__ bp) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < W) bp[w] = val_soff[w + 1] - val_soff[w];
}

struct TilePadIn {
    const unsigned long long* tile_rows;
    __device__ int32_t operator()(int64_t t) const { return (nibble_sum(tile_rows[t]) + 7) & ~7; }
};
// also the closing entry, behind the last tile
struct CooOffOut {
    const unsigned long long* tile_rows;
    int32_t* off;
    int64_t T;
    HostWords* host;
    __device__ void operator()(int64_t t, int64_t before, int32_t v) const {
        off[2 * t] = (int32_t)before;
        off[2 * t + 1] = (int32_t)before + nibble_sum(tile_rows[t]);
        if (t == T - 1) {
            off[2 * T] = (int32_t)(before + v);
            host->total = before + v;
        }
    }
};
struct McoCountIn {
    const unsigned long long* masks;
    __device__ int32_t operator()(int64_t t) const { return (__popcll(masks[2 * t]) + __popcll(masks[2 * t + 1]) + 3) & ~3; }
};
struct McoOffOut {
    int32_t* off;
    int64_t T;
    HostWords* host;
    __device__ void operator()(int64_t t, int64_t before, int32_t v) const {
        off[t] = (int32_t)before;
        if (t == T - 1) {
            off[T] = (int32_t)(before + v);
            host->total = before + v;
        }
    }
};

template <int MODE>
static int launch_fill(const FillArgs& a, cudaStream_t st) {
    fill_kernel<MODE><<<blocks_for(a.T, a.chunk * (kFillThreads / 32)), kFillThreads, 0, st>>>(a);
    MASK_CUDA_TRY(cudaGetLastError());
    return MASK_OK;
}

static FillArgs fill_args(const PackScratch& s, int32_t M, const float* d_values, const int32_t* d_val_soff, int64_t T) {
    FillArgs a{};
    a.W = window_count(M);
    // a chunk costs its searches, so it is as long as leaves the resident warps (48 an SM) one each
    a.chunk = kFillTiles;
    while (a.chunk > 16 && T < (int64_t)48 * sm_count() * a.chunk) a.chunk /= 2;
    a.rows = s.rows;
    a.cols = s.cols;
    a.distinct = s.distinct;
    a.values = d_values;
    a.pos = s.pos;
    a.soff = d_val_soff;
    a.first_window = s.first_window;
    a.T = T;
    return a;
}

}  // namespace mask

extern "C" size_t mask_pack_scratch_bytes(int32_t M, int64_t nnz) {
    if (M < 1 || nnz < 0) return 0;
    return mask::carve(nullptr, M, nnz).bytes;
}

extern "C" int mask_pack_analyze(const int32_t* d_rowptr, const int32_t* d_colind, int32_t M, int32_t K, int64_t nnz,
                                 void* d_scratch, size_t scratch_bytes, int32_t* d_val_soff, int64_t* h_T, void* stream) {
    using namespace mask;
    MASK_REQUIRE(d_rowptr && d_val_soff && h_T, "rowptr, val_soff or h_T is NULL");
    MASK_REQUIRE(M >= 1 && K >= 1 && nnz >= 0, "M and K must be positive, nnz non-negative");
    MASK_REQUIRE(nnz == 0 || d_colind, "colind is NULL");
    if (nnz >= ((int64_t)1 << 31) - kScanChunk) return fail(MASK_ERR_INDEX_OVERFLOW, "nnz does not fit int32");
    MASK_REQUIRE(d_scratch != nullptr, "scratch is NULL");
    MASK_REQUIRE((reinterpret_cast<uintptr_t>(d_scratch) & 255) == 0, "scratch must be 256-byte aligned");
    PackScratch s = carve(d_scratch, M, nnz);
    if (scratch_bytes < s.bytes) return fail(MASK_ERR_SCRATCH_TOO_SMALL, "scratch smaller than mask_pack_scratch_bytes");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int W = window_count(M);
    MASK_CUDA_TRY(cudaMemsetAsync(s.status, 0, 64, st));
    // a key is the column and the entry's index within the window
    if (K <= (1 << (32 - kSortIdxBits)))
        condense_kernel<uint32_t><<<(unsigned)W, 32, 0, st>>>(d_rowptr, d_colind, M, K, W, s.pos, s.cols, s.rows, s.distinct, s.big_list, s.hub_list, s.status);
    else
        condense_kernel<unsigned long long><<<(unsigned)W, 32, 0, st>>>(d_rowptr, d_colind, M, K, W, s.pos, s.cols, s.rows, s.distinct, s.big_list, s.hub_list, s.status);
    MASK_CUDA_TRY(cudaGetLastError());
    if (nnz > kHubMin) {
        const int most_bits = K > kHubBlocks * kHubBits && K <= kHubBlocks * kHubBitsWide ? kHubBitsWide : kHubBits;
        const int span = (int)std::min<int64_t>(((int64_t)K + 4095) / 4096 * 4096, most_bits);   // columns a block marks at a time
        const int smem = mark_set_bytes(span);
        static std::atomic<uint64_t> opted_in;
        const int rc = opt_in_shared_memory(reinterpret_cast<const void*>(condense_hub_kernel), mark_set_bytes(kHubBitsWide), opted_in);
        if (rc != MASK_OK) return rc;
        const int64_t most = std::min<int64_t>(W, nnz / kHubMin);
        condense_hub_kernel<<<(unsigned)(kHubBlocks * std::min<int64_t>(most, std::max(1, (most_bits == kHubBits ? 2 : 1) * sm_count() / kHubBlocks))), kHubThreads, smem, st>>>(
            d_rowptr, d_colind, M, K, span, s.pos, s.cols, s.distinct, s.hub_list, s.status);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    if (nnz > kSortMax) {
        constexpr int kSmem = mark_set_bytes(kBigBits);
        static std::atomic<uint64_t> opted_in;
        int rc = opt_in_shared_memory(reinterpret_cast<const void*>(condense_big_kernel), kSmem, opted_in);
        if (rc != MASK_OK) return rc;
        const int64_t most = std::min<int64_t>(W, nnz / kSortMax);
        const dim3 grid((unsigned)std::min<int64_t>(most, 2 * sm_count()));
        if (nnz > kHubMin) {   // independent of the hub windows: starts as their blocks leave
            rc = launch_overlapped(condense_big_kernel, grid, kBigThreads, kSmem, st, d_rowptr, d_colind, M, K, s.pos, s.cols, s.distinct, s.big_list, s.status);
            if (rc != MASK_OK) return rc;
        } else {
            condense_big_kernel<<<grid, kBigThreads, kSmem, st>>>(d_rowptr, d_colind, M, K, s.pos, s.cols, s.distinct, s.big_list, s.status);
            MASK_CUDA_TRY(cudaGetLastError());
        }
    }
    HostStage stage;
    int rc = stage.get(sizeof(HostWords));
    if (rc != MASK_OK) return rc;
    HostWords* host = stage.as<HostWords>();
    rc = device_scan(WindowTilesIn{s.distinct, W}, SoffOut{d_val_soff, s.first_window, W, s.status, host}, (int64_t)W + 1, s.spine, st);
    const cudaError_t e = cudaStreamSynchronize(st);   // also after a failure: a kernel may still write the host's words
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(e);
    if (host->status & 2) return fail(MASK_ERR_COLUMN_RANGE, "a column id is outside [0, K)");
    if (host->status & 1) return fail(MASK_ERR_UNSORTED_ROWS, "CSR rows must hold strictly ascending column ids");
    const int64_t T = host->total;
    if (T >= (int64_t)1 << 31 || T * kTileElems < 0) return fail(MASK_ERR_INDEX_OVERFLOW, "tile count does not fit int32");
    *h_T = T;
    return MASK_OK;
}

extern "C" int mask_srbcrs_fill(const int32_t* d_rowptr, const int32_t* d_colind, const float* d_values, int32_t M,
                                int64_t nnz, const void* d_scratch, const int32_t* d_val_soff, int64_t T,
                                int32_t* d_val_sidx, float* d_val_block_val, int32_t* d_block_partition,
                                int32_t* d_edge_to_col, int32_t* d_edge_to_row, void* stream) {
    using namespace mask;
    (void)d_colind;
    MASK_REQUIRE(d_rowptr && d_scratch && d_val_soff, "rowptr, scratch or val_soff is NULL");
    MASK_REQUIRE(M >= 1 && nnz >= 0 && T >= 0, "bad sizes");
    MASK_REQUIRE(nnz == 0 || (d_values && T > 0), "values is NULL or T is 0 for a non-empty matrix");
    MASK_REQUIRE(T == 0 || (d_val_sidx && d_val_block_val), "output arrays are NULL");
    PackScratch s = carve(const_cast<void*>(d_scratch), M, nnz);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int W = window_count(M);
    if (T > 0) {
        FillArgs a = fill_args(s, M, d_values, d_val_soff, T);
        a.sidx = d_val_sidx;
        a.block_val = d_val_block_val;
        a.whole_vectors = (reinterpret_cast<uintptr_t>(d_val_block_val) & 15) == 0;
        a.edge_to_col = d_edge_to_col;
        a.edge_to_row = d_edge_to_row;
        int rc = launch_fill<kFillSrbcrs>(a, st);
        if (rc != MASK_OK) return rc;
    }
    if (d_block_partition) {
        block_partition_kernel<<<blocks_for(W, 256), 256, 0, st>>>(d_val_soff, W, d_block_partition);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    return MASK_OK;
}

extern "C" int mask_metcf_offsets(const int32_t* d_rowptr, int32_t M, int64_t nnz, const void* d_scratch,
                                  const int32_t* d_val_soff, int64_t T, int32_t* d_val_coo_off, uint64_t* d_tile_rows,
                                  int64_t* h_nnz_pad, void* stream) {
    using namespace mask;
    (void)d_rowptr;
    MASK_REQUIRE(d_scratch && d_val_soff && d_val_coo_off && h_nnz_pad, "NULL argument");
    MASK_REQUIRE(M >= 1 && nnz >= 0 && T >= 0, "bad sizes");
    MASK_REQUIRE(T == 0 || d_tile_rows, "tile_rows is NULL");
    PackScratch s = carve(const_cast<void*>(d_scratch), M, nnz);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto* rows = reinterpret_cast<unsigned long long*>(d_tile_rows);
    *h_nnz_pad = 0;
    if (T == 0) {
        MASK_CUDA_TRY(cudaMemsetAsync(d_val_coo_off, 0, 4, st));
        return MASK_OK;
    }
    FillArgs a = fill_args(s, M, nullptr, d_val_soff, T);
    a.tile_rows = rows;
    int rc = launch_fill<kCountMetcf>(a, st);
    if (rc != MASK_OK) return rc;
    // the spine is sized for max(nnz, W+1) items and T <= nnz
    HostStage stage;
    rc = stage.get(sizeof(HostWords));
    if (rc != MASK_OK) return rc;
    rc = device_scan(TilePadIn{rows}, CooOffOut{rows, d_val_coo_off, T, stage.as<HostWords>()}, T, s.spine, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(e);
    const int64_t total = stage.as<HostWords>()->total;
    if (total >= (int64_t)1 << 31) return fail(MASK_ERR_INDEX_OVERFLOW, "nnz_pad does not fit int32");
    *h_nnz_pad = total;
    return MASK_OK;
}

extern "C" int mask_metcf_fill(const int32_t* d_rowptr, const int32_t* d_colind, const float* d_values, int32_t M,
                               int64_t nnz, const void* d_scratch, const int32_t* d_val_soff, int64_t T,
                               const int32_t* d_val_coo_off, const uint64_t* d_tile_rows, int64_t nnz_pad,
                               int32_t* d_val_sidx, int32_t* d_val_coo_idx, float* d_val_coo_val, void* stream) {
    using namespace mask;
    (void)d_colind;
    MASK_REQUIRE(d_rowptr && d_scratch && d_val_soff && d_val_coo_off, "NULL argument");
    MASK_REQUIRE(M >= 1 && nnz >= 0 && T >= 0 && nnz_pad >= 0, "bad sizes");
    MASK_REQUIRE(T == 0 || (d_val_sidx && d_tile_rows), "output arrays are NULL");
    MASK_REQUIRE(nnz_pad == 0 || (d_val_coo_idx && d_val_coo_val), "output arrays are NULL");
    PackScratch s = carve(const_cast<void*>(d_scratch), M, nnz);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (T == 0) return MASK_OK;
    FillArgs a = fill_args(s, M, d_values, d_val_soff, T);
    a.sidx = d_val_sidx;
    a.tile_rows = const_cast<unsigned long long*>(reinterpret_cast<const unsigned long long*>(d_tile_rows));
    a.off = d_val_coo_off;
    a.coo_idx = d_val_coo_idx;
    a.out_val = d_val_coo_val;
    return launch_fill<kFillMetcf>(a, st);
}

extern "C" int mask_mco_offsets(const float* d_values, int32_t M, int64_t nnz, const void* d_scratch, const int32_t* d_val_soff,
                                int64_t T, int skip_zero_values, uint64_t* d_val_mco_mask, int32_t* d_val_mco_off,
                                int64_t* h_nval, void* stream) {
    using namespace mask;
    MASK_REQUIRE(d_scratch && d_val_soff && d_val_mco_off && h_nval, "NULL argument");
    MASK_REQUIRE(M >= 1 && nnz >= 0 && T >= 0, "bad sizes");
    MASK_REQUIRE(T == 0 || d_val_mco_mask, "val_mco_mask is NULL");
    PackScratch s = carve(const_cast<void*>(d_scratch), M, nnz);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto* masks = reinterpret_cast<unsigned long long*>(d_val_mco_mask);
    *h_nval = 0;
    if (T == 0) {
        MASK_CUDA_TRY(cudaMemsetAsync(d_val_mco_off, 0, 4, st));
        return MASK_OK;
    }
    FillArgs a = fill_args(s, M, d_values, d_val_soff, T);
    a.skip_zero = skip_zero_values;
    a.masks = masks;
    int rc = launch_fill<kMaskMco>(a, st);
    if (rc != MASK_OK) return rc;
    HostStage stage;
    rc = stage.get(sizeof(HostWords));
    if (rc != MASK_OK) return rc;
    rc = device_scan(McoCountIn{masks}, McoOffOut{d_val_mco_off, T, stage.as<HostWords>()}, T, s.spine, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(e);
    const int64_t total = stage.as<HostWords>()->total;
    if (total >= (int64_t)1 << 31) return fail(MASK_ERR_INDEX_OVERFLOW, "value count does not fit int32");
    *h_nval = total;
    return MASK_OK;
}

extern "C" int mask_mco_fill(const int32_t* d_rowptr, const float* d_values, int32_t M, int64_t nnz, const void* d_scratch,
                             const int32_t* d_val_soff, int64_t T, int skip_zero_values, const uint64_t* d_val_mco_mask,
                             const int32_t* d_val_mco_off, int64_t nval, int32_t* d_val_sidx, float* d_val_mco_val,
                             void* stream) {
    using namespace mask;
    MASK_REQUIRE(d_rowptr && d_scratch && d_val_soff && d_val_mco_off, "NULL argument");
    MASK_REQUIRE(M >= 1 && nnz >= 0 && T >= 0 && nval >= 0, "bad sizes");
    MASK_REQUIRE(T == 0 || (d_val_sidx && d_val_mco_mask), "output arrays are NULL");
    MASK_REQUIRE(nval == 0 || d_val_mco_val, "val_mco_val is NULL");
    PackScratch s = carve(const_cast<void*>(d_scratch), M, nnz);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (T == 0) return MASK_OK;
    FillArgs a = fill_args(s, M, d_values, d_val_soff, T);
    a.skip_zero = skip_zero_values;
    a.masks = const_cast<unsigned long long*>(reinterpret_cast<const unsigned long long*>(d_val_mco_mask));
    a.off = d_val_mco_off;
    a.sidx = d_val_sidx;
    a.out_val = d_val_mco_val;
    return launch_fill<kFillMco>(a, st);
}
