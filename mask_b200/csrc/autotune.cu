// Column features of a packed matrix, computed on the device, and the plan decisions keyed on them.
//
// The reference leaves these decisions to an LLM strategy agent working from the statistics of its
// featurizer (examples/src_fp32/dtc/testbed/featurize_mtx.cu:298-401: tiles per window, unique
// columns, density, top-5 window share) and a catalogue of knobs (python/sparsene/op_gen/
// strategy_agent.py:414-528: tile width, placement, stages); here they are a fixed rule over
// measured features.  The window statistics (mask_features) come from a host copy of val_soff; the
// column side is measured on the device, from the 8 T entries of val_sidx:
//   * band: how far the gathered rows of B lie from the diagonal position of their window (a stencil
//     or banded matrix keeps them within a few thousand rows, so neighbouring windows share them and
//     they stay in L2 whatever their width);
//   * hub share: what fraction of all gathers goes to the most gathered columns whose rows of B fit
//     half the L2 -- at the full row width and at a half and a quarter of it.  On a power-law graph
//     that fraction is what L2 can serve; where a narrower row raises it markedly, sweeping the matrix
//     once per 256 columns instead of once per 512 saves more DRAM traffic (rows of B) than it costs
//     (tile values and ids read twice).
#include <algorithm>
#include <functional>
#include <vector>

#include "common.cuh"
#include "column_stats.h"

namespace mask {

namespace {

constexpr int kBandBuckets = 33;   // bucket b: distances in [2^(b-1), 2^b), bucket 0: distance 0
constexpr int kCountBins = 8192;   // columns gathered fewer times than this are counted by that number, the others listed

struct StatsHead {                 // what goes back to the host in one copy, followed by the list
    unsigned long long band[kBandBuckets + 1];   // last entry: gathers within local_rows of the diagonal
    uint32_t bins[kCountBins];     // columns by number of gathers
    uint32_t listed;
    int32_t local;                 // local_share >= kLocalShare, for the kernels that group the tiles
    uint32_t top_bin;              // largest of them that is not empty
    uint32_t pad;
};
constexpr double kLocalShare = 0.9;

// One thread per tile finds its window (a block's 256 tiles lie in few windows, so the search runs between the windows of
// its first and last tile); then a warp takes the ids of its 32 tiles as they lie, 32 at a time.  Ids ascend within a window, so
// those of the most gathered columns, where they are neighbours, arrive at the L2 as one request for a sector of 8 counters: with one
// thread counting the 8 ids of its tile they were 8 requests (power-law graph with 2^20 nodes, 15.8 M ids: 180 us, now 103 to 118;
// counting into 2, 4 or 8 arrays in turn, added up afterwards, 103, 103 and 98).  Ids of a warp fall into the same few distance
// buckets: the lanes that share the first one's are counted together.  (A histogram per thread instead of shared atomics, and
// blocks that stay instead of one per 256 tiles: 126 to 156 us.)
__global__ void __launch_bounds__(256) column_stats_kernel(const int32_t* __restrict__ soff, const int32_t* __restrict__ sidx, int32_t W,
                                                           int64_t T, int32_t M, int32_t K, int64_t local_rows,
                                                           uint32_t* __restrict__ counts, StatsHead* __restrict__ head) {
    __shared__ unsigned int hist[kBandBuckets + 1];
    __shared__ int range[2];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x <= kBandBuckets) hist[threadIdx.x] = 0;
    const int64_t t0 = (int64_t)blockIdx.x * 256, t = t0 + threadIdx.x;
    if (threadIdx.x < 2) {
        const int64_t key = threadIdx.x == 0 ? t0 : (t0 + 255 < T ? t0 + 255 : T - 1);
        int lo = 0, hi = W;   // last window whose first tile is <= key
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((int64_t)soff[mid] <= key) lo = mid; else hi = mid;
        }
        range[threadIdx.x] = lo;
    }
    __syncthreads();
    int lo = range[0], hi = range[1] + 1;
    int64_t diag = 0;
    if (t < T) {
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((int64_t)soff[mid] <= t) lo = mid; else hi = mid;
        }
        diag = (int64_t)lo * kWinRows * K / M;
    }
    const int64_t first = (t - lane) * kTileCols + lane, end = T * kTileCols;
    int local = 0;
    int ids[kTileCols];
#pragma unroll
    for (int j = 0; j < kTileCols; j++) ids[j] = first + 32 * j < end ? __ldg(sidx + first + 32 * j) : -1;
#pragma unroll
    for (int j = 0; j < kTileCols; j++) {
        const int id = ids[j];
        const int64_t at = __shfl_sync(0xffffffffu, diag, 4 * j + (lane >> 3));   // of tile 4 j + lane / 8
        const bool ok = id >= 0 && id < K;
        if (ok) atomicAdd(&counts[id], 1u);
        const int64_t d = id > at ? id - at : at - id;
        const int bucket = !ok ? -1 : (d == 0 ? 0 : 64 - __clzll((unsigned long long)d));
        const int lead = __shfl_sync(0xffffffffu, bucket, 0);
        const unsigned same = __ballot_sync(0xffffffffu, bucket == lead);
        if (lane == 0) { if (ok) atomicAdd(&hist[bucket], (unsigned)__popc(same)); }
        else if (ok && bucket != lead) atomicAdd(&hist[bucket], 1u);
        local += ok && d <= local_rows;
    }
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0 && local) atomicAdd(&hist[kBandBuckets], (unsigned)local);
    __syncthreads();
    if (threadIdx.x <= kBandBuckets && hist[threadIdx.x]) atomicAdd(&head->band[threadIdx.x], (unsigned long long)hist[threadIdx.x]);
}

// columns by number of gathers; those with kCountBins and more, one by one
__global__ void __launch_bounds__(512) count_bins_kernel(const uint32_t* __restrict__ counts, int32_t K, StatsHead* __restrict__ head,
                                                         uint32_t* __restrict__ list) {
    __shared__ uint32_t bins[kCountBins];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int b = 0; b < kBandBuckets; b++) total += head->band[b];
        head->local = total && (double)head->band[kBandBuckets] / (double)total >= kLocalShare;
    }
    for (int i = threadIdx.x; i < kCountBins; i += 512) bins[i] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * 512;
    for (int64_t i0 = (int64_t)blockIdx.x * 512 + threadIdx.x; i0 < K; i0 += 4 * stride) {
        uint32_t c[4];   // four columns at once: the loads do not wait for one another
#pragma unroll
        for (int k = 0; k < 4; k++) c[k] = i0 + k * stride < K ? counts[i0 + k * stride] : 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k * stride >= K) break;
            if (c[k] < (uint32_t)kCountBins) atomicAdd(&bins[c[k]], 1u);
            else list[atomicAdd(&head->listed, 1u)] = c[k];
        }
    }
    __syncthreads();
    int top = 0;
    for (int i = threadIdx.x; i < kCountBins; i += 512)
        if (bins[i]) {
            atomicAdd(&head->bins[i], bins[i]);
            top = i;
        }
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((threadIdx.x & 31) == 0 && top) atomicMax(&head->top_bin, (uint32_t)top);
}

}  // namespace

int ColumnStatsJob::enqueue(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int32_t N, cudaStream_t st) {
    int dev = 0;
    MASK_CUDA_TRY(cudaGetDevice(&dev));
    MASK_CUDA_TRY(cudaDeviceGetAttribute(&l2_, cudaDevAttrL2CacheSize, dev));
    K_ = K;
    N_ = N;
    T_ = T;
    if (T == 0) return MASK_OK;
    const int32_t W = window_count(M);
    // one allocation: what goes back to the host (with room for every column that can be listed), then counts
    const int64_t most_listed = std::min<int64_t>(K, T * kTileCols / kCountBins) + 1;
    const size_t counts_at = (sizeof(StatsHead) + (size_t)most_listed * 4 + 15) & ~(size_t)15;
    const size_t bytes = counts_at + (size_t)K * 4;
    int rc = buf_.alloc(bytes, st);
    if (rc == MASK_OK) rc = host_.get(counts_at);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cudaMemsetAsync(buf_.p, 0, bytes, st));
    // "local": a band of windows keeps rows of B alive that take at most half the L2 at this row width
    const int width0 = std::min(N, 512);
    local_rows_ = (int32_t)std::min<int64_t>(K, std::max<int64_t>(0, ((int64_t)(l2_ / 2) / ((int64_t)width0 * 4) - kWinRows) / 2));
    uint32_t* counts = buf_.as<uint32_t>(counts_at);
    d_local_ = &buf_.as<StatsHead>()->local;
    column_stats_kernel<<<(unsigned)((T + 255) / 256), 256, 0, st>>>(d_val_soff, d_val_sidx, W, T, M, K, (int64_t)local_rows_, counts,
                                                                    buf_.as<StatsHead>());
    MASK_CUDA_TRY(cudaGetLastError());
    const unsigned bin_blocks = (unsigned)std::min<int64_t>(((int64_t)K + 4095) / 4096, sm_count());
    count_bins_kernel<<<bin_blocks, 512, 0, st>>>(counts, K, buf_.as<StatsHead>(), buf_.as<uint32_t>(sizeof(StatsHead)));
    MASK_CUDA_TRY(cudaGetLastError());
    MASK_CUDA_TRY(cudaMemcpyAsync(host_.as<void>(), buf_.p, counts_at, cudaMemcpyDeviceToHost, st));
    return MASK_OK;
}

void ColumnStatsJob::finish(mask_column_features* out) const {
    *out = mask_column_features{};
    out->l2_bytes = l2_;
    out->gathers = T_ * kTileCols;
    if (T_ == 0) return;
    out->local_rows = local_rows_;
    const StatsHead& head = *host_.as<StatsHead>();
    const unsigned long long* h = head.band;
    const uint32_t* list = reinterpret_cast<const uint32_t*>(&head + 1);
    out->distinct_columns = (int32_t)(K_ - (int64_t)head.bins[0]);
    // gathers that go to the most gathered columns: the listed ones first, then bin by bin
    std::vector<uint32_t> top(list, list + head.listed);
    std::sort(top.begin(), top.end(), std::greater<uint32_t>());
    unsigned long long reach[3] = {0, 0, 0};
    int64_t left[3];
    for (int i = 0; i < 3; i++) {
        const int width = std::min(N_, 512 >> i);                               // columns of one gathered row at 4, 2, 1 slabs
        const int64_t rows = std::max<int64_t>(1, (int64_t)(l2_ / 2) / ((int64_t)width * 4));
        out->hub_columns[i] = (int32_t)std::min<int64_t>(rows, K_);
        left[i] = out->hub_columns[i];
        for (size_t j = 0; j < top.size() && left[i] > 0; j++, left[i]--) reach[i] += top[j];
    }
    for (uint32_t b = head.top_bin; b > 0; b--) {
        if (head.bins[b] == 0) continue;
        for (int i = 0; i < 3; i++) {
            const int64_t take = std::min<int64_t>(left[i], head.bins[b]);
            reach[i] += (unsigned long long)take * b;
            left[i] -= take;
        }
    }
    unsigned long long total = 0;
    for (int b = 0; b < kBandBuckets; b++) total += h[b];
    for (int i = 0; i < 3; i++) out->hub_share[i] = total ? (double)reach[i] / (double)total : 0.0;
    out->local_share = total ? (double)h[kBandBuckets] / (double)total : 1.0;
    auto percentile = [&](double q) -> int32_t {
        unsigned long long run = 0;
        for (int b = 0; b < kBandBuckets; b++) {
            run += h[b];
            if ((double)run >= q * (double)total) return b == 0 ? 0 : (int32_t)std::min<int64_t>((int64_t)1 << b, (int64_t)K_);
        }
        return K_;
    };
    out->band_p50 = percentile(0.50);
    out->band_p90 = percentile(0.90);
}

}  // namespace mask

extern "C" int mask_features_columns(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int32_t N,
                                     mask_column_features* out, void* stream) {
    using namespace mask;
    MASK_REQUIRE(out != nullptr && d_val_soff != nullptr && M >= 1 && K >= 1 && T >= 0 && N >= 1, "bad arguments");
    MASK_REQUIRE(T == 0 || d_val_sidx != nullptr, "val_sidx is NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ColumnStatsJob job;
    int rc = job.enqueue(d_val_soff, d_val_sidx, M, K, T, N, st);
    const cudaError_t e = cudaStreamSynchronize(st);   // also after a failure: the copy may be in flight
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(e);
    return without_exceptions([&] { job.finish(out); return MASK_OK; });
}

namespace mask {

// The plan table.  Keyed on: does the matrix keep its gathers local (band), and if not, how much more
// of them L2 can serve when a gathered row is half as wide (hub shares).  Chooses the number of
// 128-column slabs per column block for wide (N > 256) and medium (128 < N <= 256) products; narrow
// products have one slab.  Thresholds fitted on the five benchmark configurations (27-point stencil
// and uniform-random: 4 slabs; power-law graphs with 2^21 and 2^22 nodes: 2 slabs, 3-5 % faster than
// 4; 2^20 nodes: a tie).
void choose_plan_parameters(mask_plan* plan, const mask_column_features& f) {
    plan->col_features = f;
    plan->has_col_features = 1;
    const double half_l2 = 0.5 * (double)f.l2_bytes;
    const double b_bytes = (double)f.distinct_columns * 4.0 * 512.0;
    const bool local = f.local_share >= kLocalShare || b_bytes <= half_l2;   // the gathers stay near the diagonal, or all of B fits
    // hub-heavy (a quarter of the gathers already fit at full width) and markedly more fits at half width
    const bool narrower_rows_pay = !local && b_bytes > 8.0 * half_l2 && f.hub_share[0] >= 0.25 && f.hub_share[1] - f.hub_share[0] >= 0.02;
    plan->nslab = narrower_rows_pay ? 2 : 4;
    plan->local = f.local_share >= kLocalShare;
    plan->two_slabs_kept = plan->nslab == 2 && b_bytes >= 8.0 * f.l2_bytes && b_bytes < 12.0 * f.l2_bytes;
}

}  // namespace mask

extern "C" int mask_plan_autotune(mask_plan* plan, const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t K, void* stream) {
    using namespace mask;
    MASK_REQUIRE(plan != nullptr, "plan is NULL");
    mask_column_features f;
    int rc = mask_features_columns(d_val_soff, d_val_sidx, plan->M, K, plan->T, 512, &f, stream);
    if (rc != MASK_OK) return rc;
    choose_plan_parameters(plan, f);
    return MASK_OK;
}

extern "C" int mask_plan_column_features(const mask_plan* plan, mask_column_features* out, int32_t* nslab_wide) {
    using namespace mask;
    MASK_REQUIRE(plan != nullptr && out != nullptr, "NULL argument");
    if (!plan->has_col_features) return fail(MASK_ERR_INVALID_ARGUMENT, "mask_plan_autotune has not run on this plan");
    *out = plan->col_features;
    if (nslab_wide) *nslab_wide = plan->nslab;
    return MASK_OK;
}
