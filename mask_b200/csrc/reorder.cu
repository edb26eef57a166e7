// Row reorders of the Format-DSL host bridge, computed on the device, and the device-side CSR row
// permutation.
//
// The bridge (examples/src_fp32/acc/testbed/custom_format_e2e.cu:163-347) defines three orders by
// sequential host algorithms whose tie-breaks are part of the result; here each is restated as the
// data-parallel computation that yields the same permutation:
//   first_col_sort  key(row) = smallest in-range column (K for none); stable radix sort by key.
//   jaccard_greedy  signature(row) = min over its columns of a 64-bit mix; rows ranked by
//                   (signature, first column, id) with two stable radix sorts; the ranking is cut into
//                   buckets of 64 and one thread block per bucket runs the greedy chain (next = the
//                   remaining row most similar to the last one, ties to the smaller id), every
//                   similarity a warp-wide intersection count by binary search.
//   row_rcm         reverse Cuthill-McKee.  The sequential queue order is reproduced level by level:
//                   a node's parent is the EARLIEST queue position among its visited neighbours
//                   (atomicMin), the children of a parent follow each other in (degree, id) order, and all
//                   connected components advance together; components are then laid out by the rank of
//                   their start node (the unvisited node of least (degree, id)) and each is reversed.
//                   The traversal is one cooperative launch; a level costs about 9 us, which for meshes
//                   and other graphs with tens to hundreds of levels is much of the time (64 000-node shuffled
//                   27-point mesh, 41 levels: 0.38 of 0.93 ms with packing and plan; a launch
//                   sequence with three radix sorts and a host read per level took 13 ms).
// Applying an order -- gathering the rows of a device CSR matrix -- and undoing it are device work
// too: the SpMM kernels take the order as a row map and write output row order[new_row] directly,
// which replaces the bridge's host-side unpack_output (:1083-1100).
//
// Input contract (the packers'): column ids of a row strictly ascending.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>

#include <cooperative_groups.h>

#include "common.cuh"
#include "condense.cuh"
#include "mem.h"

namespace mask {

namespace {

__global__ void iota_kernel(int32_t* a, int32_t n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}

__device__ __forceinline__ uint64_t mix_column(uint64_t v) {   // the bridge's column hash (splitmix64 finaliser)
    v += 0x9e3779b97f4a7c15ULL;
    v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ULL;
    v = (v ^ (v >> 27)) * 0x94d049bb133111ebULL;
    return v ^ (v >> 31);
}

// one warp per row: first in-range column (K if none) and the min-hash signature over all its columns
__global__ void row_keys_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind, int32_t M, int32_t K,
                                uint32_t* __restrict__ first, uint64_t* __restrict__ sig) {
    const int64_t row = grid_warp();
    if (row >= M) return;
    const int r = (int)row, lane = threadIdx.x & 31;
    uint32_t f = (uint32_t)K;
    uint64_t s = ~0ULL;
    for (int q = rowptr[r] + lane; q < rowptr[r + 1]; q += 32) {
        const int c = colind[q];
        if (c >= 0 && c < K) f = min(f, (uint32_t)c);
        s = min(s, mix_column((uint64_t)(uint32_t)c));
    }
    for (int o = 16; o > 0; o >>= 1) {
        f = min(f, __shfl_xor_sync(0xffffffffu, f, o));
        s = min(s, __shfl_xor_sync(0xffffffffu, s, o));
    }
    if (lane == 0) {
        first[r] = f;
        if (sig) sig[r] = s;
    }
}

template <typename KeyT>
__global__ void gather_keys_kernel(const KeyT* __restrict__ key_of_row, const int32_t* __restrict__ rows, int32_t n, KeyT* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = key_of_row[rows[i]];
}

// Stable sort of `rows` (n row ids) by key_of_row[row]: keys gathered, CUB radix sort by key.
template <typename KeyT>
int sort_rows_by(const KeyT* key_of_row, int32_t* rows_in, int32_t* rows_out, int32_t n, int end_bit, cudaStream_t st) {
    if (n == 0) return MASK_OK;
    DevScratch keys, tmp;
    const size_t half = ((size_t)n * sizeof(KeyT) + 255) & ~(size_t)255;
    int rc = keys.alloc(2 * half, st);
    if (rc != MASK_OK) return rc;
    KeyT *kin = keys.as<KeyT>(), *kout = keys.as<KeyT>(half);
    gather_keys_kernel<KeyT><<<blocks_for(n, 256), 256, 0, st>>>(key_of_row, rows_in, n, kin);
    MASK_CUDA_TRY(cudaGetLastError());
    size_t bytes = 0;
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, bytes, kin, kout, rows_in, rows_out, n, 0, end_bit, st));
    rc = tmp.alloc(bytes, st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, bytes, kin, kout, rows_in, rows_out, n, 0, end_bit, st));
    return MASK_OK;
}

// |cols(a) & cols(b)| by one warp: lanes walk the shorter row and search the longer one
__device__ int warp_intersection(const int32_t* __restrict__ ci, int a0, int a1, int b0, int b1, int lane) {
    if (a1 - a0 > b1 - b0) { int t = a0; a0 = b0; b0 = t; t = a1; a1 = b1; b1 = t; }
    int hits = 0;
    for (int q = a0 + lane; q < a1; q += 32) {
        const int c = ci[q];
        int lo = b0, hi = b1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ci[mid] < c) lo = mid + 1; else hi = mid;
        }
        hits += (lo < b1 && ci[lo] == c);
    }
    for (int o = 16; o > 0; o >>= 1) hits += __shfl_xor_sync(0xffffffffu, hits, o);
    return hits;
}

// One block per bucket of 64 ranked rows: greedy chain by exact Jaccard similarity to the row placed
// last; among equally similar rows the smaller id wins.
__global__ void __launch_bounds__(256) jaccard_chain_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind,
                                                            const int32_t* __restrict__ ranked, int32_t M, int32_t* __restrict__ order) {
    __shared__ int rows[64];
    __shared__ double score[64];
    __shared__ int alive[64];
    __shared__ int cur;
    const int base = blockIdx.x * 64;
    const int n = min(64, M - base);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < 64) {
        rows[tid] = tid < n ? ranked[base + tid] : -1;
        alive[tid] = tid < n && tid > 0;
    }
    if (tid == 0) { cur = ranked[base]; order[base] = ranked[base]; }
    __syncthreads();
    for (int placed = 1; placed < n; placed++) {
        const int c0 = rowptr[cur], c1 = rowptr[cur + 1];
        for (int c = warp; c < n; c += 8) {
            if (!alive[c]) continue;
            const int r = rows[c];
            const int r0 = rowptr[r], r1 = rowptr[r + 1];
            const int inter = warp_intersection(colind, c0, c1, r0, r1, lane);
            const int uni = (c1 - c0) + (r1 - r0) - inter;
            if (lane == 0) score[c] = uni ? (double)inter / (double)uni : 1.0;
        }
        __syncthreads();
        if (warp == 0) {   // argmax of (score, -row id) over the remaining candidates
            double bs = -1.0;
            int bi = -1, br = 0x7fffffff;
            for (int c = lane; c < n; c += 32) {
                if (!alive[c]) continue;
                const double sc = score[c];
                if (sc > bs || (sc == bs && rows[c] < br)) { bs = sc; bi = c; br = rows[c]; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double os = __shfl_xor_sync(0xffffffffu, bs, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o), orow = __shfl_xor_sync(0xffffffffu, br, o);
                if (oi >= 0 && (bi < 0 || os > bs || (os == bs && orow < br))) { bs = os; bi = oi; br = orow; }
            }
            if (lane == 0) {
                alive[bi] = 0;
                cur = br;
                order[base + placed] = br;
            }
        }
        __syncthreads();
    }
}

// ---- reverse Cuthill-McKee ------------------------------------------------------------------------
// Nodes are renamed by their rank in (degree, id) order, and every node's neighbours are listed in ascending
// rank: the children a node contributes to the queue are then its new neighbours as they stand in its list,
// and no level has to be sorted.

__global__ void sym_edge_keys_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind, int32_t M,
                                     uint64_t* __restrict__ keys) {
    // one warp per row; every stored (r, c) with c != r in range gives (r, c) and (c, r); others give a sentinel
    const int64_t row = grid_warp();
    if (row >= M) return;
    const int r = (int)row, lane = threadIdx.x & 31;
    for (int q = rowptr[r] + lane; q < rowptr[r + 1]; q += 32) {
        const int c = colind[q];
        const bool ok = c >= 0 && c < M && c != r;
        keys[2 * (int64_t)q] = ok ? ((uint64_t)(uint32_t)r << 32 | (uint32_t)c) : ~0ULL;
        keys[2 * (int64_t)q + 1] = ok ? ((uint64_t)(uint32_t)c << 32 | (uint32_t)r) : ~0ULL;
    }
}
__global__ void count_sources_kernel(const uint64_t* __restrict__ keys, int64_t n, int32_t* __restrict__ deg) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && keys[i] != ~0ULL) atomicAdd(&deg[(int32_t)(keys[i] >> 32)], 1);
}
__global__ void split_targets_kernel(const uint64_t* __restrict__ keys, int64_t n, int32_t* __restrict__ adj) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) adj[i] = (int32_t)(keys[i] & 0xffffffffu);
}
// one thread per entry of a CSR matrix: its row, searched between the rows of the block's first and last entry
__device__ __forceinline__ int row_of_entry(const int32_t* __restrict__ ptr, int32_t M, int64_t first, int64_t last, int64_t e, int* range) {
    if (threadIdx.x < 2) {
        const int64_t key = threadIdx.x == 0 ? first : last;
        int lo = 0, hi = M;   // last row with ptr[row] <= key
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((int64_t)ptr[mid] <= key) lo = mid; else hi = mid;
        }
        range[threadIdx.x] = lo;
    }
    __syncthreads();
    int lo = range[0], hi = range[1] + 1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)ptr[mid] <= e) lo = mid; else hi = mid;
    }
    __syncthreads();
    return lo;
}

__global__ void row_lengths_kernel(const int32_t* __restrict__ ptr, int32_t M, int32_t* __restrict__ len) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) len[i] = ptr[i + 1] - ptr[i];
}

// Takes diagonal and out-of-range entries off the degrees; *asymmetric is set if some other entry (r, c) has no
// counterpart (c, r), or if a row is not strictly ascending: an entry listed twice would be queued twice.
__global__ void __launch_bounds__(256) check_symmetry_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ col, int32_t M,
                                                             int64_t nnz, int32_t* __restrict__ deg, int32_t* __restrict__ asymmetric) {
    __shared__ int range[2];
    const int64_t first = (int64_t)blockIdx.x * 256, e = first + threadIdx.x;
    const int64_t last = first + 255 < nnz ? first + 255 : nnz - 1;
    const int r = row_of_entry(ptr, M, first, last, e < nnz ? e : last, range);
    if (e >= nnz) return;
    const int c = col[e];
    if (e > ptr[r] && __ldg(col + e - 1) >= c) *asymmetric = 1;
    if (c < 0 || c >= M || c == r) {
        atomicSub(&deg[r], 1);
        return;
    }
    int lo = ptr[c], hi = ptr[c + 1];
    const int end = hi;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(col + mid) < r) lo = mid + 1; else hi = mid;
    }
    if (lo == end || col[lo] != r) *asymmetric = 1;
}

__global__ void scatter_rank_kernel(const int32_t* __restrict__ starts, int32_t M, int32_t* __restrict__ rank, int32_t* __restrict__ label) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) {
        rank[starts[i]] = i;
        label[i] = i;
    }
}

constexpr int kAdjSortMax = 1024;   // longest neighbour list a warp sorts

// neighbours of node starts[i] by rank; lists of more than 32 E entries are not for this E
template <int E>
__device__ __forceinline__ void sort_neighbours(const int32_t* __restrict__ col, int n, int self, int32_t M, const int32_t* __restrict__ rank,
                                                int32_t* __restrict__ out, int n_out, int lane) {
    uint32_t key[E];
#pragma unroll
    for (int i = 0; i < E; i++) {
        const int e = i * 32 + lane;
        const int c = e < n ? __ldg(col + e) : -1;
        key[i] = (c >= 0 && c < M && c != self) ? (uint32_t)rank[c] : ~0u;
    }
    warp_sort<E, uint32_t>(key, lane);
#pragma unroll
    for (int i = 0; i < E; i++)
        if (lane * E + i < n_out) out[lane * E + i] = (int32_t)key[i];
}

__global__ void __launch_bounds__(128) sort_adjacency_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ col, int32_t M,
                                                             const int32_t* __restrict__ starts, const int32_t* __restrict__ rank,
                                                             const int32_t* __restrict__ out_ptr, int32_t* __restrict__ out,
                                                             int32_t* __restrict__ long_list, int32_t* __restrict__ n_long) {
    const int64_t node = grid_warp();
    if (node >= M) return;
    const int i = (int)node, lane = threadIdx.x & 31;
    const int v = starts[i], b = ptr[v], n = ptr[v + 1] - b, o = out_ptr[i], n_out = out_ptr[i + 1] - o;
    if (n > kAdjSortMax) {
        if (lane == 0) long_list[atomicAdd(n_long, 1)] = i;
    } else if (n > 512) {
        sort_neighbours<32>(col + b, n, v, M, rank, out + o, n_out, lane);
    } else if (n > 128) {
        sort_neighbours<16>(col + b, n, v, M, rank, out + o, n_out, lane);
    } else if (n > 32) {
        sort_neighbours<4>(col + b, n, v, M, rank, out + o, n_out, lane);
    } else if (n > 0) {
        sort_neighbours<1>(col + b, n, v, M, rank, out + o, n_out, lane);
    }
}

constexpr int kLongBits = 1 << 19;
// the same for long lists: one block marks the ranks, kLongBits at a time from the smallest one left, and places
// every one by the number of marks below it
__global__ void __launch_bounds__(512) sort_long_adjacency_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ col, int32_t M,
                                                                  const int32_t* __restrict__ starts, const int32_t* __restrict__ rank,
                                                                  const int32_t* __restrict__ out_ptr, int32_t* __restrict__ out,
                                                                  const int32_t* __restrict__ long_list, const int32_t* __restrict__ n_long) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int run_before[kLongBits / 4096];
    __shared__ int warp_sum[32];
    const int total = *n_long;
    MarkSet marks{reinterpret_cast<uint32_t*>(smem), reinterpret_cast<uint16_t*>(smem + kLongBits / 8), run_before,
                  (min(M, kLongBits) + 4095) / 4096};
    for (int j = blockIdx.x; j < total; j += gridDim.x) {
        const int i = long_list[j], v = starts[i], b = ptr[v], n = ptr[v + 1] - b, o = out_ptr[i];
        int placed = 0;
        for (int r0 = 0; r0 < M;) {
            const int span = min(kLongBits, M - r0);
            int behind = INT_MAX;   // smallest rank behind this range
            __syncthreads();
            for (int k = threadIdx.x; k < marks.n_runs * 128; k += 512) marks.bits[k] = 0;
            __syncthreads();
            auto each = [&](auto f) {
#pragma unroll 4
                for (int e = threadIdx.x; e < n; e += 512) {
                    const int c = __ldg(col + b + e);
                    if (c < 0 || c >= M || c == v) continue;
                    const int d = rank[c] - r0;
                    if (d >= span) behind = min(behind, r0 + d);
                    else if (d >= 0) f(d);
                }
            };
            each([&](int d) { marks.mark(d); });
            const int here = marks.count<512>(warp_sum);
            each([&](int d) { out[o + placed + marks.rank(d)] = r0 + d; });
            placed += here;
            r0 = M <= kLongBits ? M : block_least<512>(behind, warp_sum);
        }
    }
}

// Connected components as a forest: label[i] is a node of i's tree that is smaller than i, or i if i is the root, so that
// labels end as the component's least rank.  Many threads join trees at once (Anderson and Woll, "Wait-free parallel
// algorithms for the union-find problem", 1991): a root is given a parent by compare-and-swap, everything else only ever
// moves up.

// The root of i's tree.  Every node on the way is moved up to its grandparent (path splitting: Tarjan and van Leeuwen,
// "Worst-case analysis of set union algorithms", 1984).
__device__ __forceinline__ int find_root(int32_t* label, int i) {
    for (int parent = __ldcg(label + i); parent != i;) {
        const int grandparent = __ldcg(label + parent);
        if (grandparent != parent) __stcg(label + i, grandparent);
        i = parent;
        parent = grandparent;
    }
    return i;
}
// Joins the trees of i and j: the larger root goes below the smaller one.
__device__ __forceinline__ void unite(int32_t* label, int i, int j) {
    for (;;) {
        i = find_root(label, i);
        j = find_root(label, j);
        if (i == j) return;
        const int below = max(i, j);
        if (atomicCAS(label + below, below, min(i, j)) == below) return;
    }   // `below` has got a parent meanwhile: on from there
}
constexpr int64_t kFewEdges = 1 << 17;   // up to here along every edge at once: a dozen launches cost more than the contention
__global__ void __launch_bounds__(256) hook_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ adj, int32_t M, int32_t* label) {
    __shared__ int range[2];
    const int64_t n = ptr[M];
    const int64_t first = (int64_t)blockIdx.x * 256, e = first + threadIdx.x;
    if (first >= n) return;
    const int64_t last = first + 255 < n ? first + 255 : n - 1;
    const int i = row_of_entry(ptr, M, first, last, e < n ? e : last, range);
    if (e >= n) return;
    const int j = adj[e];
    if (j < i) unite(label, i, j);   // every edge is listed from both ends
}
// With more edges: first every node points to its least neighbour if that is smaller (the start of ECL-CC: Jaiganesh and
// Burtscher, "A high-performance connected components implementation for GPUs", 2018); no two nodes write the same
// label.  Then four rounds, each along one more edge of every node and with flat trees, so that nobody follows a chain
// while it grows: a root joins the least root that its nodes see.  That leaves one component with nearly all nodes where
// the graph has one; a sample of the nodes tells which, and its nodes need not look at their other edges, because an edge
// out of it is found from its other end (Afforest: Sutton, Ben-Nun and Barak, "Optimizing parallel graph connectivity
// computation via subgraph sampling", 2018).  Uniting along every edge had all of them contend for a few roots: 64 000-node
// stencil 100 to 230 us, power-law graph of 200 000 nodes 430, now 59 and 73 in all.
__global__ void least_neighbour_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ adj, int32_t M, int32_t* __restrict__ label) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) label[i] = ptr[i] < ptr[i + 1] ? min(i, adj[ptr[i]]) : i;
}
// along the neighbour at `quarter` quarters of the list; labels are roots
__global__ void hook_roots_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ adj, int32_t M, int quarter, int32_t* label) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M || ptr[i] == ptr[i + 1]) return;
    const int a = __ldcg(label + i), b = __ldcg(label + adj[ptr[i] + (int)((int64_t)(ptr[i + 1] - ptr[i] - 1) * quarter / 4)]);
    const int hi = max(a, b), lo = min(a, b);
    if (__ldcg(label + hi) > lo) atomicMin(label + hi, lo);
}
// *most: the label that most of 256 nodes have
__global__ void __launch_bounds__(256) common_label_kernel(const int32_t* __restrict__ label, int32_t M, int32_t* __restrict__ most) {
    __shared__ int32_t seen[256];
    __shared__ int best;
    const int mine = label[(int)((int64_t)threadIdx.x * M / 256)];
    seen[threadIdx.x] = mine;
    if (threadIdx.x == 0) best = 0;
    __syncthreads();
    int n = 0;
    for (int k = 0; k < 256; k++) n += seen[k] == mine;
    atomicMax(&best, n << 8 | threadIdx.x);
    __syncthreads();
    if (threadIdx.x == (best & 255)) *most = mine;
}
// The remaining edges: a warp per node, lists longer than kAdjSortMax in the next kernel.
__global__ void __launch_bounds__(256) hook_rest_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ adj, int32_t M,
                                                        int32_t* label, const int32_t* __restrict__ most) {
    const int64_t node = grid_warp();
    if (node >= M) return;
    const int i = (int)node;
    if (__ldcg(label + i) == *most) return;
    const int b = ptr[i], e = ptr[i + 1];
    if (e - b > kAdjSortMax) return;
    for (int q = b + (threadIdx.x & 31); q < e; q += 32) unite(label, i, adj[q]);
}
__global__ void __launch_bounds__(512) hook_long_kernel(const int32_t* __restrict__ ptr, const int32_t* __restrict__ adj, int32_t* label,
                                                        const int32_t* __restrict__ most, const int32_t* __restrict__ long_list,
                                                        const int32_t* __restrict__ n_long) {
    for (int k = blockIdx.x; k < *n_long; k += gridDim.x) {
        const int i = long_list[k];
        if (__ldcg(label + i) == *most) continue;
        for (int q = ptr[i] + (int)threadIdx.x; q < ptr[i + 1]; q += 512) unite(label, i, adj[q]);
    }
}
__global__ void flatten_labels_kernel(int32_t* __restrict__ label, int32_t M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    int root = i;
    for (int parent = __ldcg(label + root); parent != root; parent = __ldcg(label + root)) root = parent;
    __stcg(label + i, root);
}
struct IsRoot {
    const int32_t* label;
    __device__ bool operator()(int i) const { return label[i] == i; }
};

// Breadth-first levels of all components at once, in Cuthill-McKee queue order, as one cooperative launch.
// Per level: (1) every unvisited neighbour records the earliest queue position that reaches it, (2) every queue
// node counts the neighbours that recorded it, (3) the counts are scanned and the children written behind the
// queue.  A block takes a run of consecutive queue nodes, a warp a node (nodes with long lists: the block).
// Levels of at most kSmallLevel nodes are walked by one block alone, without grid-wide barriers.  Positions are
// unsigned: a stride past the last of 2^31 - 1 nodes stays a number.
struct BfsArgs {
    const int32_t* ptr;
    const int32_t* adj;
    int32_t* queue;
    int32_t* pos;        // queue position, -1 before
    uint32_t* parent;    // earliest queue position that reaches the node, ~0u before
    int32_t* children;   // per node of the level
    int32_t* block_sum;  // per block
    int32_t* state;      // [0] base of the level, [1] its size
    const int32_t* n_start;
    const int32_t* n_sorted_long;   // lists longer than kAdjSortMax
    int32_t M;
};
constexpr int kBfsThreads = 512, kBfsWarps = kBfsThreads / 32;
constexpr int kBlockList = 1024;   // lists longer than this are walked by the whole block
constexpr int kSmallLevel = 64;

static_assert(kBlockList >= kAdjSortMax, "no list that long if none is longer than kAdjSortMax");
constexpr int kKept = 2;   // nodes of a level that a warp keeps the lists of (if at most 32 long)

constexpr int kMaxLong = 256;

// A warp's first nodes of the level, from one phase to the next: what it knows need not be loaded through the chain
// queue -> ptr -> adjacency -> parent again (64 000-node stencil, 41 levels: 442 us, now 376).
struct BfsKept {
    int nb[kKept];         // this lane's neighbour, -1: none
    bool kept[kKept];
    unsigned child[kKept];
};

struct BfsShared {
    int warp_sum[kBfsWarps];
    int n_long;            // nodes of the block's share with long lists; too many of them: every node to a warp
    uint32_t long_at[kMaxLong];
    __device__ __forceinline__ bool by_block(int len) const { return len > kBlockList && n_long <= kMaxLong; }
};

// `width` lanes (a warp or the block) record queue position qpos with the unvisited neighbours of its node.
__device__ __forceinline__ void bfs_mark(const BfsArgs& p, uint32_t qpos, int lane, int width) {
    const int v = __ldcg(p.queue + qpos), b = p.ptr[v], e = p.ptr[v + 1];
    for (int q = b + lane; q < e; q += width) {
        const int nb = p.adj[q];
        if (__ldcg(p.pos + nb) < 0 && __ldcg(p.parent + nb) > qpos) atomicMin(p.parent + nb, qpos);
    }
}
__device__ __forceinline__ int warp_total(int x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
__device__ __forceinline__ int block_exclusive(int x, BfsShared& s, int* total) {   // all threads
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int y = x;
    for (int o = 1; o < 32; o <<= 1) {
        const int z = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += z;
    }
    __syncthreads();
    if (lane == 31) s.warp_sum[warp] = y;
    __syncthreads();
    int before = 0, all = 0;
    for (int i = 0; i < kBfsWarps; i++) {
        const int v = s.warp_sum[i];
        all += v;
        if (i < warp) before += v;
    }
    *total = all;
    return before + y - x;
}

// The queue nodes [lo, hi) of the level that begins at `base`: marks.
__device__ __forceinline__ void bfs_mark_range(const BfsArgs& p, uint32_t base, uint32_t lo, uint32_t hi, BfsShared& s, BfsKept& keep) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s.n_long = 0;
    if (*p.n_sorted_long > 0) {
        __syncthreads();
        for (uint32_t i = lo + threadIdx.x; i < hi; i += kBfsThreads) {
            const int v = __ldcg(p.queue + base + i);
            if (p.ptr[v + 1] - p.ptr[v] > kBlockList) {
                const int k = atomicAdd(&s.n_long, 1);
                if (k < kMaxLong) s.long_at[k] = i;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kKept; t++) {
        const uint32_t i = lo + warp + t * kBfsWarps;
        keep.kept[t] = false;
        if (i >= hi) continue;
        const int v = __ldcg(p.queue + base + i), b = p.ptr[v], e = p.ptr[v + 1];
        if (e - b > 32) {
            if (!s.by_block(e - b)) bfs_mark(p, base + i, lane, 32);
            continue;
        }
        keep.kept[t] = true;
        const int nb = b + lane < e ? p.adj[b + lane] : -1;
        keep.nb[t] = nb;
        if (nb >= 0 && __ldcg(p.pos + nb) < 0 && __ldcg(p.parent + nb) > base + i) atomicMin(p.parent + nb, base + i);
    }
    for (uint32_t i = lo + warp + kKept * kBfsWarps; i < hi; i += kBfsWarps) {
        const int v = __ldcg(p.queue + base + i);
        if (!s.by_block(p.ptr[v + 1] - p.ptr[v])) bfs_mark(p, base + i, lane, 32);
    }
    if (s.n_long <= kMaxLong)
        for (int k = 0; k < s.n_long; k++) bfs_mark(p, base + s.long_at[k], threadIdx.x, kBfsThreads);
}
__device__ __forceinline__ bool is_kept(const BfsKept& keep, int t) {
    bool x = false;
#pragma unroll
    for (int k = 0; k < kKept; k++) x |= t == k && keep.kept[k];
    return x;
}
// Counts children per node; returns the sum over the range (to every thread).
__device__ __forceinline__ int bfs_count_range(const BfsArgs& p, uint32_t base, uint32_t lo, uint32_t hi, BfsShared& s, BfsKept& keep) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int sum = 0;
#pragma unroll
    for (int t = 0; t < kKept; t++) {
        if (!keep.kept[t]) continue;
        const uint32_t i = lo + warp + t * kBfsWarps;
        keep.child[t] = __ballot_sync(0xffffffffu, keep.nb[t] >= 0 && __ldcg(p.parent + max(keep.nb[t], 0)) == base + i);
        const int c = __popc(keep.child[t]);
        if (lane == 0) { p.children[i] = c; sum += c; }
    }
    uint32_t i = lo + warp;
    for (int t = 0; i < hi; i += kBfsWarps, t++) {
        if (is_kept(keep, t)) continue;
        const int v = __ldcg(p.queue + base + i), b = p.ptr[v], e = p.ptr[v + 1];
        if (s.by_block(e - b)) continue;
        int c = 0;
        for (int q = b + lane; q < e; q += 32) c += __ldcg(p.parent + p.adj[q]) == base + i;
        c = warp_total(c);
        if (lane == 0) { p.children[i] = c; sum += c; }
    }
    for (int k = 0; k < s.n_long && s.n_long <= kMaxLong; k++) {
        const uint32_t i = s.long_at[k];
        const int v = __ldcg(p.queue + base + i), b = p.ptr[v], e = p.ptr[v + 1];
        int c = 0, all = 0;
        for (int q = b + threadIdx.x; q < e; q += kBfsThreads) c += __ldcg(p.parent + p.adj[q]) == base + i;
        block_exclusive(c, s, &all);
        if (threadIdx.x == 0) { p.children[i] = all; sum += all; }
    }
    int total = 0;
    block_exclusive(sum, s, &total);
    return total;
}
// Writes the children of the range behind queue position `at` and numbers them.
__device__ __forceinline__ void bfs_place_range(const BfsArgs& p, uint32_t base, uint32_t lo, uint32_t hi, int at, BfsShared& s, const BfsKept& keep) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();   // children[] of the range has been written by this block
    for (uint32_t c0 = lo; c0 < hi; c0 += kBfsThreads) {
        const int mine = c0 + threadIdx.x < hi ? __ldcg(p.children + c0 + threadIdx.x) : 0;
        int all = 0;
        const int before = block_exclusive(mine, s, &all);
        if (c0 + threadIdx.x < hi) p.children[c0 + threadIdx.x] = at + before;   // now: where they go
        at += all;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kKept; t++) {
        if (!keep.kept[t]) continue;
        if (keep.child[t] >> lane & 1) {
            const int o = __ldcg(p.children + lo + warp + t * kBfsWarps) + __popc(keep.child[t] & ((1u << lane) - 1u));
            p.queue[o] = keep.nb[t];
            p.pos[keep.nb[t]] = o;
        }
    }
    uint32_t i = lo + warp;
    for (int t = 0; i < hi; i += kBfsWarps, t++) {
        if (is_kept(keep, t)) continue;
        const int v = __ldcg(p.queue + base + i), b = p.ptr[v], e = p.ptr[v + 1];
        if (s.by_block(e - b)) continue;
        int to = __ldcg(p.children + i);
        for (int q0 = b; q0 < e; q0 += 32) {
            const int nb = q0 + lane < e ? p.adj[q0 + lane] : -1;
            const bool child = nb >= 0 && __ldcg(p.parent + nb) == base + i;
            const unsigned m = __ballot_sync(0xffffffffu, child);
            if (child) {
                const int o = to + __popc(m & ((1u << lane) - 1u));
                p.queue[o] = nb;
                p.pos[nb] = o;
            }
            to += __popc(m);
        }
    }
    for (int k = 0; k < s.n_long && s.n_long <= kMaxLong; k++) {
        const uint32_t i = s.long_at[k];
        const int v = __ldcg(p.queue + base + i), b = p.ptr[v], e = p.ptr[v + 1];
        int to = __ldcg(p.children + i);
        for (int q0 = b; q0 < e; q0 += kBfsThreads) {
            const int nb = q0 + (int)threadIdx.x < e ? p.adj[q0 + threadIdx.x] : -1;
            const bool child = nb >= 0 && __ldcg(p.parent + nb) == base + i;
            int all = 0;
            const int before = block_exclusive(child, s, &all);
            if (child) {
                p.queue[to + before] = nb;
                p.pos[nb] = to + before;
            }
            to += all;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kBfsThreads) bfs_kernel(const BfsArgs p) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ BfsShared s;
    BfsKept keep;
    int base = 0, n = *p.n_start;
    for (uint32_t i = blockIdx.x * kBfsThreads + threadIdx.x; i < (uint32_t)n; i += gridDim.x * kBfsThreads) p.pos[__ldcg(p.queue + i)] = i;
    grid.sync();
    while (n > 0) {
        if (n <= kSmallLevel) {
            if (blockIdx.x == 0) {
                while (n > 0 && n <= kSmallLevel) {
                    bfs_mark_range(p, base, 0, n, s, keep);
                    __syncthreads();
                    const int next = bfs_count_range(p, base, 0, n, s, keep);
                    bfs_place_range(p, base, 0, n, base + n, s, keep);
                    base += n;
                    n = next;
                }
                if (threadIdx.x == 0) { p.state[0] = base; p.state[1] = n; }
            }
            grid.sync();
            base = __ldcg(p.state);
            n = __ldcg(p.state + 1);
            grid.sync();   // everybody has read the state
            continue;
        }
        const int share = (n + gridDim.x - 1) / gridDim.x;
        const int lo = min(n, (int)blockIdx.x * share), hi = lo + min(share, n - lo);
        bfs_mark_range(p, base, lo, hi, s, keep);
        grid.sync();
        const int sum = bfs_count_range(p, base, lo, hi, s, keep);
        if (threadIdx.x == 0) p.block_sum[blockIdx.x] = sum;
        grid.sync();
        int x = 0, all = 0, before = 0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += kBfsThreads) {
            const int v = __ldcg(p.block_sum + i);
            all += v;
            if (i < (int)blockIdx.x) x += v;
        }
        block_exclusive(x, s, &before);
        int next = 0;
        block_exclusive(all, s, &next);
        bfs_place_range(p, base, lo, hi, base + n + before, s, keep);
        base += n;
        n = next;
        grid.sync();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) p.state[0] = base;
}

// item i of the final order before it is sorted by component: the queue from its end
__global__ void reversed_queue_kernel(const int32_t* __restrict__ queue, const int32_t* __restrict__ label, const int32_t* __restrict__ starts,
                                      int32_t M, uint32_t* __restrict__ key, int32_t* __restrict__ row) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const int v = queue[M - 1 - i];
    key[i] = (uint32_t)label[v];
    row[i] = starts[v];
}

inline int bits_for(int64_t n) {   // bits of the numbers below n
    int b = 1;
    while (((int64_t)1 << b) < n) b++;
    return b;
}

// Both directions of every off-diagonal entry, deduplicated, as a CSR matrix: for patterns that are not symmetric.
int symmetrised_pattern(const int32_t* rowptr, const int32_t* colind, int32_t M, int64_t nnz, DevScratch& ptr_b, DevScratch& adj_b,
                        int64_t* n_edges_out, cudaStream_t st) {
    DevScratch keys, keys_sorted, tmp, n_unique_d, deg_b;
    const int64_t n_keys = 2 * nnz;
    if (n_keys >= ((int64_t)1 << 31)) return fail(MASK_ERR_INDEX_OVERFLOW, "too many entries for the device reorder");
    int rc = keys.alloc((size_t)n_keys * 8, st);
    if (rc == MASK_OK) rc = keys_sorted.alloc((size_t)n_keys * 8, st);
    if (rc == MASK_OK) rc = n_unique_d.alloc(8, st);
    if (rc == MASK_OK) rc = deg_b.alloc(((size_t)M + 1) * 4, st);
    if (rc == MASK_OK) rc = ptr_b.alloc(((size_t)M + 1) * 4, st);
    if (rc != MASK_OK) return rc;
    const unsigned row_blocks = blocks_for((int64_t)M * 32, 256);
    sym_edge_keys_kernel<<<row_blocks, 256, 0, st>>>(rowptr, colind, M, keys.as<uint64_t>());
    MASK_CUDA_TRY(cudaGetLastError());
    uint64_t *k0 = keys.as<uint64_t>(), *k1 = keys_sorted.as<uint64_t>();
    size_t b1 = 0, b2 = 0, b3 = 0;
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, b1, k0, k1, (int)n_keys, 0, 64, st));
    MASK_CUDA_TRY(cub::DeviceSelect::Unique(nullptr, b2, k1, k0, n_unique_d.as<int64_t>(), (int)n_keys, st));
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(nullptr, b3, deg_b.as<int32_t>(), ptr_b.as<int32_t>() + 1, M, st));
    rc = tmp.alloc(std::max(b1, std::max(b2, b3)), st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp.p, b1, k0, k1, (int)n_keys, 0, 64, st));
    MASK_CUDA_TRY(cub::DeviceSelect::Unique(tmp.p, b2, k1, k0, n_unique_d.as<int64_t>(), (int)n_keys, st));
    HostStage host;
    rc = host.get(8);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cudaMemcpyAsync(host.as<int64_t>(), n_unique_d.p, 8, cudaMemcpyDeviceToHost, st));
    MASK_CUDA_TRY(cudaStreamSynchronize(st));
    int64_t n_edges = *host.as<int64_t>();
    if (n_edges > 0) {   // the sentinel (all ones) sorts last and, if present, is one unique key: drop it
        MASK_CUDA_TRY(cudaMemcpyAsync(host.as<int64_t>(), k0 + (n_edges - 1), 8, cudaMemcpyDeviceToHost, st));
        MASK_CUDA_TRY(cudaStreamSynchronize(st));
        if (*host.as<uint64_t>() == ~0ULL) n_edges--;
    }
    rc = adj_b.alloc((size_t)std::max<int64_t>(n_edges, 1) * 4, st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cudaMemsetAsync(deg_b.p, 0, ((size_t)M + 1) * 4, st));
    if (n_edges > 0) {
        const unsigned eb = blocks_for(n_edges, 256);
        count_sources_kernel<<<eb, 256, 0, st>>>(k0, n_edges, deg_b.as<int32_t>());
        split_targets_kernel<<<eb, 256, 0, st>>>(k0, n_edges, adj_b.as<int32_t>());
        MASK_CUDA_TRY(cudaGetLastError());
    }
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(tmp.p, b3, deg_b.as<int32_t>(), ptr_b.as<int32_t>() + 1, M, st));
    MASK_CUDA_TRY(cudaMemsetAsync(ptr_b.p, 0, 4, st));
    *n_edges_out = n_edges;
    return MASK_OK;
}

// `host`: 4 bytes; after a failure a copy into them may be in flight
int order_rcm_device(const int32_t* rowptr, const int32_t* colind, int32_t M, int64_t nnz, int32_t* order, const HostStage& host, cudaStream_t st) {
    const unsigned node_blocks = blocks_for(M, 256);
    const int32_t *ptr = rowptr, *col = colind;
    int64_t n_edges = nnz;
    DevScratch deg_b, flag_b, sym_ptr, sym_adj;
    int rc = deg_b.alloc(((size_t)M + 1) * 4, st);
    if (rc == MASK_OK) rc = flag_b.alloc(64, st);
    if (rc != MASK_OK) return rc;
    int32_t* deg = deg_b.as<int32_t>();
    int32_t* flags = flag_b.as<int32_t>();   // [0] asymmetric, [1] long lists, [2] start nodes, [4..5] state of the traversal, [6] most common label
    MASK_CUDA_TRY(cudaMemsetAsync(flags, 0, 64, st));
    row_lengths_kernel<<<node_blocks, 256, 0, st>>>(ptr, M, deg);
    if (nnz > 0) check_symmetry_kernel<<<blocks_for(nnz, 256), 256, 0, st>>>(ptr, col, M, nnz, deg, flags);
    MASK_CUDA_TRY(cudaGetLastError());
    MASK_CUDA_TRY(cudaMemcpyAsync(host.as<int32_t>(), flags, 4, cudaMemcpyDeviceToHost, st));
    MASK_CUDA_TRY(cudaStreamSynchronize(st));
    if (*host.as<int32_t>()) {
        rc = symmetrised_pattern(rowptr, colind, M, nnz, sym_ptr, sym_adj, &n_edges, st);
        if (rc != MASK_OK) return rc;
        ptr = sym_ptr.as<int32_t>();
        col = sym_adj.as<int32_t>();
        row_lengths_kernel<<<node_blocks, 256, 0, st>>>(ptr, M, deg);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    // node arrays, one allocation
    const size_t row_words = ((size_t)M + 1 + 63) & ~(size_t)63;
    enum { kIds, kStarts, kSortedDeg, kOutPtr, kRank, kLabel, kQueue, kPos, kParent, kChildren, kKey, kKeyOut, kRow, kLong, kArrays };
    DevScratch nodes, adj_b, tmp;
    rc = nodes.alloc(row_words * kArrays * 4, st);
    if (rc == MASK_OK) rc = adj_b.alloc((size_t)std::max<int64_t>(n_edges, 1) * 4, st);
    if (rc != MASK_OK) return rc;
    auto arr = [&](int which) { return nodes.as<int32_t>(row_words * which * 4); };
    uint32_t *udeg = reinterpret_cast<uint32_t*>(deg), *usorted = reinterpret_cast<uint32_t*>(arr(kSortedDeg));
    uint32_t *key = reinterpret_cast<uint32_t*>(arr(kKey)), *key_out = reinterpret_cast<uint32_t*>(arr(kKeyOut));
    const int bits = bits_for((int64_t)M + 1);
    cub::CountingInputIterator<int> counting(0);
    size_t b1 = 0, b2 = 0, b3 = 0;
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, b1, udeg, usorted, arr(kIds), arr(kStarts), M, 0, bits, st));
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(nullptr, b2, arr(kSortedDeg), arr(kOutPtr) + 1, M, st));
    MASK_CUDA_TRY(cub::DeviceSelect::If(nullptr, b3, counting, arr(kQueue), flags + 2, M, IsRoot{arr(kLabel)}, st));
    rc = tmp.alloc(std::max(b1, std::max(b2, b3)), st);
    if (rc != MASK_OK) return rc;
    // ranks in (degree, id) order, adjacency in ranks
    iota_kernel<<<node_blocks, 256, 0, st>>>(arr(kIds), M);
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, b1, udeg, usorted, arr(kIds), arr(kStarts), M, 0, bits, st));
    scatter_rank_kernel<<<node_blocks, 256, 0, st>>>(arr(kStarts), M, arr(kRank), arr(kLabel));
    MASK_CUDA_TRY(cudaMemsetAsync(arr(kOutPtr), 0, 4, st));
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(tmp.p, b2, arr(kSortedDeg), arr(kOutPtr) + 1, M, st));
    int32_t* adj = adj_b.as<int32_t>();
    sort_adjacency_kernel<<<blocks_for((int64_t)M * 32, 128), 128, 0, st>>>(ptr, col, M, arr(kStarts), arr(kRank), arr(kOutPtr), adj, arr(kLong),
                                                                            flags + 1);
    MASK_CUDA_TRY(cudaGetLastError());
    if (n_edges > kAdjSortMax) {
        constexpr int kSmem = mark_set_bytes(kLongBits);
        MASK_CUDA_TRY(cudaFuncSetAttribute(sort_long_adjacency_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        const int64_t most = std::min<int64_t>(n_edges / kAdjSortMax, 2 * sm_count());
        sort_long_adjacency_kernel<<<(unsigned)most, 512, kSmem, st>>>(ptr, col, M, arr(kStarts), arr(kRank), arr(kOutPtr), adj, arr(kLong), flags + 1);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    // components; their least ranks, ascending, begin the queue
    if (n_edges > 0) {
        if (n_edges <= kFewEdges) {
            hook_kernel<<<blocks_for(n_edges, 256), 256, 0, st>>>(arr(kOutPtr), adj, M, arr(kLabel));
        } else {
            least_neighbour_kernel<<<node_blocks, 256, 0, st>>>(arr(kOutPtr), adj, M, arr(kLabel));
            flatten_labels_kernel<<<node_blocks, 256, 0, st>>>(arr(kLabel), M);
            for (int quarter : {4, 2, 1, 3}) {
                hook_roots_kernel<<<node_blocks, 256, 0, st>>>(arr(kOutPtr), adj, M, quarter, arr(kLabel));
                flatten_labels_kernel<<<node_blocks, 256, 0, st>>>(arr(kLabel), M);
            }
            common_label_kernel<<<1, 256, 0, st>>>(arr(kLabel), M, flags + 6);
            hook_rest_kernel<<<blocks_for((int64_t)M * 32, 256), 256, 0, st>>>(arr(kOutPtr), adj, M, arr(kLabel), flags + 6);
            hook_long_kernel<<<(unsigned)std::min<int64_t>(n_edges / kAdjSortMax, 2 * sm_count()), 512, 0, st>>>(
                arr(kOutPtr), adj, arr(kLabel), flags + 6, arr(kLong), flags + 1);
        }
    }
    flatten_labels_kernel<<<node_blocks, 256, 0, st>>>(arr(kLabel), M);
    MASK_CUDA_TRY(cudaGetLastError());
    MASK_CUDA_TRY(cub::DeviceSelect::If(tmp.p, b3, counting, arr(kQueue), flags + 2, M, IsRoot{arr(kLabel)}, st));
    MASK_CUDA_TRY(cudaMemsetAsync(arr(kPos), 0xff, (size_t)M * 4, st));
    MASK_CUDA_TRY(cudaMemsetAsync(arr(kParent), 0xff, (size_t)M * 4, st));
    BfsArgs a{arr(kOutPtr), adj, arr(kQueue), arr(kPos), reinterpret_cast<uint32_t*>(arr(kParent)), arr(kChildren), arr(kRow), flags + 4,
              flags + 2, flags + 1, M};
    // block sums: one word per block, in an array that is not used yet
    const unsigned blocks = (unsigned)std::min<int64_t>(sm_count(), ((int64_t)M + kBfsWarps - 1) / kBfsWarps);
    void* args[] = {&a};
    MASK_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(bfs_kernel), dim3(blocks), dim3(kBfsThreads), args, 0, st));
    MASK_CUDA_TRY(cudaMemcpyAsync(host.as<int32_t>(), flags + 4, 4, cudaMemcpyDeviceToHost, st));
    // components by the rank of their start, each in reversed queue order
    reversed_queue_kernel<<<node_blocks, 256, 0, st>>>(arr(kQueue), arr(kLabel), arr(kStarts), M, key, arr(kRow));
    MASK_CUDA_TRY(cudaGetLastError());
    MASK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, b1, key, key_out, arr(kRow), order, M, 0, bits, st));
    MASK_CUDA_TRY(cudaStreamSynchronize(st));
    if (*host.as<int32_t>() != M) return fail(MASK_ERR_INVALID_ARGUMENT, "row_rcm: the traversal did not reach every row");
    return MASK_OK;
}

}  // namespace

// ---- device: gather the rows of a CSR matrix in a given order ------------------------------------
struct PermutedLength {
    const int32_t* rowptr;
    const int32_t* order;
    __device__ int32_t operator()(int32_t i) const { const int r = order[i]; return rowptr[r + 1] - rowptr[r]; }
};
// one warp per new row copies its entries
__global__ void gather_rows_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ colind,
                                   const float* __restrict__ values, const int32_t* __restrict__ order,
                                   const int32_t* __restrict__ rowptr_out, int32_t M, int32_t* __restrict__ colind_out,
                                   float* __restrict__ values_out) {
    const int64_t row = grid_warp();
    if (row >= M) return;
    const int i = (int)row, lane = threadIdx.x & 31;
    const int r = order[i];
    const int src = rowptr[r], n = rowptr[r + 1] - src, dst = rowptr_out[i];
    for (int j = lane; j < n; j += 32) {
        colind_out[dst + j] = colind[src + j];
        values_out[dst + j] = values[src + j];
    }
}

}  // namespace mask

extern "C" int mask_reorder_rows(int kind, const int32_t* d_rowptr, const int32_t* d_colind, int32_t M, int32_t K,
                                 int32_t* d_row_order, void* stream) {
    using namespace mask;
    MASK_REQUIRE(d_rowptr && d_row_order && M >= 1 && K >= 1, "bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned node_blocks = blocks_for(M, 256), row_blocks = blocks_for((int64_t)M * 32, 256);
    if (kind == MASK_REORDER_NONE) {
        iota_kernel<<<node_blocks, 256, 0, st>>>(d_row_order, M);
        MASK_CUDA_TRY(cudaGetLastError());
        return MASK_OK;
    }
    MASK_REQUIRE(kind == MASK_REORDER_ROW_RCM || kind == MASK_REORDER_FIRST_COL_SORT || kind == MASK_REORDER_JACCARD_GREEDY,
                 "unknown reorder kind");
    HostStage host;
    int rc = host.get(4);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cudaMemcpyAsync(host.as<int32_t>(), d_rowptr + M, 4, cudaMemcpyDeviceToHost, st));
    MASK_CUDA_TRY(cudaStreamSynchronize(st));
    const int32_t nnz32 = *host.as<int32_t>();
    MASK_REQUIRE(nnz32 == 0 || d_colind, "colind is NULL");
    if (kind == MASK_REORDER_ROW_RCM) {
        if (M != K) return fail(MASK_ERR_INVALID_ARGUMENT, "row_rcm needs a square matrix");
        rc = order_rcm_device(d_rowptr, d_colind, M, nnz32, d_row_order, host, st);
        if (rc != MASK_OK) cudaStreamSynchronize(st);   // before the host words go to someone else
        return rc;
    }
    DevScratch first, sig, ids, by_first;
    rc = first.alloc((size_t)M * 4, st);
    if (rc == MASK_OK) rc = sig.alloc((size_t)M * 8, st);
    if (rc == MASK_OK) rc = ids.alloc((size_t)M * 4, st);
    if (rc == MASK_OK) rc = by_first.alloc((size_t)M * 4, st);
    if (rc != MASK_OK) return rc;
    row_keys_kernel<<<row_blocks, 256, 0, st>>>(d_rowptr, d_colind, M, K, first.as<uint32_t>(), sig.as<uint64_t>());
    iota_kernel<<<node_blocks, 256, 0, st>>>(ids.as<int32_t>(), M);
    MASK_CUDA_TRY(cudaGetLastError());
    const int col_bits = bits_for((int64_t)K + 1);   // K stands for "no column"
    if (kind == MASK_REORDER_FIRST_COL_SORT) return sort_rows_by<uint32_t>(first.as<uint32_t>(), ids.as<int32_t>(), d_row_order, M, col_bits, st);
    // (signature, first column, id): stable by first column, then stable by signature
    rc = sort_rows_by<uint32_t>(first.as<uint32_t>(), ids.as<int32_t>(), by_first.as<int32_t>(), M, col_bits, st);
    if (rc == MASK_OK) rc = sort_rows_by<uint64_t>(sig.as<uint64_t>(), by_first.as<int32_t>(), ids.as<int32_t>(), M, 64, st);
    if (rc != MASK_OK) return rc;
    jaccard_chain_kernel<<<blocks_for(M, 64), 256, 0, st>>>(d_rowptr, d_colind, ids.as<int32_t>(), M, d_row_order);
    MASK_CUDA_TRY(cudaGetLastError());
    return MASK_OK;
}

extern "C" int mask_csr_permute_rows(const int32_t* d_rowptr, const int32_t* d_colind, const float* d_values, int32_t M,
                                     const int32_t* d_row_order, int32_t* d_rowptr_out, int32_t* d_colind_out,
                                     float* d_values_out, void* stream) {
    using namespace mask;
    MASK_REQUIRE(d_rowptr && d_row_order && d_rowptr_out && M >= 1, "bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cub::TransformInputIterator<int32_t, PermutedLength, cub::CountingInputIterator<int32_t>> lengths(
        cub::CountingInputIterator<int32_t>(0), PermutedLength{d_rowptr, d_row_order});
    size_t bytes = 0;
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(nullptr, bytes, lengths, d_rowptr_out + 1, M, st));
    DevScratch tmp;
    int rc = tmp.alloc(bytes, st);
    if (rc != MASK_OK) return rc;
    MASK_CUDA_TRY(cub::DeviceScan::InclusiveSum(tmp.p, bytes, lengths, d_rowptr_out + 1, M, st));
    MASK_CUDA_TRY(cudaMemsetAsync(d_rowptr_out, 0, 4, st));
    if (d_colind && d_values && d_colind_out && d_values_out) {
        gather_rows_kernel<<<blocks_for((int64_t)M * 32, 256), 256, 0, st>>>(d_rowptr, d_colind, d_values, d_row_order, d_rowptr_out, M, d_colind_out,
                                                                             d_values_out);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    return MASK_OK;
}
