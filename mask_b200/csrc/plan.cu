// Task planners and the execution-plan handle: the reference's mappings on the host, the default one on the device.
#include "plan.h"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>

#include "common.cuh"
#include "column_stats.h"
#include "scan.cuh"

namespace mask {

// Strict load balance: every group holds exactly `workload` tiles, windows are cut wherever a
// group fills up (examples/src_fp32/sr_bcrs/testbed/main_strict_lb_16x8.cu:208-256).
static void strict_lb(const int32_t* soff, int32_t W, int32_t workload, std::vector<int32_t>& rbo,
                      std::vector<int32_t>& rb2w, std::vector<int32_t>& go) {
    rbo.clear(); rb2w.clear(); go.clear();
    go.push_back(0);
    int32_t load = 0;
    for (int32_t w = 0; w < W; w++) {
        int32_t s = soff[w];
        const int32_t e = soff[w + 1];
        while (s < e) {
            const int32_t take = std::min(workload - load, e - s);
            rbo.push_back(s);
            rb2w.push_back(w);
            s += take;
            load += take;
            if (load == workload) {
                go.push_back((int32_t)rb2w.size());
                load = 0;
            }
        }
    }
    rbo.push_back(soff[W]);
    if (load != 0 || go.size() == 1) go.push_back((int32_t)rb2w.size());
}

// Multi-binding: windows above twice the mean tile count (mean over all windows) are cut into
// ceil(x/mean) near-equal tasks (examples/src_fp32/sr_bcrs/testbed/main_multi_bind_16x8.cu:207-271).
static void multi_bind(const int32_t* soff, int32_t W, std::vector<int32_t>& task_win,
                       std::vector<int32_t>& win_split, std::vector<int32_t>& task_soff) {
    task_win.clear(); task_soff.clear();
    win_split.assign((size_t)W, 0);
    double sum = 0.0;
    for (int32_t w = 0; w < W; w++) sum += (double)(soff[w + 1] - soff[w]);
    const double avg = W > 0 ? sum / (double)W : 0.0;
    task_soff.push_back(0);
    for (int32_t w = 0; w < W; w++) {
        const int32_t x = soff[w + 1] - soff[w];
        if (x == 0) continue;
        int32_t parts = 1;
        if (avg > 0.0 && (double)x > 2.0 * avg) {
            parts = std::max(1, std::min((int32_t)std::ceil((double)x / avg), 9999));
            if (parts > 1) win_split[w] = 1;
        }
        const int32_t base = x / parts, rem = x % parts;
        for (int32_t i = 0; i < parts; i++) {
            task_win.push_back(w);
            task_soff.push_back(task_soff.back() + base + (i < rem ? 1 : 0));
        }
    }
}

// Tiles in one piece of a split window, and in one group of the warp-level kernel, when nobody asked for a
// size.  That kernel has 15 one-warp blocks per SM, each of which takes about half a microsecond per tile:
// with fewer than 128 tiles for every resident warp the pieces get shorter, so that all of them have work and
// no long chain of tiles is left at the end.  Not below kMinPiece, where filling a block's pipeline costs more
// than the balance gains, and not below the mean window: cutting every window adds a partial tile and a fix-up
// for each (uniform 4096-node matrix, 42 tiles a window, N = 512: 16.9 us whole, 23.8 us in three pieces).
// With very many tiles the pieces get longer again: the partial tiles are then what counts (2^22-node power-law
// graph, 15 M tiles, N = 512: pieces of 128 tiles write and read 5.6 GB of them, pieces of 512 0.6 GB).
constexpr int32_t kMinPiece = 16;
constexpr int32_t kWarpBlocksPerSm = 15;
constexpr int64_t kManyTiles = 30000;
static int32_t default_piece_tiles(int64_t T, int32_t W) {
    const int64_t resident = (int64_t)sm_count() * kWarpBlocksPerSm;
    const int64_t piece = std::max<int64_t>((T + resident - 1) / resident, (T + W - 1) / W);
    if (T > 128 * kManyTiles) return (int32_t)std::min<int64_t>(512, T / kManyTiles);
    return (int32_t)std::max<int64_t>(kMinPiece, std::min<int64_t>(128, piece));
}

static int32_t default_group_tiles(int64_t T) {
    // The SpMM grid is resident (two blocks per SM) and deals groups round-robin, so the blocks that
    // run at the same time work on neighbouring groups.  Groups are kept SHORT on purpose: what the
    // resident blocks touch together is then a narrow band of windows, and rows of B shared by
    // neighbouring windows (stencils, banded matrices) are fetched from DRAM once and found in L2
    // by the other blocks.  Groups of 800 tiles measured twice as slow as groups of 128 on a
    // 27-point stencil and on a power-law graph for exactly that reason.
    // Small matrices: one group per resident block (every group a block takes costs it a pipeline
    // restart, and with fewer groups than blocks nothing is left to balance).
    const int64_t resident = (int64_t)sm_count() * 2;
    const int64_t g = (T + resident - 1) / resident;
    return (int32_t)std::max<int64_t>(16, std::min<int64_t>(128, g));
}

// Fills the fragment / group tables of `p` from val_soff on the host: the reference's mappings, and one group per window.
static void build_tables(mask_plan& p, const int32_t* soff) {
    const int32_t W = p.W;
    const int32_t G = p.group_tiles;
    auto& fo = p.h_frag_off; auto& fw = p.h_frag_win; auto& go = p.h_group_off;
    fo.clear(); fw.clear(); go.clear();
    go.push_back(0);
    constexpr int kMaxFragsPerGroup = 32;

    if (p.policy == MASK_POLICY_STRICT_LB || p.policy == MASK_POLICY_MULTI_BIND) {
        // the reference tables, plus an empty fragment for every window without tiles so that
        // its rows of C are written
        std::vector<int32_t> rbo, rb2w, rgo, tsoff, wsplit;
        if (p.policy == MASK_POLICY_STRICT_LB) {
            strict_lb(soff, W, G, rbo, rb2w, rgo);
        } else {
            multi_bind(soff, W, rb2w, wsplit, tsoff);
            rbo = tsoff;
            rgo.resize(rb2w.size() + 1);
            for (size_t i = 0; i <= rb2w.size(); i++) rgo[i] = (int32_t)i;
        }
        const size_t nf = rb2w.size();
        size_t gi = 1;  // next reference group boundary to emit
        int32_t next_w = 0;
        int in_group = 0;
        for (size_t f = 0; f < nf; f++) {
            while (next_w < rb2w[f]) {  // windows skipped by the reference tables are empty
                fo.push_back(soff[next_w]); fw.push_back(next_w); next_w++;
                if (++in_group == kMaxFragsPerGroup) { go.push_back((int32_t)fw.size()); in_group = 0; }
            }
            next_w = std::max(next_w, rb2w[f] + 1);
            fo.push_back(rbo[f]); fw.push_back(rb2w[f]); in_group++;
            if (gi < rgo.size() && (size_t)rgo[gi] == f + 1) {
                go.push_back((int32_t)fw.size()); in_group = 0; gi++;
            }
        }
        while (next_w < W) {
            fo.push_back(soff[next_w]); fw.push_back(next_w); next_w++;
            if (++in_group == kMaxFragsPerGroup) { go.push_back((int32_t)fw.size()); in_group = 0; }
        }
        if (go.back() != (int32_t)fw.size()) go.push_back((int32_t)fw.size());
    } else {   // MASK_POLICY_ROW
        for (int32_t w = 0; w < W; w++) {
            fo.push_back(soff[w]); fw.push_back(w); go.push_back(w + 1);
        }
    }
    fo.push_back(soff[W]);

    p.F = (int64_t)fw.size();
    p.G = (int64_t)go.size() - 1;
}

// ---- MASK_POLICY_AUTO: tables built on the device ---------------------------------------------------
// A window of more than 5/4 of a piece is cut into near-equal pieces (each costs one partial tile in scratch, and
// the fix-up pass sums them in tile order).  Groups are runs of fragments of about equal cost: tiles plus
// kFragCost per fragment for the rows of C it writes.  Walking the windows one by one on the host, with their
// tile counts copied there and the tables back, took 0.4 ms for 65 536 windows; this takes 0.1.
constexpr int32_t kFragCost = 4;
constexpr int64_t kHigh = (int64_t)1 << 32;   // the scans carry two counts: one in each half

struct PlanCounts {          // on the device in front of the tables, and on the host
    int32_t frags, heads, groups, warp_groups, bad, group_pieces, warp_first, chunks_done;
    int32_t status[4];
};

struct TableArgs {
    const int32_t* soff;
    int32_t W, piece, group;
    int64_t T, max_frags;
    int32_t* frag_off; int32_t* frag_win; int32_t* frag_slot; int2* heads;
    int32_t* group_off; int32_t* group_tile;
    int4* warp_group; int4* warp_first;
    PlanCounts* counts;
    PlanCounts* host;        // pinned: the counts for the host, `bad` until the kernels that know them write them
    const int32_t* local;    // NULL: not known to be
    int32_t resident;        // resident blocks of the tcgen05 kernel
    int32_t takers;          // resident blocks of the warp-level kernel
    int32_t same_groups;     // the warp-level kernel takes the plan's own groups
};

struct PiecesIn {            // pieces of a window | 1 if it is split
    TableArgs a;
    __device__ int64_t operator()(int64_t w) const {
        const int64_t x = a.soff[w + 1] - a.soff[w], piece = a.piece;
        return x > piece + piece / 4 ? (x + piece - 1) / piece + kHigh : 1;
    }
};
struct PiecesOut {
    TableArgs a;
    __device__ void operator()(int64_t w, int64_t before, int64_t v) const {
        const int64_t first = before & (kHigh - 1), parts = v & (kHigh - 1);
        const int32_t split_before = (int32_t)(before >> 32);
        const bool split = v >= kHigh;
        const int32_t s = a.soff[w], x = a.soff[w + 1] - s;
        if (w == 0) {
            for (int i = 0; i < 4; i++) a.counts->status[i] = 0;
            if (s != 0) a.counts->bad = 1;
        }
        if (first + parts > a.max_frags || x < 0) {   // only if val_soff is not what it should be
            a.counts->bad = 1;
            return;
        }
        const int32_t base = (int32_t)(x / parts), rem = (int32_t)(x % parts);
        const int32_t slot = split ? (int32_t)(first - (w - split_before)) : -1;   // unsplit windows are one fragment each
        int32_t at = s;
        for (int32_t i = 0; i < parts; i++) {
            a.frag_off[first + i] = at;
            a.frag_win[first + i] = (int32_t)w;
            a.frag_slot[first + i] = split ? slot + i : -1;
            at += base + (i < rem ? 1 : 0);
        }
        if (split) a.heads[split_before] = make_int2((int)first, (int)parts);
        const int64_t group = a.group;
        if (x > group + group / 4) atomicAdd(&a.counts->group_pieces, (int32_t)((x + group - 1) / group));
        if (w == a.W - 1) {
            a.frag_off[first + parts] = at;
            if (at != a.T) a.counts->bad = 1;
            a.counts->frags = (int32_t)(first + parts);
            a.counts->heads = split_before + (split ? 1 : 0);
        }
    }
};

__device__ __forceinline__ int64_t cost_before(const TableArgs& a, int64_t f) { return (int64_t)a.frag_off[f] + kFragCost * f; }

// The tcgen05 kernel's groups.  Its blocks take every resident-th group, so there are a whole number of groups for
// each of them, of at most 9/8 of the plan's group size (100 000 rows, N = 100: 4.02 rounds 85 us, 4 rounds 72 us).
// A fragment belongs to the group that the cost before its middle falls into.
struct GroupsIn {
    TableArgs a;
    __device__ int32_t operator()(int64_t f) const {
        const int32_t F = a.counts->frags;
        if (a.counts->bad || f >= F) return 0;
        if (f == 0) return 1;
        const int64_t total = a.T + (int64_t)kFragCost * F;
        const int64_t c0 = cost_before(a, f - 1), c1 = cost_before(a, f), c2 = cost_before(a, f + 1);
        int64_t size2 = 2 * (int64_t)a.group;
        if (!a.same_groups) {
            const int64_t most = (int64_t)a.resident * (a.group + a.group / 8), rounds = (total + most - 1) / most;
            size2 = 2 * total / (a.resident * rounds) + 1;
            if (size2 < 2 * kMinPiece) size2 = 2 * kMinPiece;
        }
        return (c0 + c1) / size2 != (c1 + c2) / size2;
    }
};
struct GroupsOut {
    TableArgs a;
    __device__ void operator()(int64_t f, int64_t before, int32_t v) const {
        const int32_t F = a.counts->frags;
        if (a.counts->bad || f >= F) return;
        const int32_t g = (int32_t)before;
        if (v) { a.group_off[g] = (int32_t)f; a.group_tile[g] = a.frag_off[f]; }
        if (f == F - 1) {
            a.group_off[g + v] = F;
            a.group_tile[g + v] = (int32_t)a.T;
            a.counts->groups = g + v;
            a.host->frags = F;
            a.host->heads = a.counts->heads;
            a.host->groups = g + v;
            a.host->group_pieces = a.counts->group_pieces;
            a.host->bad = 0;
        }
    }
};

// The warp-level kernel's groups: runs of fragments, closed before their cost passes 5/4 of a target.
//
// Balance: 15 x 148 blocks are resident and take groups in order as they come free, so the target is a resident
// block's share of the cost still left, between 16 and 128 tiles: long groups first, short ones at the end.  Twice
// the share leaves a second round half empty (100 000 rows, 20 tiles a window, N = 64: 67 us against 44), half of it
// starts more blocks for nothing (a start costs about three tiles' time; power-law graph with 130 000 nodes, N = 48:
// 82 us against 80), and groups cut by the middles of their fragments as above are too uneven (N = 64: 46 us).
// Locality: what the resident warps touch together should stay in L2; where windows share rows of B with their
// neighbours, short groups keep the band narrow (27-point stencil with 10^6 rows, N = 128: one window a group
// 517 us, 128 tiles a group 585 us).
//
// A fragment that alone is far more than the target of its place would still run when everything else has ended: its warp
// takes 0.6 to 1 us a tile, and 150 tiles begun 165 us into a product kept it going from 190 to 248 us.  Such groups are listed
// a second time, to be taken before all others, and are empty in their place (power-law graphs, N = 128: 300 000 nodes 211 -> 171 us,
// in ME-TCF 251 -> 201, 130 000 nodes 103 -> 84; N = 512 3 to 7 %).  The line at 3/2 of where a group ends: at twice that, 130 000 nodes
// 88 us; shorter pieces instead cost more in the fix-up than they even out (two thirds of a piece: 86 us, 1 1/2: 94).
//
// Where a group ends depends on where it begins, so this is a walk; but from every fragment the end is known at
// once.  Pointer doubling in shared memory finds for every fragment of a chunk where a walk that enters there leaves
// the chunk and after how many groups; one thread then walks from chunk to chunk; and every chunk writes the groups of
// the walk that enters it, itself cut into 32 parts in the same way.
constexpr int kChunk = 2048, kChunkThreads = 1024, kPart = kChunk / 32;   // a group has at most 41 fragments: less than a part

__device__ __forceinline__ int64_t warp_group_target(const TableArgs& a, int64_t c, int64_t total) {
    if (a.local && *a.local) return kMinPiece;
    const int64_t target = (total - c) / a.takers;
    return target < kMinPiece ? kMinPiece : (target > 128 ? 128 : target);
}
__device__ __forceinline__ int64_t warp_group_end(const TableArgs& a, int64_t f, int64_t F, int64_t total) {
    const int64_t c = cost_before(a, f), target = warp_group_target(a, c, total);
    const int64_t limit = c + target * 5 / 4;
    int64_t lo = f + 1, hi = f + 2 + target * 5 / 4 / kFragCost;   // the end is in [lo, hi)
    if (hi > F + 1) hi = F + 1;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (cost_before(a, mid) <= limit) lo = mid; else hi = mid;
    }
    return lo;
}

// to[i] (i of n): next fragment of a walk -> where the walk leaves i's block of `width`; cnt[i]: groups begun there
__device__ __forceinline__ void double_pointers(int32_t* to, int32_t* cnt, int n, int width) {
    constexpr int kPer = kChunk / kChunkThreads;
    for (int step = 1; step < width; step *= 2) {
        int32_t t[kPer], c[kPer];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            const int i = j * kChunkThreads + threadIdx.x, end = min(n, (i / width + 1) * width);
            const bool inside = i < n && to[i] < end;
            t[j] = inside ? to[to[i]] : (i < n ? to[i] : 0);
            c[j] = inside ? cnt[i] + cnt[to[i]] : (i < n ? cnt[i] : 0);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            const int i = j * kChunkThreads + threadIdx.x;
            if (i < n) { to[i] = t[j]; cnt[i] = c[j]; }
        }
    }
    __syncthreads();
}

// exit_to[f], groups[f]: where a walk that enters its chunk at f leaves it, and how many groups it begins there
__global__ void __launch_bounds__(kChunkThreads) warp_group_jumps_kernel(const TableArgs a, int32_t* __restrict__ exit_to, int32_t* __restrict__ groups) {
    __shared__ int32_t to[kChunk], cnt[kChunk];
    const int64_t F = a.counts->frags, base = (int64_t)blockIdx.x * kChunk;
    if (a.counts->bad || base >= F) return;
    const int n = (int)(F - base < kChunk ? F - base : kChunk);
    const int64_t total = a.T + (int64_t)kFragCost * F;
    for (int i = threadIdx.x; i < n; i += kChunkThreads) {
        to[i] = (int32_t)(warp_group_end(a, base + i, F, total) - base);
        cnt[i] = 1;
    }
    double_pointers(to, cnt, n, kChunk);
    for (int i = threadIdx.x; i < n; i += kChunkThreads) {
        exit_to[base + i] = (int32_t)base + to[i];
        groups[base + i] = cnt[i];
    }
}
// entry[c], first[c]: where the walk from fragment 0 enters chunk c, and how many groups begin before.  A group is shorter than a
// chunk, but not than what is left for the last one: that can be passed over, and is then entered behind its end.
__global__ void warp_group_walk_kernel(const TableArgs a, const int32_t* __restrict__ exit_to, const int32_t* __restrict__ groups,
                                       int32_t* __restrict__ entry, int32_t* __restrict__ first) {
    const int32_t F = a.counts->frags;
    if (a.counts->bad) return;
    int32_t f = 0, g = 0;
    for (int64_t c = 0; c * kChunk < F; c++) {
        entry[c] = f;
        first[c] = g;
        if (f < F) {
            g += groups[f];
            f = exit_to[f];
        }
    }
}
__global__ void __launch_bounds__(kChunkThreads) warp_group_write_kernel(const TableArgs a, const int32_t* __restrict__ entry, const int32_t* __restrict__ first) {
    __shared__ int32_t next[kChunk], to[kChunk], cnt[kChunk], part_entry[32], part_first[32];
    const int64_t F = a.counts->frags, base = (int64_t)blockIdx.x * kChunk;
    if (a.counts->bad || base >= F) return;
    const int n = (int)(F - base < kChunk ? F - base : kChunk);
    const int64_t total = a.T + (int64_t)kFragCost * F;
    for (int i = threadIdx.x; i < n; i += kChunkThreads) {
        next[i] = to[i] = (int32_t)(warp_group_end(a, base + i, F, total) - base);
        cnt[i] = 1;
    }
    double_pointers(to, cnt, n, kPart);
    if (threadIdx.x == 0) {
        int32_t i = entry ? entry[blockIdx.x] - (int32_t)base : 0, g = first ? first[blockIdx.x] : 0;
        for (int p = 0; p < 32; p++) {
            part_entry[p] = i;
            part_first[p] = g;
            if (i < n) { g += cnt[i]; i = to[i]; }
        }
        if (base + n == F) a.host->warp_groups = g;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kChunkThreads) to[i] = -1;   // from here on: number of the group that begins here
    __syncthreads();
    if (threadIdx.x < 32) {
        const int end = min(n, ((int)threadIdx.x + 1) * kPart);
        int32_t g = part_first[threadIdx.x];
        for (int32_t i = part_entry[threadIdx.x]; i < end; i = next[i], g++) to[i] = g;
    }
    __syncthreads();
    const bool local = a.local && *a.local;
    for (int i = threadIdx.x; i < n; i += kChunkThreads) {
        if (to[i] < 0) continue;
        const int64_t f = base + i;
        const int32_t t0 = a.frag_off[f];
        int4 group = make_int4((int)f, (int)(base + next[i]), t0, a.frag_off[base + next[i]] - t0);
        if (!local && next[i] == i + 1 && 2 * (group.w + kFragCost) > 3 * (warp_group_target(a, cost_before(a, f), total) * 5 / 4)) {
            a.warp_first[atomicAdd(&a.counts->warp_first, 1)] = group;   // in any order: groups do not depend on one another
            group.y = group.x;
        }
        a.warp_group[to[i]] = group;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&a.counts->chunks_done, 1) == (F + kChunk - 1) / kChunk - 1) a.host->warp_first = *(volatile int32_t*)&a.counts->warp_first;
    }
}

// Groups listed first have more than 3/2 5/4 kMinPiece - kFragCost = 26 tiles.
static int64_t warp_first_max(int64_t T) { return T / 26 + 1; }

static int enqueue_warp_groups(const TableArgs& a, DevScratch& work, cudaStream_t st) {
    const int64_t chunks = (a.max_frags + kChunk - 1) / kChunk;
    int32_t *entry = nullptr, *first = nullptr;
    if (chunks > 1) {
        int rc = work.alloc((size_t)(2 * a.max_frags + 2 * chunks) * 4, st);
        if (rc != MASK_OK) return rc;
        int32_t* exit_to = work.as<int32_t>();
        int32_t* groups = exit_to + a.max_frags;
        entry = groups + a.max_frags;
        first = entry + chunks;
        warp_group_jumps_kernel<<<(unsigned)chunks, kChunkThreads, 0, st>>>(a, exit_to, groups);
        MASK_CUDA_TRY(cudaGetLastError());
        warp_group_walk_kernel<<<1, 1, 0, st>>>(a, exit_to, groups, entry, first);
        MASK_CUDA_TRY(cudaGetLastError());
    }
    warp_group_write_kernel<<<(unsigned)chunks, kChunkThreads, 0, st>>>(a, entry, first);
    MASK_CUDA_TRY(cudaGetLastError());
    return MASK_OK;
}

// Enqueues the tables of an AUTO plan; their sizes are in `counts` (pinned) when they are complete.
static int enqueue_auto_tables(mask_plan& p, const int32_t* d_val_soff, bool same_groups, const int32_t* d_local, DevScratch& spine,
                               DevScratch& work, PlanCounts* counts, cudaStream_t st) {
    TableArgs a{};
    a.soff = d_val_soff;
    a.W = p.W;
    a.piece = p.piece_tiles;
    a.group = p.group_tiles;
    a.T = p.T;
    a.max_frags = (int64_t)p.W + p.T / p.piece_tiles + 1;
    a.local = d_local;
    a.resident = 2 * sm_count();
    a.takers = sm_count() * kWarpBlocksPerSm;
    a.same_groups = same_groups;
    a.host = counts;
    *counts = PlanCounts{};
    counts->bad = 1;
    if (a.max_frags >= ((int64_t)1 << 31) - 1) return fail(MASK_ERR_INDEX_OVERFLOW, "the number of tasks does not fit int32");
    size_t at = sizeof(PlanCounts) / 4;
    auto section = [&](int64_t n) { const size_t o = at; at += ((size_t)n + 3) & ~(size_t)3; return o; };
    const int64_t n = a.max_frags;
    const size_t o_fo = section(n + 1), o_fw = section(n), o_fs = section(n), o_go = section(n + 1), o_gt = section(n + 1),
                 o_wg = section(4 * n), o_wf = section(4 * warp_first_max(p.T)), o_hd = section(2 * std::min<int64_t>(p.W, p.T / p.piece_tiles + 1));
    int rc = device_alloc(reinterpret_cast<void**>(&p.d_tables), at * sizeof(int32_t), st);
    if (rc == MASK_OK) rc = spine.alloc(scan_spine_words(n) * 8, st);
    if (rc != MASK_OK) return rc;
    a.counts = reinterpret_cast<PlanCounts*>(p.d_tables);
    a.frag_off = p.d_frag_off = p.d_tables + o_fo;
    a.frag_win = p.d_frag_win = p.d_tables + o_fw;
    a.frag_slot = p.d_frag_slot = p.d_tables + o_fs;
    a.group_off = p.d_group_off = p.d_tables + o_go;
    a.group_tile = p.d_group_tile = p.d_tables + o_gt;
    a.warp_group = reinterpret_cast<int4*>(p.d_tables + o_wg);
    a.warp_first = reinterpret_cast<int4*>(p.d_tables + o_wf);
    p.d_warp_group = same_groups ? nullptr : a.warp_group;
    p.d_warp_first = a.warp_first;
    a.heads = reinterpret_cast<int2*>(p.d_tables + o_hd);
    p.d_heads = a.heads;
    p.d_status = p.d_tables + offsetof(PlanCounts, status) / 4;
    MASK_CUDA_TRY(cudaMemsetAsync(a.counts, 0, sizeof(PlanCounts), st));
    rc = device_scan(PiecesIn{a}, PiecesOut{a}, p.W, spine.as<int64_t>(), st);
    if (rc == MASK_OK) rc = device_scan(GroupsIn{a}, GroupsOut{a}, n, spine.as<int64_t>(), st);
    if (rc == MASK_OK && !same_groups) rc = enqueue_warp_groups(a, work, st);
    if (rc != MASK_OK) return rc;
    return MASK_OK;
}

// One device array for all tables, filled by one copy: sections start on 16-byte boundaries.
static int upload_tables(mask_plan& p, const int32_t* soff, cudaStream_t st) {
    const auto& fo = p.h_frag_off; const auto& fw = p.h_frag_win; const auto& go = p.h_group_off;
    p.Gw = p.G;
    // split windows: first fragment and number of pieces; pieces are numbered in fragment order
    std::vector<int32_t> heads;
    p.P = 0;
    auto whole = [&](int64_t f) { return fo[f] == soff[fw[f]] && fo[f + 1] == soff[fw[f] + 1]; };
    for (int64_t f = 0; f < p.F; f++) {
        if (whole(f)) continue;
        if (f == 0 || fw[f - 1] != fw[f]) { heads.push_back((int32_t)f); heads.push_back(0); }
        heads.back()++;
        p.P++;
    }
    p.H = (int64_t)heads.size() / 2;
    p.P_group = p.P;
    size_t at = 0;
    auto section = [&](size_t n) { const size_t o = at; at += (n + 3) & ~(size_t)3; return o; };
    const size_t o_fo = section(fo.size()), o_fw = section(fw.size()), o_fs = section(fw.size()), o_go = section(go.size()),
                 o_gt = section(go.size()), o_hd = section(heads.size()), o_st = section(4);
    HostStage stage;
    int rc = stage.get(at * sizeof(int32_t));
    if (rc != MASK_OK) return rc;
    int32_t* h = stage.as<int32_t>();
    std::copy(fo.begin(), fo.end(), h + o_fo);
    std::copy(fw.begin(), fw.end(), h + o_fw);
    std::copy(go.begin(), go.end(), h + o_go);
    std::copy(heads.begin(), heads.end(), h + o_hd);
    std::fill(h + o_st, h + o_st + 4, 0);
    int32_t slot = 0;
    for (int64_t f = 0; f < p.F; f++) h[o_fs + f] = whole(f) ? -1 : slot++;
    for (size_t g = 0; g < go.size(); g++) h[o_gt + g] = fo[go[g]];
    rc = device_alloc(reinterpret_cast<void**>(&p.d_tables), at * sizeof(int32_t), st);
    if (rc != MASK_OK) return rc;
    p.d_frag_off = p.d_tables + o_fo;
    p.d_frag_win = p.d_tables + o_fw;
    p.d_frag_slot = p.d_tables + o_fs;
    p.d_group_off = p.d_tables + o_go;
    p.d_group_tile = p.d_tables + o_gt;
    p.d_heads = reinterpret_cast<const int2*>(p.d_tables + o_hd);
    p.d_status = p.d_tables + o_st;
    cudaError_t e = cudaMemcpyAsync(p.d_tables, h, at * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);   // the plan may be used on any stream from here on
    MASK_CUDA_TRY(e);
    MASK_CUDA_TRY(e2);
    return MASK_OK;
}

}  // namespace mask

extern "C" int mask_plan_strict_lb(const int32_t* h_val_soff, int32_t M, int32_t workload, int32_t* row_block_offset,
                                   int32_t* row_block_to_window, int32_t* group_offset, int64_t* n_frag,
                                   int64_t* n_groups) {
    using namespace mask;
    MASK_REQUIRE(h_val_soff != nullptr && M >= 1 && workload >= 1 && n_frag && n_groups, "bad arguments");
    return without_exceptions([&] {
        std::vector<int32_t> rbo, rb2w, go;
        strict_lb(h_val_soff, window_count(M), workload, rbo, rb2w, go);
        *n_frag = (int64_t)rb2w.size();
        *n_groups = (int64_t)go.size() - 1;
        if (row_block_offset) std::memcpy(row_block_offset, rbo.data(), rbo.size() * sizeof(int32_t));
        if (row_block_to_window && !rb2w.empty()) std::memcpy(row_block_to_window, rb2w.data(), rb2w.size() * sizeof(int32_t));
        if (group_offset) std::memcpy(group_offset, go.data(), go.size() * sizeof(int32_t));
        return MASK_OK;
    });
}

extern "C" int mask_plan_multi_bind(const int32_t* h_val_soff, int32_t M, int32_t* task_window, int32_t* window_split,
                                    int32_t* task_soff, int64_t* n_tasks) {
    using namespace mask;
    MASK_REQUIRE(h_val_soff != nullptr && M >= 1 && n_tasks, "bad arguments");
    return without_exceptions([&] {
        std::vector<int32_t> tw, ws, ts;
        multi_bind(h_val_soff, window_count(M), tw, ws, ts);
        *n_tasks = (int64_t)tw.size();
        if (task_window && !tw.empty()) std::memcpy(task_window, tw.data(), tw.size() * sizeof(int32_t));
        if (window_split && !ws.empty()) std::memcpy(window_split, ws.data(), ws.size() * sizeof(int32_t));
        if (task_soff) std::memcpy(task_soff, ts.data(), ts.size() * sizeof(int32_t));
        return MASK_OK;
    });
}

namespace mask {

// With d_val_sidx the column features are measured and the plan table is applied as well.
static int create_plan(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int policy,
                       int32_t group_tiles, cudaStream_t st, mask_plan** out) {
    mask_plan* p = new (std::nothrow) mask_plan();
    if (!p) return fail(MASK_ERR_OUT_OF_MEMORY, "out of host memory");
    p->M = M;
    p->W = window_count(M);
    p->T = T;
    p->policy = policy;
    p->group_tiles = group_tiles > 0 ? group_tiles : (policy == MASK_POLICY_STRICT_LB ? 64 : default_group_tiles(T));
    // a piece may be longer than a group: it then is a group of its own
    p->piece_tiles = (group_tiles > 0 || policy != MASK_POLICY_AUTO) ? p->group_tiles : default_piece_tiles(T, p->W);
    HostStage stage;
    ColumnStatsJob job;
    DevScratch spine, work;
    auto body = [&]() -> int {
        MASK_CUDA_TRY(cudaGetDevice(&p->device));
        int rc = d_val_sidx ? job.enqueue(d_val_soff, d_val_sidx, M, K, T, 512, st) : MASK_OK;
        if (rc != MASK_OK) return rc;
        const bool on_device = policy == MASK_POLICY_AUTO;
        const size_t bytes = on_device ? sizeof(PlanCounts) : ((size_t)p->W + 1) * sizeof(int32_t);
        rc = stage.get(bytes);
        if (rc != MASK_OK) return rc;
        if (on_device) {
            rc = enqueue_auto_tables(*p, d_val_soff, group_tiles > 0, job.device_local(), spine, work, stage.as<PlanCounts>(), st);
            if (rc != MASK_OK) return rc;
        } else {
            MASK_CUDA_TRY(cudaMemcpyAsync(stage.as<int32_t>(), d_val_soff, bytes, cudaMemcpyDeviceToHost, st));
        }
        MASK_CUDA_TRY(cudaStreamSynchronize(st));   // the plan may be used on any stream from here on
        if (d_val_sidx) {
            mask_column_features f;
            job.finish(&f);
            choose_plan_parameters(p, f);
        }
        if (on_device) {
            const PlanCounts& c = *stage.as<PlanCounts>();
            if (c.bad) return fail(MASK_ERR_INVALID_ARGUMENT, "val_soff does not start at 0 / end at T");
            p->F = c.frags;
            p->H = c.heads;
            p->P = p->F - (p->W - p->H);
            p->P_group = c.group_pieces;
            p->G = c.groups;
            p->Gw = group_tiles > 0 ? p->G : c.warp_groups;
            p->warp_first = group_tiles > 0 ? 0 : c.warp_first;
            return MASK_OK;
        }
        const int32_t* soff = stage.as<int32_t>();
        if (soff[0] != 0 || (int64_t)soff[p->W] != T) return fail(MASK_ERR_INVALID_ARGUMENT, "val_soff does not start at 0 / end at T");
        if (policy == MASK_POLICY_REF_AUTO) {  // the bridge's automatic choice between its own two mappings
            mask_features f;
            mask_features_from_soff(soff, M, 0, &f);
            p->policy = f.heavy_tail ? MASK_POLICY_STRICT_LB : MASK_POLICY_ROW;
            if (group_tiles <= 0) p->group_tiles = 64;
        }
        build_tables(*p, soff);
        return upload_tables(*p, soff, st);
    };
    const int rc = without_exceptions(body);
    if (rc != MASK_OK) cudaStreamSynchronize(st);   // copies into the staging buffers may be in flight
    if (rc != MASK_OK) {
        mask_plan_destroy(p);
        return rc;
    }
    *out = p;
    return MASK_OK;
}

}  // namespace mask

extern "C" int mask_plan_create(const int32_t* d_val_soff, int32_t M, int64_t T, int policy, int32_t group_tiles,
                                void* stream, mask_plan** out) {
    using namespace mask;
    MASK_REQUIRE(out != nullptr, "out is NULL");
    *out = nullptr;
    MASK_REQUIRE(d_val_soff != nullptr && M >= 1 && T >= 0, "bad arguments");
    MASK_REQUIRE(policy >= MASK_POLICY_AUTO && policy <= MASK_POLICY_REF_AUTO, "unknown policy");
    if (T >= (int64_t)1 << 31) return fail(MASK_ERR_INDEX_OVERFLOW, "T does not fit int32");
    return create_plan(d_val_soff, nullptr, M, 0, T, policy, group_tiles, static_cast<cudaStream_t>(stream), out);
}

extern "C" int mask_plan_create_tuned(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int policy,
                                      int32_t group_tiles, void* stream, mask_plan** out) {
    using namespace mask;
    MASK_REQUIRE(out != nullptr, "out is NULL");
    *out = nullptr;
    MASK_REQUIRE(d_val_soff != nullptr && M >= 1 && K >= 1 && T >= 0, "bad arguments");
    MASK_REQUIRE(T == 0 || d_val_sidx != nullptr, "val_sidx is NULL");
    MASK_REQUIRE(policy >= MASK_POLICY_AUTO && policy <= MASK_POLICY_REF_AUTO, "unknown policy");
    if (T >= (int64_t)1 << 31) return fail(MASK_ERR_INDEX_OVERFLOW, "T does not fit int32");
    return create_plan(d_val_soff, T > 0 ? d_val_sidx : nullptr, M, K, T, policy, group_tiles, static_cast<cudaStream_t>(stream), out);
}

extern "C" void mask_plan_destroy(mask_plan* p) {
    if (!p) return;
    // kernels that read the tables may still be running on any stream
    int cur = -1;
    const bool elsewhere = p->d_tables && cudaGetDevice(&cur) == cudaSuccess && cur != p->device;
    if (elsewhere) cudaSetDevice(p->device);
    if (p->d_tables) {
        cudaDeviceSynchronize();
        mask::device_free(p->d_tables, nullptr);
    }
    cudaFree(p->d_vals_tf32);
    if (elsewhere) cudaSetDevice(cur);
    delete p;
}

extern "C" size_t mask_plan_scratch_bytes(const mask_plan* p, int32_t N) {
    if (!p || N <= 0) return 0;
    return (size_t)p->P * mask::kWinRows * (size_t)N * sizeof(float);
}

extern "C" int mask_plan_info(const mask_plan* p, int64_t* n_frag, int64_t* n_groups, int64_t* n_partial,
                              int32_t* group_tiles) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr, "plan is NULL");
    if (n_frag) *n_frag = p->F;
    if (n_groups) *n_groups = p->G;
    if (n_partial) *n_partial = p->P;
    if (group_tiles) *group_tiles = p->group_tiles;
    return MASK_OK;
}

extern "C" int mask_plan_warp_groups(const mask_plan* p, int64_t* n_first, int64_t* n_groups, int32_t* h_groups) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr, "plan is NULL");
    if (n_first) *n_first = p->warp_first;
    if (n_groups) *n_groups = p->Gw;
    if (!h_groups || p->Gw == 0) return MASK_OK;
    if (p->warp_first) MASK_CUDA_TRY(cudaMemcpy(h_groups, p->d_warp_first, (size_t)p->warp_first * sizeof(int4), cudaMemcpyDeviceToHost));
    h_groups += 4 * (size_t)p->warp_first;
    if (p->d_warp_group) {
        MASK_CUDA_TRY(cudaMemcpy(h_groups, p->d_warp_group, (size_t)p->Gw * sizeof(int4), cudaMemcpyDeviceToHost));
        return MASK_OK;
    }
    std::vector<int32_t> off((size_t)p->Gw + 1), tile((size_t)p->Gw + 1);
    MASK_CUDA_TRY(cudaMemcpy(off.data(), p->d_group_off, off.size() * sizeof(int32_t), cudaMemcpyDeviceToHost));
    MASK_CUDA_TRY(cudaMemcpy(tile.data(), p->d_group_tile, tile.size() * sizeof(int32_t), cudaMemcpyDeviceToHost));
    for (int64_t i = 0; i < p->Gw; i++, h_groups += 4) {
        h_groups[0] = off[i];
        h_groups[1] = off[i + 1];
        h_groups[2] = tile[i];
        h_groups[3] = tile[i + 1] - tile[i];
    }
    return MASK_OK;
}

extern "C" int mask_plan_set_row_map(mask_plan* p, const int32_t* d_row_order) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr, "plan is NULL");
    p->d_row_map = d_row_order;
    return MASK_OK;
}

extern "C" int mask_plan_set_peer_outputs(mask_plan* p, float* const* d_peer_ptrs, int32_t n_peers) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr, "plan is NULL");
    MASK_REQUIRE(n_peers >= 0 && n_peers <= 15 && (n_peers == 0 || d_peer_ptrs != nullptr), "bad peer list");
    p->d_peer_out = n_peers ? d_peer_ptrs : nullptr;
    p->n_peer_out = n_peers;
    return MASK_OK;
}

extern "C" int mask_plan_status(const mask_plan* p, int32_t* h_status, void* stream) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr && h_status != nullptr, "NULL argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    MASK_CUDA_TRY(cudaMemcpyAsync(h_status, p->d_status, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    MASK_CUDA_TRY(cudaMemsetAsync(p->d_status, 0, sizeof(int32_t), st));   // one expiry must not mark every later call
    MASK_CUDA_TRY(cudaStreamSynchronize(st));
    return MASK_OK;
}

extern "C" int mask_plan_export(const mask_plan* p, int32_t* frag_offset, int32_t* frag_window, int32_t* group_offset) {
    using namespace mask;
    MASK_REQUIRE(p != nullptr, "plan is NULL");
    if (p->policy == MASK_POLICY_AUTO) {   // these tables were built on the device
        if (frag_offset) MASK_CUDA_TRY(cudaMemcpy(frag_offset, p->d_frag_off, ((size_t)p->F + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost));
        if (frag_window && p->F) MASK_CUDA_TRY(cudaMemcpy(frag_window, p->d_frag_win, (size_t)p->F * sizeof(int32_t), cudaMemcpyDeviceToHost));
        if (group_offset) MASK_CUDA_TRY(cudaMemcpy(group_offset, p->d_group_off, ((size_t)p->G + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost));
        return MASK_OK;
    }
    if (frag_offset) std::memcpy(frag_offset, p->h_frag_off.data(), p->h_frag_off.size() * sizeof(int32_t));
    if (frag_window && p->F) std::memcpy(frag_window, p->h_frag_win.data(), p->h_frag_win.size() * sizeof(int32_t));
    if (group_offset) std::memcpy(group_offset, p->h_group_off.data(), p->h_group_off.size() * sizeof(int32_t));
    return MASK_OK;
}
