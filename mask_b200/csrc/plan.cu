// Task planners (host) and the execution-plan handle.
#include "plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "column_stats.h"

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
// for each (uniform 4096-node matrix, 42 tiles a window, N = 512: 23 us whole, 29 us in three pieces).
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

// Fills the fragment / group tables of `p` from val_soff on the host.
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
    } else {
        // Groups are closed on fragment boundaries once their cost (tiles plus a fixed share per fragment
        // for the rows of C it writes) reaches G; a window of more than 5/4 of a piece is cut into near-equal
        // pieces (each piece costs one partial tile in scratch and the fix-up pass sums them in tile order).
        constexpr int32_t kWindowCost = 4;
        const int32_t piece = p.piece_tiles;
        const int32_t split_above = piece + piece / 4;
        const size_t most = (size_t)W + (size_t)(p.T / std::max(piece, 1)) + 1;   // fragments
        fo.resize(most + 1);
        fw.resize(most);
        go.resize(most + 1);
        int32_t *fo_at = fo.data(), *fw_at = fw.data(), *go_at = go.data() + 1;
        int32_t load = 0, n_frag = 0, closed = 0;
        auto add = [&](int32_t tile, int32_t w) { *fo_at++ = tile; *fw_at++ = w; n_frag++; };
        auto close = [&]() {
            if (closed != n_frag) *go_at++ = closed = n_frag;
            load = 0;
        };
        for (int32_t w = 0; w < W; w++) {
            const int32_t s = soff[w], x = soff[w + 1] - s;
            if (p.policy == MASK_POLICY_ROW) {
                add(s, w); close();
                continue;
            }
            if (x > split_above) {
                const int32_t parts = (x + piece - 1) / piece, base = x / parts, rem = x % parts;
                int32_t at = s;
                if (piece >= G) close();
                for (int32_t i = 0; i < parts; i++) {
                    add(at, w);
                    at += base + (i < rem ? 1 : 0);
                    load += base + kWindowCost;
                    if (load >= G || piece >= G) close();
                }
                continue;
            }
            if (load > 0 && load + x + kWindowCost > G + G / 8) close();
            add(s, w);
            load += x + kWindowCost;
            if (load >= G) close();
        }
        close();
        fo.resize(n_frag);
        fw.resize(n_frag);
        go.resize(go_at - go.data());
    }
    fo.push_back(soff[W]);

    p.F = (int64_t)fw.size();
    p.G = (int64_t)go.size() - 1;

}

// Groups of the warp-level kernel: the same fragments in shorter runs, closed before their cost passes 5/4 of a
// target.  Two reasons to keep them short.  Balance: 15 x 148 blocks are resident and take groups in order as they
// come free, so the target is a resident block's share of what is still left: long groups first, short ones at
// the end.  Twice the share leaves a second round half empty (100 000 rows, 20 tiles a window, N = 64: 67 us
// against 44), half of it starts more blocks for nothing (a start costs about three tiles' time; power-law graph
// with 130 000 nodes, N = 48: 82 us against 80).  Locality: what the resident warps touch together should stay
// in L2; where windows share rows of B with their neighbours, a window a group keeps the band narrow
// (27-point stencil with 10^6 rows, N = 128: 517 us, with 128 tiles a group 585 us).
static void build_warp_groups(mask_plan& p) {
    p.h_warp_off.clear();
    if (p.policy != MASK_POLICY_AUTO || !p.auto_groups) return;   // the plan's own groups
    constexpr int32_t kFragCost = 4, kMaxTarget = 128;
    const int64_t takers = (int64_t)sm_count() * kWarpBlocksPerSm;
    const auto& fo = p.h_frag_off;
    int64_t left = p.T + kFragCost * p.F;   // cost of the fragments not dealt yet
    auto target_now = [&]() { return p.local ? (int64_t)kMinPiece : std::max<int64_t>(kMinPiece, std::min<int64_t>(kMaxTarget, left / takers)); };
    int64_t load = 0, limit = target_now() * 5 / 4;
    p.h_warp_off.reserve((size_t)p.F + 1);
    p.h_warp_off.push_back(0);
    for (int64_t f = 0; f < p.F; f++) {
        const int64_t cost = fo[f + 1] - fo[f] + kFragCost;
        if (load > 0 && load + cost > limit) {
            p.h_warp_off.push_back((int32_t)f);
            left -= load;
            load = 0;
            limit = target_now() * 5 / 4;
        }
        load += cost;
    }
    if (p.F > 0) p.h_warp_off.push_back((int32_t)p.F);
}

// One device array for all tables, filled by one copy: sections start on 16-byte boundaries.
static int upload_tables(mask_plan& p, const int32_t* soff, cudaStream_t st) {
    const auto& fo = p.h_frag_off; const auto& fw = p.h_frag_win; const auto& go = p.h_group_off;
    const auto& wo = p.h_warp_off.empty() ? p.h_group_off : p.h_warp_off;
    p.Gw = (int64_t)wo.size() - 1;
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
    size_t at = 0;
    auto section = [&](size_t n) { const size_t o = at; at += (n + 3) & ~(size_t)3; return o; };
    const size_t o_fo = section(fo.size()), o_fw = section(fw.size()), o_fs = section(fw.size()), o_go = section(go.size()),
                 o_gt = section(go.size()), o_wo = section(wo.size()), o_wt = section(wo.size()), o_hd = section(heads.size()),
                 o_st = section(4);
    HostStage stage;
    int rc = stage.get(at * sizeof(int32_t));
    if (rc != MASK_OK) return rc;
    int32_t* h = stage.as<int32_t>();
    std::copy(fo.begin(), fo.end(), h + o_fo);
    std::copy(fw.begin(), fw.end(), h + o_fw);
    std::copy(go.begin(), go.end(), h + o_go);
    std::copy(wo.begin(), wo.end(), h + o_wo);
    std::copy(heads.begin(), heads.end(), h + o_hd);
    std::fill(h + o_st, h + o_st + 4, 0);
    int32_t slot = 0;
    for (int64_t f = 0; f < p.F; f++) h[o_fs + f] = whole(f) ? -1 : slot++;
    for (size_t g = 0; g < go.size(); g++) h[o_gt + g] = fo[go[g]];
    for (size_t g = 0; g < wo.size(); g++) h[o_wt + g] = fo[wo[g]];
    rc = device_alloc(reinterpret_cast<void**>(&p.d_tables), at * sizeof(int32_t), st);
    if (rc != MASK_OK) return rc;
    p.d_frag_off = p.d_tables + o_fo;
    p.d_frag_win = p.d_tables + o_fw;
    p.d_frag_slot = p.d_tables + o_fs;
    p.d_group_off = p.d_tables + o_go;
    p.d_group_tile = p.d_tables + o_gt;
    p.d_warp_off = p.d_tables + o_wo;
    p.d_warp_tile = p.d_tables + o_wt;
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
    std::vector<int32_t> rbo, rb2w, go;
    strict_lb(h_val_soff, (M + kWinRows - 1) / kWinRows, workload, rbo, rb2w, go);
    *n_frag = (int64_t)rb2w.size();
    *n_groups = (int64_t)go.size() - 1;
    if (row_block_offset) std::memcpy(row_block_offset, rbo.data(), rbo.size() * sizeof(int32_t));
    if (row_block_to_window && !rb2w.empty()) std::memcpy(row_block_to_window, rb2w.data(), rb2w.size() * sizeof(int32_t));
    if (group_offset) std::memcpy(group_offset, go.data(), go.size() * sizeof(int32_t));
    return MASK_OK;
}

extern "C" int mask_plan_multi_bind(const int32_t* h_val_soff, int32_t M, int32_t* task_window, int32_t* window_split,
                                    int32_t* task_soff, int64_t* n_tasks) {
    using namespace mask;
    MASK_REQUIRE(h_val_soff != nullptr && M >= 1 && n_tasks, "bad arguments");
    std::vector<int32_t> tw, ws, ts;
    multi_bind(h_val_soff, (M + kWinRows - 1) / kWinRows, tw, ws, ts);
    *n_tasks = (int64_t)tw.size();
    if (task_window && !tw.empty()) std::memcpy(task_window, tw.data(), tw.size() * sizeof(int32_t));
    if (window_split && !ws.empty()) std::memcpy(window_split, ws.data(), ws.size() * sizeof(int32_t));
    if (task_soff) std::memcpy(task_soff, ts.data(), ts.size() * sizeof(int32_t));
    return MASK_OK;
}

namespace mask {

// With d_val_sidx the column features are measured and the plan table is applied as well: the kernels that
// measure run while the host builds the tables (both take 0.15 to 0.2 ms on a graph with 2^20 nodes).
static int create_plan(const int32_t* d_val_soff, const int32_t* d_val_sidx, int32_t M, int32_t K, int64_t T, int policy,
                       int32_t group_tiles, cudaStream_t st, mask_plan** out) {
    mask_plan* p = new mask_plan();
    p->M = M;
    p->W = (M + kWinRows - 1) / kWinRows;
    p->T = T;
    p->policy = policy;
    p->group_tiles = group_tiles > 0 ? group_tiles : (policy == MASK_POLICY_STRICT_LB ? 64 : default_group_tiles(T));
    p->auto_groups = group_tiles <= 0;
    // a piece may be longer than a group: it then is a group of its own
    p->piece_tiles = (group_tiles > 0 || policy != MASK_POLICY_AUTO) ? p->group_tiles : default_piece_tiles(T, p->W);
    HostStage stage;
    ColumnStatsJob job;
    cudaEvent_t have_soff = nullptr;
    auto body = [&]() -> int {
        MASK_CUDA_TRY(cudaGetDevice(&p->device));
        const size_t bytes = ((size_t)p->W + 1) * sizeof(int32_t);
        int rc = stage.get(bytes);
        if (rc != MASK_OK) return rc;
        const int32_t* soff = stage.as<int32_t>();
        MASK_CUDA_TRY(cudaMemcpyAsync(stage.as<int32_t>(), d_val_soff, bytes, cudaMemcpyDeviceToHost, st));
        if (d_val_sidx) {
            MASK_CUDA_TRY(cudaEventCreateWithFlags(&have_soff, cudaEventDisableTiming));
            MASK_CUDA_TRY(cudaEventRecord(have_soff, st));
            rc = job.enqueue(d_val_soff, d_val_sidx, M, K, T, 512, st);
            if (rc != MASK_OK) return rc;
            MASK_CUDA_TRY(cudaEventSynchronize(have_soff));
        } else {
            MASK_CUDA_TRY(cudaStreamSynchronize(st));
        }
        if (soff[0] != 0 || (int64_t)soff[p->W] != T) return fail(MASK_ERR_INVALID_ARGUMENT, "val_soff does not start at 0 / end at T");
        if (policy == MASK_POLICY_REF_AUTO) {  // the bridge's automatic choice between its own two mappings
            mask_features f;
            mask_features_from_soff(soff, M, 0, &f);
            p->policy = f.heavy_tail ? MASK_POLICY_STRICT_LB : MASK_POLICY_ROW;
            if (group_tiles <= 0) p->group_tiles = 64;
        }
        build_tables(*p, soff);
        if (d_val_sidx) {
            MASK_CUDA_TRY(cudaStreamSynchronize(st));
            mask_column_features f;
            job.finish(&f);
            choose_plan_parameters(p, f);
        }
        build_warp_groups(*p);
        return upload_tables(*p, soff, st);
    };
    const int rc = body();
    if (rc != MASK_OK) cudaStreamSynchronize(st);   // copies into the staging buffers may be in flight
    if (have_soff) cudaEventDestroy(have_soff);
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
    if (frag_offset) std::memcpy(frag_offset, p->h_frag_off.data(), p->h_frag_off.size() * sizeof(int32_t));
    if (frag_window && p->F) std::memcpy(frag_window, p->h_frag_win.data(), p->h_frag_win.size() * sizeof(int32_t));
    if (group_offset) std::memcpy(group_offset, p->h_group_off.data(), p->h_group_off.size() * sizeof(int32_t));
    return MASK_OK;
}
