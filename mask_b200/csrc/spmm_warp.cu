// Warp-level SpMM: one warp per thread block, one group of tiles per block, 32*NQ columns; every encoding.
//
// What bounds it is the rate at which gathered rows of B reach an SM: a gather of random rows alone measures
// 19.5 TB/s over the GPU out of L2 and 7 TB/s out of DRAM, most of it with many warps and shallow rings.  So the
// block is a single warp: no barrier, no idle partner when N does not fill four warps' columns, and the hardware
// hands the next group to whichever SM has a free slot.  S = 3 ring slots of 4.5 KB leave room for 15 blocks per
// SM, which also hide each other's dependent chains.  At full width the tcgen05 kernel reads the tiles once instead
// of four times: see use_warp_kernel.  27-point stencil of 60^3 nodes, N = 256 (profiled): 54 bytes per cycle and SM of the 69
// of the bare gather, shared memory 61 %, tensor pipe 38 %, issue slots 38 %.
//
// The rest is the chain of one warp: 15 warps an SM do not hide it all.  With every gather taken out the loop still took
// 78 % of its time when it spent 205 instructions on a tile and 128 columns; it now spends 128 (that stencil 195 -> 182 us, power-law
// graph of 2^20 nodes at N = 512 3.14 -> 2.76 ms, of 2^21 nodes at N = 64 1.29 -> 1.19): ids are loaded
// four tiles at a time into a register and handed out by shuffles instead of passing through a ring in shared memory, shared
// addresses are 32-bit sums of a lane's constant and the slot, fragments are an outer loop, and what the end of a
// fragment needs is loaded when it begins.
//
// Each ring slot holds one step: KT tiles, for each the 8 gathered rows of B (32*NQ columns) and the tile
// operand.  What a tile of the compact encodings is rebuilt from is copied one step earlier, and the tile is rebuilt between the
// products of the one before it (MCO, power-law graph of 2^20 nodes, N = 128: 880 -> 779 us; ME-TCF, uniform 10^5 rows: 58.8 -> 54.9).
// All synchronisation is cp.async.wait_group + __syncwarp.
//
// Copy mapping and fragment mapping.  The load/store unit handles a 128-bit access one quarter-warp
// (8 lanes) at a time and spends one pass per distinct 128-byte line, so the copy is issued with lane l ->
// (row l/8, chunk l%8): a quarter-warp reads one contiguous line.  The MMA sums over its 8 k indices in any
// order, so index k (and k + 4) stands for tile column 2k (and 2k + 1): a lane then finds the two values it
// needs of a tile row side by side (one 64-bit load) and reads rows 2k and 2k + 1 of the gathered block.
// Chunk c of row r is stored at position c ^ (r & 6) of its line: writes (one row, 8 chunks) and fragment
// reads (rows 0, 2, 4, 6 and two chunks each) touch every bank once.  (Dealing the lanes of a row by the lines
// it covers when rows do not start on 128-byte lines halves the passes, and cost more in instructions than it
// saved: N = 100 84 -> 110 us.)
#include "spmm_common.cuh"
#include "tile_index.h"

namespace mask {

__device__ __forceinline__ void cpa16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <int NQ, int KT, int S, int FMT>
struct WarpLayout {
    static constexpr bool kDense = FMT == kFmtSrbcrs;
    static constexpr int kBBytes = KT * NQ * 1024;   // gathered rows of one step
    // per tile: the dense tile; ME-TCF 32 indices + 32 values of the run, then [begin, end); MCO 16 B of mask + up to 128 values
    static constexpr int kATile = kDense ? 512 : (FMT == kFmtMco ? 528 : 272);
    static constexpr int kRunAt = 256;
    static constexpr int kAStep = KT * kATile;
    static constexpr int kARing = kDense || KT == 1 ? S : S + 1;
    static constexpr int kA = S * kBBytes;
    static constexpr int kTile = kA + kARing * kAStep;         // ME-TCF: the tile being rebuilt
    static constexpr int kBytes = kTile + (FMT == kFmtMetcf ? 512 : 0);
};

// Ids (and runs) are loaded a batch at a time, 32 ids in one coalesced load, and handed out by shuffles.
template <int KT>
struct WarpIds {
    static constexpr int kTiles = KT > 4 ? KT : 4;   // tiles in a batch
    static constexpr int kRegs = kTiles / 4;
};

// Shared memory by 32-bit address.  The loads name "memory" as the stores and copies do: they read what other lanes wrote, and
// without it nothing keeps the compiler from moving them across the __syncwarp() between the two.
__device__ __forceinline__ float4 lds128(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds64(uint32_t at) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float lds32(uint32_t at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void sts32(uint32_t at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t at, int x, int y) { asm volatile("st.shared.v2.s32 [%0], {%1,%2};" ::"r"(at), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ void sts128_zero(uint32_t at) { asm volatile("st.shared.v4.s32 [%0], {%1,%1,%1,%1};" ::"r"(at), "r"(0) : "memory"); }

// COMP: three products per MMA (hi*hi and the two residual terms).
template <int NQ, int KT, int S, int MINB, int FMT, bool GUARD, bool COMP>
__global__ void __launch_bounds__(32, MINB) spmm_warp_kernel(const SpmmArgs p) {
    using L = WarpLayout<NQ, KT, S, FMT>;
    using I = WarpIds<KT>;
    constexpr bool METCF = FMT == kFmtMetcf, MCO = FMT == kFmtMco, DENSE = L::kDense;
    constexpr int kAhead = DENSE ? 0 : 1;   // steps by which the copies of the tiles are ahead of those of the gathered rows
    extern __shared__ __align__(128) unsigned char smem[];

    let_next_kernel_start();
    const int lane = threadIdx.x;
    const int g = lane >> 2, k = lane & 3;
    const int col_base = blockIdx.y * (32 * NQ);
    int4 group;
    if (p.warp_group) {
        const int b = (int)blockIdx.x - p.n_warp_first;
        group = b < 0 ? p.warp_first[blockIdx.x] : p.warp_group[b];
    } else {
        const int f0 = p.group_off[blockIdx.x], f1 = p.group_off[blockIdx.x + 1], t = p.group_tile[blockIdx.x];
        group = make_int4(f0, f1, t, p.group_tile[blockIdx.x + 1] - t);
    }
    int f = group.x;
    const int f_end = group.y, t0 = group.z, n_tiles = group.w;   // tiles are indexed 0..n_tiles-1 below
    if (f >= f_end) return;
    int f_tend = p.frag_off[f + 1] - t0;
    // loaded ahead: the end of the following fragment, window and slot of the current one
    int f_next = p.frag_off[min((int64_t)f + 2, p.n_frag)] - t0;
    int win = p.frag_win[f], part = p.frag_slot[f];

    wait_for_previous_kernel();

    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);

    // copy side: row lr (and lr + 4), chunk lc of every 32-column group
    const int lr = lane >> 3, lc = lane & 7;
    const uint32_t cp0 = ring + (uint32_t)(lr * 128 + ((lc ^ (lr & 6)) << 4));
    const uint32_t cp1 = ring + (uint32_t)((lr + 4) * 128 + ((lc ^ (lr & 6) ^ 4) << 4));
    const uint32_t cpa = ring + L::kA + lane * 16 + (MCO ? 16 : 0);
    bool qok[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) qok[q] = !GUARD || (col_base + 32 * q + 4 * lc) < p.N;
    const char* Bcol = reinterpret_cast<const char*>(p.B + col_base + 4 * lc);
    // from a register in the blocks that are faster so (see warp_blocks_per_sm)
    const uint32_t ldb_bytes = NQ == 3 || (DENSE && NQ == 1) ? (uint32_t)(p.ldb * 4) : p.ldb_bytes;
    // what this lane copies of a tile: 16 bytes of a dense one, 4 indices or values of a ME-TCF run, 4 values of a MCO run
    const char* a_src = DENSE ? reinterpret_cast<const char*>(p.val_blk + (int64_t)t0 * kTileElems + lane * 4)
                              : (METCF && lane < 8 ? reinterpret_cast<const char*>(p.coo_idx) : reinterpret_cast<const char*>(p.coo_val)) + (METCF ? lc : lane) * 16;
    const unsigned long long* mask_src = MCO ? p.mco_mask + 2 * (int64_t)t0 : nullptr;
    // fragment side: chunk g of rows 2k and 2k + 1; tile columns 2k, 2k + 1 of rows g and g + 8
    const uint32_t fb = ring + 2 * k * 128 + ((g ^ (2 * k)) << 4);
    const int i0 = 8 * g + 2 * k;
    const int ao0 = DENSE ? sw223(i0) : sw123(i0), ao1 = DENSE ? sw223(i0 + 64) : sw123(i0 + 64);
    const uint32_t fa0 = ring + (METCF ? L::kTile : L::kA) + ao0 * 4, fa1 = ring + (METCF ? L::kTile : L::kA) + ao1 * 4;

    float acc[NQ][4][4];
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[q][j][i] = 0.f;

    // ---- copies ------------------------------------------------------------------------------------------
    static_assert(ids_before_tile(1) == kTileCols, "");
    const int32_t* idp = p.val_sidx + (int64_t)t0 * kTileCols + lane;
    auto load_ids = [&](int (&id)[I::kRegs], int tile) {
#pragma unroll
        for (int i = 0; i < I::kRegs; i++) {
            const bool in = NQ == 3 ? tile + 4 * i < n_tiles - (lane >> 3) : tile + 4 * i + (lane >> 3) < n_tiles;
            id[i] = in ? __ldg(idp + ids_before_tile(tile + 4 * i)) : 0;
        }
    };
    auto load_runs = [&](int2& run, int tile) {
        if (lane < I::kTiles && tile + lane < n_tiles)
            run = METCF ? __ldg(reinterpret_cast<const int2*>(p.coo_off) + t0 + tile + lane)
                        : make_int2(__ldg(p.coo_off + t0 + tile + lane), __ldg(p.coo_off + t0 + tile + lane + 1));
    };
    int id[I::kRegs], id_next[I::kRegs];
    int2 run, run_next;
    load_ids(id, 0);
    if (!DENSE) load_runs(run, 0);
    load_ids(id_next, I::kTiles);
    if (!DENSE) load_runs(run_next, I::kTiles);

    int b_tile = 0, a_tile = 0;   // first tiles whose rows, and whose own copies, have not been issued
    auto issue_rows = [&](uint32_t slot) {   // gathered rows of the next step
#pragma unroll
        for (int u = 0; u < KT; u++) {
            if (b_tile + u < n_tiles) {
                const int ids = id[u / 4], from = (KT < 4 ? (b_tile + u) & 3 : u & 3) * 8 + lr;
                const uint32_t row0 = (uint32_t)__shfl_sync(0xffffffffu, ids, from), row1 = (uint32_t)__shfl_sync(0xffffffffu, ids, from + 4);
                const char* r0 = Bcol + (uint64_t)row0 * ldb_bytes;
                const char* r1 = Bcol + (uint64_t)row1 * ldb_bytes;
                const uint32_t to = slot + u * NQ * 1024;
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    if (qok[q]) {
                        cpa16(cp0 + to + q * 1024, r0 + q * 128);
                        cpa16(cp1 + to + q * 1024, r1 + q * 128);
                    }
                }
            }
        }
        b_tile += KT;
        if (KT >= 4 || (b_tile & 3) == 0) {   // on to the next batch
#pragma unroll
            for (int i = 0; i < I::kRegs; i++) id[i] = id_next[i];
            load_ids(id_next, b_tile + I::kTiles);
        }
    };
    auto issue_tiles = [&](uint32_t slot) {   // the next step's tiles, or what they are rebuilt from
#pragma unroll
        for (int u = 0; u < KT; u++) {
            if (a_tile + u < n_tiles) {
                const uint32_t to = cpa + slot + u * L::kATile;
                if (DENSE) {
                    cpa16(to, a_src + u * (kTileElems * 4));
                } else {
                    const int src = KT < 4 ? (a_tile + u) & 3 : u;
                    const int b = __shfl_sync(0xffffffffu, run.x, src), e = __shfl_sync(0xffffffffu, run.y, src);
                    if (METCF) {   // the first 32 entries (runs start on multiples of 8 entries and are padded to 8)
                        if (lane < 16 && b + 4 * lc < ((e + 7) & ~7)) cpa16(to, a_src + (int64_t)b * 4);
                        if (lane == 16) sts64(to, b, e);   // 256 bytes from the tile's first copy
                    } else {       // mask, then the values (runs are multiples of 4 values)
                        if (lane == 0) cpa16(to - 16, mask_src + 2 * u);
                        if (b + 4 * lane < e) cpa16(to, a_src + (int64_t)b * 4);
                    }
                }
            }
        }
        a_tile += KT;
        if (DENSE) a_src += KT * kTileElems * 4;
        if (MCO) mask_src += 2 * KT;
        if (!DENSE && (KT >= 4 || (a_tile & 3) == 0)) {
            run = run_next;
            load_runs(run_next, a_tile + I::kTiles);
        }
    };

    // ---- operand of a tile: (g, 2k), (g + 8, 2k), (g, 2k + 1), (g + 8, 2k + 1) ------------------------------
    // Dense tiles are read where they are used.  The others are rebuilt while the tile before them is multiplied, in
    // three stages between the products, so that none of their chains of dependent accesses is waited for.
    float af[4];
    int2 rb_run;
    float rb_idx, rb_val;
    auto rebuild0 = [&](uint32_t at, int tile) {   // at: the tile's place in shared memory; behind the last tile: empty
        if (METCF) {
            const float2 r = lds64(ring + at + L::kRunAt);
            rb_run = tile < n_tiles ? make_int2(__float_as_int(r.x), __float_as_int(r.y)) : make_int2(0, 0);
            rb_idx = lds32(ring + at + lane * 4);   // behind the run: not used
            rb_val = lds32(ring + at + 128 + lane * 4);
            sts128_zero(ring + L::kTile + lane * 16);
        }
    };
    auto rebuild1 = [&]() {
        if (METCF) {
            __syncwarp();
            if (lane < rb_run.y - rb_run.x) sts32(ring + L::kTile + __float_as_int(rb_idx) * 4, rb_val);
            for (int e = rb_run.x + 32 + lane; e < rb_run.y; e += 32) sts32(ring + L::kTile + __ldg(p.coo_idx + e) * 4, __ldg(p.coo_val + e));
        }
    };
    auto rebuild2 = [&](uint32_t at) {
        if (MCO) {
            // values lie in ascending bit order: a value's place is the number of mask bits below its own.  Bits
            // 32i..32i+31 are rows 4i..4i+3.
            const float4 w = lds128(ring + at);
            const uint32_t mx = __float_as_uint(w.x), my = __float_as_uint(w.y), mz = __float_as_uint(w.z), mw = __float_as_uint(w.w);
            const int sh = ao0 & 31;
            const uint32_t below = (1u << sh) - 1u;
            const bool up = g >= 4;   // row g is in the second word of its half
            const int n0 = __popc(mx), n1 = n0 + __popc(my);
            const uint32_t w0 = up ? my : mx, w1 = up ? mw : mz;
            const uint32_t c0 = ring + at + 16 + 4 * ((up ? n0 : 0) + __popc(w0 & below)), c1 = ring + at + 16 + 4 * (n1 + (up ? __popc(mz) : 0) + __popc(w1 & below));
            const uint32_t b0 = w0 >> sh, b1 = w1 >> sh;
            af[0] = af[1] = af[2] = af[3] = 0.f;
            if (b0 & 1u) af[0] = lds32(c0);
            if (b0 & 2u) af[2] = lds32(c0 + (b0 & 1u) * 4);
            if (b1 & 1u) af[1] = lds32(c1);
            if (b1 & 2u) af[3] = lds32(c1 + (b1 & 1u) * 4);
        } else {
            if (METCF) __syncwarp();
            const float2 v0 = lds64(fa0 + (METCF ? 0 : at)), v1 = lds64(fa1 + (METCF ? 0 : at));
            af[0] = v0.x; af[1] = v1.x; af[2] = v0.y; af[3] = v1.y;
        }
    };

    // ---- prologue: operands of the first S - 1 steps ---------------------------------------------------
    if (kAhead) issue_tiles(0);
#pragma unroll
    for (int j = 0; j < S - 1; j++) {
        issue_rows(j * L::kBBytes);
        issue_tiles((j + kAhead) * L::kAStep);
        cpa_commit();
    }
    uint32_t b_slot = (S - 1) * L::kBBytes;                  // of the step before the current one: refilled next
    uint32_t a_fill = (S - 1 + kAhead) % L::kARing * L::kAStep;  // the slot of tiles that is filled next
    uint32_t a_slot = 0;                                     // the tile whose operand is read next
    auto next_tile = [&]() { a_slot = a_slot == L::kARing * L::kAStep - L::kATile ? 0u : a_slot + L::kATile; };
    if (!DENSE) {
        cpa_wait<S - 2>();
        __syncwarp();
        rebuild0(L::kA + a_slot, 0);
        rebuild1();
        rebuild2(L::kA + a_slot);
        next_tile();
    }

    // ---- main loop, fragment by fragment -----------------------------------------------------------------
    int t = 0;
    for (;;) {
        for (; t < f_tend; t++) {
            const int u = t & (KT - 1);
            if (u == 0) {
                cpa_wait<S - 2>();       // this step has landed (this thread's copies) ...
                __syncwarp();            // ... and everybody's; also: all lanes are done with the slot refilled here
                issue_rows(b_slot);
                issue_tiles(a_fill);
                cpa_commit();
                a_fill = a_fill == (L::kARing - 1) * L::kAStep ? 0u : a_fill + L::kAStep;
                b_slot = b_slot == (S - 1) * L::kBBytes ? 0u : b_slot + L::kBBytes;
            } else if (METCF) {
                __syncwarp();            // all lanes have read the rebuilt tile
            }
            const uint32_t bt = fb + b_slot + u * NQ * 1024;
            if (DENSE) {
                rebuild2(a_slot);
                next_tile();
            }
            uint32_t a[4], al[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                a[i] = COMP ? tf32_hi(af[i]) : rna_bits(af[i]);
                if (COMP) al[i] = tf32_lo(af[i], a[i]);
            }
            // Loads do not pass the rebuilding's stores: for ME-TCF two groups of columns are read before them, the others
            // between its stages (each where it is used: uniform 10^5 rows, N = 128, 56.7 us, so 54.9).
            float4 v[NQ][2];
            auto read_rows = [&](int q) { v[q][0] = lds128(bt + q * 1024); v[q][1] = lds128(bt + q * 1024 + 128); };
            if (METCF) {
#pragma unroll
                for (int q = 0; q < 2 && q < NQ; q++) read_rows(q);
            }
            if (!DENSE) rebuild0(L::kA + a_slot, t + 1);
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                if (!METCF) read_rows(q);
                const float b0[4] = {v[q][0].x, v[q][0].y, v[q][0].z, v[q][0].w}, b1[4] = {v[q][1].x, v[q][1].y, v[q][1].z, v[q][1].w};
                if constexpr (COMP) {
                    uint32_t h0[4], h1[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) { h0[j] = tf32_hi(b0[j]); h1[j] = tf32_hi(b1[j]); }
                    // small terms first; four accumulators in turn, so that no product waits for the one before it
#pragma unroll
                    for (int j = 0; j < 4; j++) mma_tf32(acc[q][j], al, h0[j], h1[j]);
#pragma unroll
                    for (int j = 0; j < 4; j++) mma_tf32(acc[q][j], a, tf32_lo(b0[j], h0[j]), tf32_lo(b1[j], h1[j]));
#pragma unroll
                    for (int j = 0; j < 4; j++) mma_tf32(acc[q][j], a, h0[j], h1[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) mma_tf32(acc[q][j], a, rna_bits(b0[j]), rna_bits(b1[j]));
                }
                if (!DENSE && q == 0) {
                    rebuild1();
                    if (METCF) {
#pragma unroll
                        for (int r = 2; r < NQ; r++) read_rows(r);
                    }
                }
                if (!DENSE && q == (NQ > 1 ? 1 : 0)) {
                    rebuild2(L::kA + a_slot);
                    next_tile();
                }
            }
        }
        write_fragment<NQ, GUARD>(p, win, part, col_base, g, k, acc);
        if (++f >= f_end) break;
        f_tend = f_next;
        f_next = p.frag_off[min((int64_t)f + 2, p.n_frag)] - t0;
        win = p.frag_win[f];
        part = p.frag_slot[f];
    }
    cpa_wait<0>();
}

// Tiles per step: one (two at 32 columns) where many blocks are resident, up to four times as many where few are.
static constexpr int warp_step_tiles(int nq, int depth) { return (nq == 1 ? 2 : 1) << depth; }
// Blocks per SM: as many as shared memory holds, except where the registers of the compensated products need
// more room (N = 256, 200 000-node power-law graph: 12 blocks of 165 registers 500 us, 14 blocks 508, 15 of 128 562).
// The registers of 24 blocks of 64 columns (80) and of 18 blocks of 96 (96) are all in use, so that how an address is written decides what is
// spilled: a row's length of B from the launch arguments instead of a register takes 64 and 128 columns 1 to 8 % less time, SR-BCRS
// blocks of 32 columns 5 % more, blocks of 96 1 % more; the first form of the ids' bound costs blocks of 96 columns 1 to 2 %.
// Bitmaps take a tile's room more (WarpLayout), which costs some shapes a block.
static constexpr int warp_blocks_per_sm(int fmt, int nq, int depth, bool comp) {
    constexpr int blocks[4][3] = {{22, 12, 6}, {24, 13, 7}, {18, 10, 5}, {15, 8, 4}};
    constexpr int mco_blocks[4][3] = {{20, 10, 5}, {24, 13, 6}, {18, 9, 5}, {15, 7, 3}};
    constexpr int comp_blocks[4] = {22, 16, 14, 12};
    if (comp && depth == 0) return comp_blocks[nq - 1];
    return (fmt == kFmtMco ? mco_blocks : blocks)[nq - 1][depth];
}

// Columns per warp (32 nq) and tiles per step for `groups` groups of tiles.  With fewer blocks than an SM holds the
// gathers are bound by their latency: a block has two steps in flight, so the steps get longer, and the columns are
// dealt to more blocks, as long as all of them are resident at once (short groups: within a sixteenth; a second
// round of long ones doubles the time).  The longest step that fits comes first, then the fewest columns that pad no
// more than the widest block would.  us, one tile and all columns a step / as chosen here: uniform 16 384
// rows, N = 64 18.6 / 9.1, N = 128 20.6 / 13.6; 15^3 stencil, N = 64 7.2 / 5.2, N = 256 10.7 / 6.8; power-law graph
// of 20 000 nodes, N = 64 21.3 / 15.2.  Bitmaps by the blocks of the other encodings, more than are resident, / by their own: groups of 20
// tiles, 870 of them at N = 32 12.0 / 7.9, 1600 12.4 / 11.9, 450 at N = 64 12.0 / 7.6, 1030 13.0 / 11.5, 590 at N = 128 15.3 / 11.6.  But at 128
// columns and two tiles a step an eighth block begun late costs less than 64 columns and one tile: 1180 groups of 20 tiles 16.8 / 19.4, of 45
// 31.4 / 40.1, of 8 9.3 / 9.4.  So does a tenth of 96 columns for more than 9 1/2 an SM of more than 16 tiles: 1440 groups of 20 17.1 / 18.0, of 45
// 32.7 / 37.7, but of 16 14.8 / 14.1, and 1400 of 45 32.0 / 25.8.  With four times the resident blocks, long steps lose a quarter to a half, but for blocks of
// 64 columns: 13 of them with two tiles a step finish a long window sooner than 24 with one, and that is what a power-law graph waits
// for.  us, one tile a step / two, by thousands of tiles (power-law, then uniform matrices):
//   N = 64     160 T       214        446        489        1003       1973        4890           128       505        1277
//   SR-BCRS    49 / 44     58 / 56    104 / 104  115 / 114  218 / 224  404 / 429   1014 / 1055    33 / 31   100 / 111  429 / 427
//   ME-TCF     71 / 55     89 / 69    147 / 130  161 / 142  294 / 273  522 / 513   1239 / 1208    43 / 39   131 / 128  362 / 356
//   MCO        71 / 54     90 / 67    144 / 125  156 / 137  286 / 266  514 / 498   1226 / 1187    40 / 37   132 / 125  357 / 378
//   N = 48
//   SR-BCRS    54 / 45     63 / 56    107 / 104  116 / 113  214 / 222  384 / 420   961 / 1023     32 / 31   95 / 104   393 / 392
//   ME-TCF     78 / 58     97 / 73    158 / 136  172 / 146  313 / 280  558 / 525   1338 / 1250    46 / 41   144 / 135  358 / 349
//   MCO        79 / 55     99 / 68    157 / 126  170 / 138  313 / 266  562 / 496   1345 / 1187    44 / 38   146 / 126  357 / 362
// So SR-BCRS takes two up to 400 000 tiles, tiles that are rebuilt always, but for bitmaps of large matrices without hubs.  Not with a
// stencil's short windows (60^3, N = 64, SR-BCRS: 59 / 62).
static void choose_warp_shape(const mask_plan* plan, int fmt, int N, bool comp, int tuned_nq, int* nq_out, int* depth_out) {
    const int64_t groups = plan->Gw, T = plan->T, sms = sm_count();
    const int slabs = (N + 127) / 128, widest = (N + 32 * slabs - 1) / (32 * slabs);
    const bool tuned = tuned_nq >= 1 && tuned_nq <= 4;
    for (int depth = 2; depth >= 0; depth--) {
        for (int nq = tuned ? tuned_nq : 1; nq <= (tuned ? tuned_nq : widest); nq++) {
            const int blocks = (N + 32 * nq - 1) / (32 * nq);
            if (blocks * nq > slabs * widest && !tuned) continue;
            int per_sm = warp_blocks_per_sm(fmt, nq, depth, comp);
            if (fmt == kFmtMco && depth == 1 && (nq == 4 || (nq == 3 && T > 16 * groups && 2 * groups * blocks > 19 * sms))) per_sm++;
            const int64_t resident = sms * per_sm;
            if (groups * blocks <= resident + (T <= 24 * groups ? resident / 16 : 0)) {
                *nq_out = nq;
                *depth_out = depth;
                return;
            }
        }
    }
    *nq_out = tuned ? tuned_nq : widest;
    const bool hubs = plan->col_features.hub_share[0] >= 0.25;
    const bool two = fmt == kFmtSrbcrs ? T <= 400000 : (fmt == kFmtMetcf || hubs || T <= 1000000);
    *depth_out = *nq_out == 2 && !comp && !plan->local && two ? 1 : 0;
}

void warp_shape(const mask_plan* plan, int fmt, int N, bool comp, int tuned_nq, int* columns, int* step_tiles) {
    int nq, depth;
    choose_warp_shape(plan, fmt, N, comp, tuned_nq, &nq, &depth);
    *columns = 32 * nq;
    *step_tiles = warp_step_tiles(nq, depth);
}

template <int NQ, int DEPTH, int FMT, bool GUARD, bool COMP>
static int launch_warp_variant(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st) {
    constexpr int KT = warp_step_tiles(NQ, DEPTH), S = 3;
    using L = WarpLayout<NQ, KT, S, FMT>;
    constexpr int kBlocks = warp_blocks_per_sm(FMT, NQ, DEPTH, COMP);
    // an SM has 228 KB, in units of 128 bytes, and keeps 1 KB a block for itself
    static_assert(kBlocks * ((L::kBytes + 127) / 128 * 128 + 1024) <= 228 * 1024, "more blocks than an SM's shared memory holds");
    auto kern = spmm_warp_kernel<NQ, KT, S, kBlocks, FMT, GUARD, COMP>;
    static std::atomic<uint64_t> opted_in;
    const int rc = opt_in_shared_memory(reinterpret_cast<const void*>(kern), L::kBytes, opted_in);
    if (rc != MASK_OK) return rc;
    dim3 grid((unsigned)(plan->Gw + a.n_warp_first), (unsigned)((a.N + 32 * NQ - 1) / (32 * NQ)));
    if (grid.y > 65535) return fail(MASK_ERR_INVALID_ARGUMENT, "N too large");
    return launch_overlapped(kern, grid, 32, L::kBytes, st, a);
}

template <int FMT, bool COMP>
static int launch_warp_shape(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st, int nq, int depth) {
    const bool guard = a.N % (32 * nq) != 0;
#define MASK_CASE(NQ, DEPTH)                                                               \
    case NQ * 3 + DEPTH:                                                                   \
        return guard ? launch_warp_variant<NQ, DEPTH, FMT, true, COMP>(plan, a, st)        \
                     : launch_warp_variant<NQ, DEPTH, FMT, false, COMP>(plan, a, st);
#define MASK_CASES(NQ) MASK_CASE(NQ, 0) MASK_CASE(NQ, 1) MASK_CASE(NQ, 2)
    switch (nq * 3 + depth) { MASK_CASES(1) MASK_CASES(2) MASK_CASES(3) MASK_CASES(4) }
#undef MASK_CASES
#undef MASK_CASE
    return fail(MASK_ERR_INVALID_ARGUMENT, "no such kernel");
}

template <int FMT>
int launch_spmm_warp(const mask_plan* plan, const SpmmArgs& a_in, cudaStream_t st, int tuned_nq) {
    SpmmArgs a = a_in;
    a.group_tile = plan->d_group_tile;
    a.warp_group = plan->d_warp_group;
    a.warp_first = plan->d_warp_first;
    a.n_warp_first = plan->warp_first;
    a.n_frag = plan->F;
    a.ldb_bytes = (uint32_t)(a.ldb * 4);
    int nq, depth;
    choose_warp_shape(plan, FMT, a.N, a.tf32x3, tuned_nq, &nq, &depth);
    if constexpr (FMT == kFmtSrbcrs)
        if (a.tf32x3) return launch_warp_shape<FMT, true>(plan, a, st, nq, depth);
    return launch_warp_shape<FMT, false>(plan, a, st, nq, depth);
}
template int launch_spmm_warp<kFmtSrbcrs>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);
template int launch_spmm_warp<kFmtMetcf>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);
template int launch_spmm_warp<kFmtMco>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);

}  // namespace mask
