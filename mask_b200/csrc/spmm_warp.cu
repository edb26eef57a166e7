// Warp-level SpMM: one warp per thread block, one group of tiles per block, 32*NQ columns; every encoding.
//
// What bounds it is the rate at which gathered rows of B reach an SM: a gather of random rows alone measures
// 19.5 TB/s over the GPU out of L2 and 7 TB/s out of DRAM, most of it with many warps and shallow rings.  So the
// block is a single warp: no barrier, no idle partner when N does not fill four warps' columns, and the hardware
// hands the next group to whichever SM has a free slot.  S = 3 ring slots of 4.5 KB leave room for 15 blocks per
// SM, which also hide each other's dependent chains.  (Four-warp blocks, in which two warps of a block idled at
// N = 64 and the blocks finished together, took 1.87 ms on a 2^21-node power-law graph at N = 64, now 1.28 ms; the
// tcgen05 kernel took 0.32 ms at N = 128 on a 300 000-node graph in ME-TCF, here 0.25 ms.  At full width the
// tcgen05 kernel reads the tiles once instead of four times and is the better one where L2 serves the gathers: see
// use_warp_kernel.)  27-point stencil, N = 128: 16.7 TB/s from L2, 85 % of the gather alone.  Power-law graph of 2^18 nodes,
// N = 512 (profiled): 12.8 TB/s, 60 % of the sectors from L2, no unit above 60 % -- L1 58, issue slots 55, L2 54, DRAM 49,
// tensor pipe 35: the latency of the gathers with 15 warps an SM, two steps each in flight.
//
// Each ring slot holds one step: KT tiles, for each the 8 gathered rows of B (32*NQ columns) and the tile
// operand or what it is rebuilt from.  Gathered-row ids (and the value runs of the compact encodings) go
// through a ring of their own, S - 1 steps further ahead, so that they have landed when the copies that
// need them as addresses are issued.  All synchronisation is cp.async.wait_group + __syncwarp.
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
    // per tile: the dense tile; ME-TCF 32 indices + 32 values of the run; MCO 16 B of mask + up to 128 values
    static constexpr int kATile = kDense ? 512 : (FMT == kFmtMco ? 528 : 256);
    static constexpr int kSlot = kBBytes + KT * kATile;
    // per tile in the id ring: 8 ids, then (compact encodings) the [begin, end) of its run
    static constexpr int kIdTile = kDense ? 32 : 48;
    static constexpr int kIdRing = FMT == kFmtMetcf ? 8 : 4;   // steps; ME-TCF still needs a step's run when it consumes it
    static constexpr int kIdStep = KT * kIdTile;
    static constexpr int kIds = S * kSlot;
    static constexpr int kTile = kIds + kIdRing * kIdStep;     // ME-TCF: the tile being rebuilt
    static constexpr int kBytes = kTile + (FMT == kFmtMetcf ? 512 : 0);
};

// COMP: three products per MMA (hi*hi and the two residual terms).
template <int NQ, int KT, int S, int MINB, int FMT, bool GUARD, bool COMP>
__global__ void __launch_bounds__(32, MINB) spmm_warp_kernel(const SpmmArgs p) {
    using L = WarpLayout<NQ, KT, S, FMT>;
    constexpr bool METCF = FMT == kFmtMetcf, MCO = FMT == kFmtMco;
    extern __shared__ __align__(128) unsigned char smem[];

    let_next_kernel_start();
    const int lane = threadIdx.x;
    const int g = lane >> 2, k = lane & 3;
    const int col_base = blockIdx.y * (32 * NQ);
    int f = p.group_off[blockIdx.x];
    const int f_end = p.group_off[blockIdx.x + 1];
    const int t0 = p.group_tile[blockIdx.x];
    const int n_tiles = p.group_tile[blockIdx.x + 1] - t0;   // indexed 0..n_tiles-1 below
    if (f >= f_end) return;
    int f_tend = p.frag_off[f + 1] - t0;
    int f_next = p.frag_off[min((int64_t)f + 2, p.n_frag)] - t0;   // end of the following fragment, loaded ahead

    wait_for_previous_kernel();

    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);

    // copy side: row lr (and lr + 4), chunk lc of every 32-column group
    const int lr = lane >> 3, lc = lane & 7;
    const uint32_t cp0 = (uint32_t)(lr * 128 + ((lc ^ (lr & 6)) << 4));
    const uint32_t cp1 = (uint32_t)((lr + 4) * 128 + ((lc ^ (lr & 6) ^ 4) << 4));
    bool qok[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) qok[q] = !GUARD || (col_base + 32 * q + 4 * lc) < p.N;
    const char* Bcol = reinterpret_cast<const char*>(p.B + col_base + 4 * lc);
    const uint32_t ldb_bytes = (uint32_t)(p.ldb * 4);
    // fragment side: chunk g of rows 2k and 2k + 1; tile columns 2k, 2k + 1 of rows g and g + 8
    const int frag_off = 2 * k * 128 + ((g ^ (2 * k)) << 4);
    const int i0 = 8 * g + 2 * k;
    const int ao0 = (L::kDense ? sw223(i0) : sw123(i0)) * 4, ao1 = (L::kDense ? sw223(i0 + 64) : sw123(i0 + 64)) * 4;

    float acc[NQ][4][4];
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[q][j][i] = 0.f;

    // ids (and runs) of step j -> id ring
    auto issue_ids = [&](int j) {
        const uint32_t dst = ring + L::kIds + (j & (L::kIdRing - 1)) * L::kIdStep;
        const int u = lane >> 1, tt = j * KT + u;
        if (lane < 2 * KT && tt < n_tiles)
            cpa16(dst + u * L::kIdTile + (lane & 1) * 16, p.val_sidx + ((int64_t)t0 + tt) * kTileCols + (lane & 1) * 4);
        if (METCF) {
            const int v = lane - 16, tv = j * KT + v;
            if (v >= 0 && v < KT && tv < n_tiles)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + v * L::kIdTile + 32), "l"(p.coo_off + 2 * ((int64_t)t0 + tv)) : "memory");
        } else if (MCO) {
            const int v = (lane - 16) >> 1, tv = j * KT + v;
            if (lane >= 16 && v < KT && tv < n_tiles)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + v * L::kIdTile + 32 + (lane & 1) * 4),
                             "l"(p.coo_off + (int64_t)t0 + tv + (lane & 1)) : "memory");
        }
    };
    // operands of step j -> slot (byte offset); the step's ids are visible
    auto issue_step = [&](int j, int slot) {
        const unsigned char* idp = smem + L::kIds + (j & (L::kIdRing - 1)) * L::kIdStep;
#pragma unroll
        for (int u = 0; u < KT; u++) {
            const int tt = j * KT + u;
            if (tt < n_tiles) {
                const int* id = reinterpret_cast<const int*>(idp + u * L::kIdTile);
                const uint32_t dst = ring + slot + u * NQ * 1024;
                const char* r0 = Bcol + (uint64_t)(uint32_t)id[lr] * ldb_bytes;
                const char* r1 = Bcol + (uint64_t)(uint32_t)id[lr + 4] * ldb_bytes;
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    if (qok[q]) {
                        cpa16(dst + cp0 + q * 1024, r0 + q * 128);
                        cpa16(dst + cp1 + q * 1024, r1 + q * 128);
                    }
                }
                const uint32_t at = ring + slot + L::kBBytes + u * L::kATile;
                if (L::kDense) {
                    cpa16(at + lane * 16, p.val_blk + ((int64_t)t0 + tt) * kTileElems + lane * 4);
                } else {
                    const int2 run = *reinterpret_cast<const int2*>(idp + u * L::kIdTile + 32);
                    if (METCF) {   // the first 32 entries (runs start on multiples of 8 entries and are padded to 8)
                        const int chunk = lane & 7;
                        if (lane < 16 && run.x + 4 * chunk < ((run.y + 7) & ~7)) {
                            const void* src = lane < 8 ? static_cast<const void*>(p.coo_idx + run.x + 4 * chunk)
                                                       : static_cast<const void*>(p.coo_val + run.x + 4 * chunk);
                            cpa16(at + lane * 16, src);
                        }
                    } else {       // mask, then the values (runs are multiples of 4 values)
                        if (lane == 0) cpa16(at, p.mco_mask + 2 * ((int64_t)t0 + tt));
                        if (run.x + 4 * lane < run.y) cpa16(at + 16 + lane * 16, p.coo_val + run.x + 4 * lane);
                    }
                }
            }
        }
    };

    // ---- prologue: ids of the first 2S - 2 steps, operands of the first S - 1 ------------------------
#pragma unroll
    for (int j = 0; j < 2 * S - 2; j++) issue_ids(j);
    cpa_commit();
    cpa_wait<0>();
    __syncwarp();
#pragma unroll
    for (int j = 0; j < S - 1; j++) {
        issue_step(j, j * L::kSlot);
        cpa_commit();
    }

    // ---- main loop: one trip per tile ------------------------------------------------------------------
    int step = 0, next_slot = (S - 1) * L::kSlot, slot = -L::kSlot;
    for (int t = 0;; t++) {
        while (t == f_tend && f < f_end) {  // fragment finished (also: fragments without tiles)
            flush_fragment<NQ>(p, f, col_base, g, k, acc);
            f++;
            f_tend = f < f_end ? f_next : -1;
            f_next = p.frag_off[min((int64_t)f + 2, p.n_frag)] - t0;
        }
        if (f >= f_end) break;
        const int u = t & (KT - 1);
        if (u == 0) {
            cpa_wait<S - 2>();       // this step has landed (this thread's copies) ...
            __syncwarp();            // ... and everybody's; also: all lanes are done with the slot refilled here
            issue_step(step + S - 1, next_slot);
            issue_ids(step + 2 * S - 2);
            cpa_commit();
            step++;
            slot += L::kSlot;
            if (slot == S * L::kSlot) slot = 0;
            next_slot = slot;        // the slot consumed now is the next one to be refilled
        }
        const unsigned char* bt = smem + slot + u * NQ * 1024 + frag_off;
        // ME-TCF: the gathered rows before the tile is rebuilt, as many as registers hold, so that their loads overlap
        // that chain (300 000-node power-law graph, N = 128: 275 us, now 252; all four groups of columns spill: 344).
        constexpr int kEarly = METCF ? (NQ <= 2 ? NQ : (NQ == 4 ? 2 : 0)) : 0;
        float4 early[kEarly > 0 ? kEarly : 1][2];
#pragma unroll
        for (int q = 0; q < kEarly; q++) {
            early[q][0] = *reinterpret_cast<const float4*>(bt + q * 1024);
            early[q][1] = *reinterpret_cast<const float4*>(bt + q * 1024 + 128);
        }
        const unsigned char* at = smem + slot + L::kBBytes + u * L::kATile;
        float af[4];   // (g, 2k), (g + 8, 2k), (g, 2k + 1), (g + 8, 2k + 1)
        if (MCO) {
            // values lie in ascending bit order: a value's place is the number of mask bits below its own.  Bits
            // 32i..32i+31 are rows 4i..4i+3.
            const uint4 m = *reinterpret_cast<const uint4*>(at);
            const float* vals = reinterpret_cast<const float*>(at + 16);
            const int sh = (ao0 >> 2) & 31;
            const uint32_t below = (1u << sh) - 1u;
            const bool up = g >= 4;   // row g is in the second word of its half
            const int n0 = __popc(m.x), n1 = n0 + __popc(m.y);
            const uint32_t w0 = up ? m.y : m.x, w1 = up ? m.w : m.z;
            const int c0 = (up ? n0 : 0) + __popc(w0 & below), c1 = n1 + (up ? __popc(m.z) : 0) + __popc(w1 & below);
            const uint32_t b0 = w0 >> sh, b1 = w1 >> sh;
            af[0] = (b0 & 1u) ? vals[c0] : 0.f;
            af[2] = (b0 & 2u) ? vals[c0 + (b0 & 1u)] : 0.f;
            af[1] = (b1 & 1u) ? vals[c1] : 0.f;
            af[3] = (b1 & 2u) ? vals[c1 + (b1 & 1u)] : 0.f;
        } else {
            if (METCF) {   // rebuild the 16x8 tile: zero, then tile[idx] = value over the run
                float* tile = reinterpret_cast<float*>(smem + L::kTile);
                const int2 run = *reinterpret_cast<const int2*>(smem + L::kIds + ((step - 1) & (L::kIdRing - 1)) * L::kIdStep + u * L::kIdTile + 32);
                const int rcnt = run.y - run.x;
                const int idx = reinterpret_cast<const int*>(at)[lane];   // behind the run: not used
                const float val = reinterpret_cast<const float*>(at + 128)[lane];
                if (KT > 1 && u > 0) __syncwarp();   // the previous tile's fragments have been read
                reinterpret_cast<float4*>(tile)[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                __syncwarp();
                if (lane < rcnt) tile[idx] = val;
                for (int e = run.x + 32 + lane; e < run.y; e += 32) tile[__ldg(p.coo_idx + e)] = __ldg(p.coo_val + e);
                __syncwarp();
                at = smem + L::kTile;
            }
            const float2 v0 = *reinterpret_cast<const float2*>(at + ao0), v1 = *reinterpret_cast<const float2*>(at + ao1);
            af[0] = v0.x; af[1] = v1.x; af[2] = v0.y; af[3] = v1.y;
        }
        if constexpr (COMP) {
            uint32_t a[4], al[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { a[i] = tf32_hi(af[i]); al[i] = tf32_lo(af[i], a[i]); }
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const float4 v0 = *reinterpret_cast<const float4*>(bt + q * 1024);
                const float4 v1 = *reinterpret_cast<const float4*>(bt + q * 1024 + 128);
                const float b0[4] = {v0.x, v0.y, v0.z, v0.w}, b1[4] = {v1.x, v1.y, v1.z, v1.w};
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
            }
        } else {
            const uint32_t a[4] = {rna_bits(af[0]), rna_bits(af[1]), rna_bits(af[2]), rna_bits(af[3])};
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const float4 v0 = q < kEarly ? early[q][0] : *reinterpret_cast<const float4*>(bt + q * 1024);
                const float4 v1 = q < kEarly ? early[q][1] : *reinterpret_cast<const float4*>(bt + q * 1024 + 128);
                mma_tf32(acc[q][0], a, rna_bits(v0.x), rna_bits(v1.x));
                mma_tf32(acc[q][1], a, rna_bits(v0.y), rna_bits(v1.y));
                mma_tf32(acc[q][2], a, rna_bits(v0.z), rna_bits(v1.z));
                mma_tf32(acc[q][3], a, rna_bits(v0.w), rna_bits(v1.w));
            }
        }
    }
    cpa_wait<0>();
}

// Tiles per step: one (two at 32 columns) where many blocks are resident, up to four times as many where few are.
static constexpr int warp_step_tiles(int nq, int depth) { return (nq == 1 ? 2 : 1) << depth; }
// Blocks per SM: as many as shared memory holds, except where the registers of the compensated products need
// more room (N = 256, 200 000-node power-law graph: 12 blocks of 165 registers 500 us, 14 blocks 508, 15 of 128 562).
static constexpr int warp_blocks_per_sm(int nq, int depth, bool comp) {
    constexpr int blocks[4][3] = {{22, 12, 6}, {24, 13, 7}, {18, 10, 5}, {15, 8, 4}};
    constexpr int comp_blocks[4] = {22, 16, 14, 12};
    return comp && depth == 0 ? comp_blocks[nq - 1] : blocks[nq - 1][depth];
}

// Columns per warp (32 nq) and tiles per step for `groups` groups of tiles.  With fewer blocks than an SM holds the
// gathers are bound by their latency: a block has two steps in flight, so the steps get longer, and the columns are
// dealt to more blocks, as long as all of them are resident at once (short groups: within a sixteenth; a second
// round of long ones doubles the time).  The longest step that fits comes first, then the fewest columns that pad no
// more than the widest block would.  us, one tile and all columns a step / as chosen here: uniform 16 384
// rows, N = 64 18.6 / 9.1, N = 128 20.6 / 13.6; 15^3 stencil, N = 64 7.2 / 5.2, N = 256 10.7 / 6.8; power-law graph
// of 20 000 nodes, N = 64 21.3 / 15.2.  With four times the resident blocks, long steps lose a quarter to a half.
static void choose_warp_shape(int64_t groups, int64_t T, int N, bool comp, int tuned_nq, int* nq_out, int* depth_out) {
    const int slabs = (N + 127) / 128, widest = (N + 32 * slabs - 1) / (32 * slabs);
    const bool tuned = tuned_nq >= 1 && tuned_nq <= 4;
    for (int depth = 2; depth >= 0; depth--) {
        for (int nq = tuned ? tuned_nq : 1; nq <= (tuned ? tuned_nq : widest); nq++) {
            const int blocks = (N + 32 * nq - 1) / (32 * nq);
            if (blocks * nq > slabs * widest && !tuned) continue;
            const int64_t resident = (int64_t)sm_count() * warp_blocks_per_sm(nq, depth, comp);
            if (groups * blocks <= resident + (T <= 24 * groups ? resident / 16 : 0)) {
                *nq_out = nq;
                *depth_out = depth;
                return;
            }
        }
    }
    *nq_out = tuned ? tuned_nq : widest;
    *depth_out = 0;
}

template <int NQ, int DEPTH, int FMT, bool GUARD, bool COMP>
static int launch_warp_variant(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st) {
    constexpr int KT = warp_step_tiles(NQ, DEPTH), S = 3;
    using L = WarpLayout<NQ, KT, S, FMT>;
    auto kern = spmm_warp_kernel<NQ, KT, S, warp_blocks_per_sm(NQ, DEPTH, COMP), FMT, GUARD, COMP>;
    static std::atomic<uint64_t> opted_in;
    const int rc = opt_in_shared_memory(reinterpret_cast<const void*>(kern), L::kBytes, opted_in);
    if (rc != MASK_OK) return rc;
    dim3 grid((unsigned)plan->Gw, (unsigned)((a.N + 32 * NQ - 1) / (32 * NQ)));
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
    a.group_off = plan->d_warp_off;
    a.group_tile = plan->d_warp_tile;
    a.n_frag = plan->F;
    int nq, depth;
    choose_warp_shape(plan->Gw, plan->T, a.N, a.tf32x3, tuned_nq, &nq, &depth);
    if constexpr (FMT == kFmtSrbcrs)
        if (a.tf32x3) return launch_warp_shape<FMT, true>(plan, a, st, nq, depth);
    return launch_warp_shape<FMT, false>(plan, a, st, nq, depth);
}
template int launch_spmm_warp<kFmtSrbcrs>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);
template int launch_spmm_warp<kFmtMetcf>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);
template int launch_spmm_warp<kFmtMco>(const mask_plan*, const SpmmArgs&, cudaStream_t, int);

}  // namespace mask
