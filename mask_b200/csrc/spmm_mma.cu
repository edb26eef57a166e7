// Warp-level TF32 SpMM kernels for SR-BCRS 16x8 and ME-TCF on sm_100a.
//
// One warp owns a 16 x CW slab of C (CW = 32*NQ columns) and walks a contiguous range of 16x8
// tiles that the plan assigned to its thread block.  For every tile it needs the 8 gathered rows
// of B restricted to its CW columns; those are loaded STRAIGHT INTO MMA FRAGMENT REGISTERS with
// 128-bit loads (each warp-wide load covers 4 rows x 128 contiguous bytes), double-buffered in
// registers two tiles ahead.  No shared-memory staging of B, no block-wide barrier: the kernel
// is a stream of coalesced loads feeding mma.sync.m16n8k8.tf32, which is what an HBM/L2-bound
// gather wants.  The four warps of a block take adjacent column slabs of the same tiles, so the
// tile values and column ids are fetched from L2 once per block and hit L1 for the other warps.
//
// Column permutation trick.  For a group of 32 columns starting at cb, lane (g = lane/4,
// k = lane%4) loads float4 B[row_k][cb+4g .. cb+4g+3] and B[row_{k+4}][same].  Component j of
// those vectors is the B fragment of MMA j, whose n index g therefore stands for column
// cb + 4g + j.  The accumulator fragment of MMA j holds n' = 2k, 2k+1, i.e. columns
// cb + 8k + j and cb + 8k + 4 + j, so over j = 0..3 a lane owns 8 consecutive columns of rows g
// and g+8 and stores them with 128-bit stores.
//
// Operand rounding.  The reference kernel rounds both operands with cvt.rna.tf32.f32
// (examples/src_fp32/sr_bcrs/testbed/kernel.inc:809-814).  The tensor core ignores the low 13
// mantissa bits of a TF32 operand, so adding 0x1000 to the FP32 bit pattern beforehand is
// exactly round-to-nearest, ties away from zero, for every finite value (values that round past
// FLT_MAX become infinity, as with cvt.rna; infinities are unchanged).  A NaN whose payload has
// all of bits 12..22 set would wrap; non-finite inputs are outside the contract of the format
// anyway, because a dense tile multiplies stored zeros by every gathered row.
//
// Windows split across blocks write their partial 16xN tiles to scratch; a second kernel sums
// them in fragment order, so no atomics and no zero-fill of C are needed.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "plan.h"
#include "spmm_common.cuh"

namespace mask {


// Development knobs (mask_tune): 0 = library default.
static int g_tune_nq = 0;
static int g_tune_min_blocks = 0;
static int g_tune_async = 1;   // 1 = warp-level kernel of spmm_warp.cu, 0 = register pipeline (below)
extern int g_session_chunk_cols;      // api.cu: column chunks of the host-buffer pipeline
static int g_tune_sweep = 1;   // 1 = persistent tcgen05 kernel except where the warp-level one measures faster, 2 = always, 0 = warp-level kernels only
static int g_tune_nslab = 0;   // persistent kernel: 128-column slabs per column block (0 = the plan's choice)
static int g_tune_tma = 0;     // 1 = the TMA-fed kernel where the plan holds rounded tile values (spmm_tma.cu); measured slower, off by default

template <int NQ, int FMT, int MIN_BLOCKS>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, MIN_BLOCKS) spmm_mma_kernel(const SpmmArgs p) {
    constexpr bool METCF = FMT == kFmtMetcf, MCO = FMT == kFmtMco;
    // ME-TCF / MCO: one private 16x8 tile per warp, rebuilt from the tile's COO run or bitmap
    // (MCO: a second 128-float area stages the tile's compact values).
    __shared__ __align__(16) float restore[FMT != kFmtSrbcrs ? kWarpsPerBlock * (MCO ? 2 : 1) : 1][kTileElems];

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int g = lane >> 2;
    const int k = lane & 3;
    const int col_base = (blockIdx.y * kWarpsPerBlock + warp) * (32 * NQ);
    if (col_base >= p.N) return;

    int f = p.group_off[blockIdx.x];
    const int f_end = p.group_off[blockIdx.x + 1];
    if (f >= f_end) return;
    int64_t t = p.frag_off[f];
    const int64_t t_end = p.frag_off[f_end];
    int64_t f_tend = p.frag_off[f + 1];

    // position of this lane's A fragment elements inside a stored tile
    int ao[4];
    if (FMT != kFmtSrbcrs) {
        ao[0] = sw123(8 * g + k);       ao[1] = sw123(8 * (g + 8) + k);
        ao[2] = sw123(8 * g + k + 4);   ao[3] = sw123(8 * (g + 8) + k + 4);
    } else {
        ao[0] = sw223(8 * g + k);       ao[1] = sw223(8 * (g + 8) + k);
        ao[2] = sw223(8 * g + k + 4);   ao[3] = sw223(8 * (g + 8) + k + 4);
    }

    bool qok[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) qok[q] = (col_base + 32 * q + 4 * g) < p.N;

    float acc[NQ][4][4];
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[q][j][i] = 0.f;

    // ---- register pipeline state -----------------------------------------------------------
    float4 breg[2][NQ][2];   // B fragments of the two tiles in flight
    float areg[2][4];        // SR-BCRS: A fragment values; ME-TCF: [0] = this lane's COO value
    int aidx[2];             // ME-TCF: this lane's COO index (or -1)
    int2 run[2];             // ME-TCF: [begin, end) of the tile's COO run
    int2 ix[2];              // gathered-row ids (k, k+4) of tiles t+2, t+3
    int2 nrun[2];            // ME-TCF: runs of tiles t+2, t+3
    ulonglong2 mk[2];        // MCO: mask words of the two tiles in flight
    float4 mv[2];            // MCO: this lane's chunk of the tile's compact values

    const float* Bcol = p.B + col_base + 4 * g;

    auto load_ix = [&](int slot, int64_t tt) {
        if (tt < t_end) {
            ix[slot].x = __ldg(p.val_sidx + tt * kTileCols + k);
            ix[slot].y = __ldg(p.val_sidx + tt * kTileCols + k + 4);
            if (METCF) {
                nrun[slot].x = __ldg(p.coo_off + 2 * tt);
                nrun[slot].y = __ldg(p.coo_off + 2 * tt + 1);
            }
            if (MCO) {
                nrun[slot].x = __ldg(p.coo_off + tt);
                nrun[slot].y = __ldg(p.coo_off + tt + 1);
            }
        }
    };
    auto load_tile = [&](int buf, int64_t tt, int2 id, int2 rn) {
        if (tt < t_end) {
            const float* r0 = Bcol + (int64_t)id.x * p.ldb;
            const float* r1 = Bcol + (int64_t)id.y * p.ldb;
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                if (qok[q]) {
                    breg[buf][q][0] = ldg_f4(r0 + 32 * q);
                    breg[buf][q][1] = ldg_f4(r1 + 32 * q);
                } else {
                    breg[buf][q][0] = make_float4(0.f, 0.f, 0.f, 0.f);
                    breg[buf][q][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            if (METCF) {
                run[buf] = rn;
                const int e = rn.x + lane;
                if (e < rn.y) {
                    aidx[buf] = __ldg(p.coo_idx + e);
                    areg[buf][0] = __ldg(p.coo_val + e);
                } else {
                    aidx[buf] = -1;
                }
            } else if (MCO) {
                run[buf] = rn;
                mk[buf] = __ldg(reinterpret_cast<const ulonglong2*>(p.mco_mask) + tt);
                if (rn.x + 4 * lane < rn.y) mv[buf] = ldg_f4(p.coo_val + rn.x + 4 * lane);   // runs are multiples of 4 values
            } else {
                const float* a = p.val_blk + tt * kTileElems;
#pragma unroll
                for (int i = 0; i < 4; i++) areg[buf][i] = __ldg(a + ao[i]);
            }
        }
    };

    auto flush = [&](int ff) {
        const int w = p.frag_win[ff];
        const int slot = p.frag_slot[ff];
        float* dst;
        int64_t ld;
        int rows_ok;
        if (slot < 0) {
            dst = p.C + (int64_t)w * kWinRows * p.ldc;
            ld = p.ldc;
            rows_ok = p.M - w * kWinRows;
        } else {
            dst = p.scratch + (int64_t)slot * kWinRows * p.N;
            ld = p.N;
            rows_ok = kWinRows;
        }
        const bool relu = p.relu && slot < 0;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int c0 = col_base + 32 * q + 8 * k;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = g + 8 * h;
                float4 v0 = make_float4(acc[q][0][2 * h], acc[q][1][2 * h], acc[q][2][2 * h], acc[q][3][2 * h]);
                float4 v1 = make_float4(acc[q][0][2 * h + 1], acc[q][1][2 * h + 1], acc[q][2][2 * h + 1],
                                        acc[q][3][2 * h + 1]);
                if (relu) {
                    v0.x = fmaxf(v0.x, 0.f); v0.y = fmaxf(v0.y, 0.f); v0.z = fmaxf(v0.z, 0.f); v0.w = fmaxf(v0.w, 0.f);
                    v1.x = fmaxf(v1.x, 0.f); v1.y = fmaxf(v1.y, 0.f); v1.z = fmaxf(v1.z, 0.f); v1.w = fmaxf(v1.w, 0.f);
                }
                if (r < rows_ok) {
                    float* row = (slot < 0 && p.row_map) ? p.C + (int64_t)p.row_map[w * kWinRows + r] * p.ldc
                                                         : dst + (int64_t)r * ld;
                    if (c0 < p.N) *reinterpret_cast<float4*>(row + c0) = v0;
                    if (c0 + 4 < p.N) *reinterpret_cast<float4*>(row + c0 + 4) = v1;
                    if (slot < 0) {  // the same row into every peer's copy of C
                        const int64_t off = row - p.C;
                        for (int j = 0; j < p.n_peer_out; j++) {
                            float* prow = p.peer_out[j] + p.peer_col + off;
                            if (c0 < p.N) *reinterpret_cast<float4*>(prow + c0) = v0;
                            if (c0 + 4 < p.N) *reinterpret_cast<float4*>(prow + c0 + 4) = v1;
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[q][j][i] = 0.f;
        }
    };

    auto consume = [&](int buf) {
        uint32_t a[4];
        if (METCF) {
            float* tile = restore[warp];
            __syncwarp();
            reinterpret_cast<float4*>(tile)[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
            if (aidx[buf] >= 0) tile[aidx[buf]] = areg[buf][0];
            // runs longer than one entry per lane (more than 32 stored entries in the tile)
            for (int e = run[buf].x + 32 + lane; e < run[buf].y; e += 32) tile[__ldg(p.coo_idx + e)] = __ldg(p.coo_val + e);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = rna_bits(tile[ao[i]]);
        } else if (MCO) {
            float* tile = restore[2 * warp];
            float* vals = restore[2 * warp + 1];
            __syncwarp();
            if (run[buf].x + 4 * lane < run[buf].y) reinterpret_cast<float4*>(vals)[lane] = mv[buf];
            __syncwarp();
            reinterpret_cast<uint4*>(tile)[lane] = mco_expand(mk[buf].x, mk[buf].y, reinterpret_cast<const uint32_t*>(vals), lane);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = __float_as_uint(tile[ao[i]]);   // already rounded by mco_expand
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = rna_bits(areg[buf][i]);
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const float4 v0 = breg[buf][q][0], v1 = breg[buf][q][1];
            mma_tf32(acc[q][0], a, rna_bits(v0.x), rna_bits(v1.x));
            mma_tf32(acc[q][1], a, rna_bits(v0.y), rna_bits(v1.y));
            mma_tf32(acc[q][2], a, rna_bits(v0.z), rna_bits(v1.z));
            mma_tf32(acc[q][3], a, rna_bits(v0.w), rna_bits(v1.w));
        }
    };

    // ---- prologue: ids of tiles t..t+3, fragments of tiles t, t+1 ---------------------------
    {
        int2 id0 = make_int2(0, 0), id1 = make_int2(0, 0), rn0 = make_int2(0, 0), rn1 = make_int2(0, 0);
        load_ix(0, t);
        load_ix(1, t + 1);
        id0 = ix[0]; id1 = ix[1]; rn0 = nrun[0]; rn1 = nrun[1];
        load_ix(0, t + 2);
        load_ix(1, t + 3);
        load_tile(0, t, id0, rn0);
        load_tile(1, t + 1, id1, rn1);
    }

    // ---- main loop, two tiles per trip so that buffer indices stay compile-time --------------
    while (true) {
#pragma unroll
        for (int s = 0; s < 2; s++) {
            while (t == f_tend && f < f_end) {  // fragment finished (also: fragments with no tile)
                flush(f);
                f++;
                f_tend = (f < f_end) ? p.frag_off[f + 1] : -1;
            }
            if (f >= f_end) return;
            consume(s);
            const int2 id = ix[s], rn = nrun[s];
            load_ix(s, t + 4);
            load_tile(s, t + 2, id, rn);
            t++;
        }
    }
}

// Sums the partial tiles of every split window in fragment (= tile) order and writes C.  heads: first
// fragment and number of pieces of each split window; the pieces' partial tiles lie one behind the other, so
// the reads of a thread are independent and eight of them are in flight at a time (walking the fragment
// tables piece by piece instead was a chain of dependent loads: 0.78 ms for 85 000 pieces at N = 512, now 0.57).
__global__ void __launch_bounds__(256) spmm_fixup_kernel(const int2* heads, const int32_t* frag_win, const int32_t* frag_slot,
                                                        const float* scratch, float* C, int64_t ldc, int32_t M,
                                                        int32_t N, int32_t n_out, int32_t vec_out, int32_t relu, const int32_t* row_map,
                                                        float* const* peer_out, int32_t n_peer_out, int32_t peer_col) {
    let_next_kernel_start();
    const int2 head = heads[blockIdx.x];
    const int w = frag_win[head.x];
    const int nvec = N >> 2;
    const int64_t tile_vecs = (int64_t)kWinRows * nvec;
    wait_for_previous_kernel();
    const float4* first = reinterpret_cast<const float4*>(scratch) + (int64_t)frag_slot[head.x] * tile_vecs;
    for (int v = blockIdx.y * blockDim.x + threadIdx.x; v < kWinRows * nvec; v += gridDim.y * blockDim.x) {
        const int r = v / nvec, c = (v - r * nvec) << 2;
        if (w * kWinRows + r >= M) continue;
        const float4* at = first + v;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        int i = 0;
        for (; i + 8 <= head.y; i += 8, at += 8 * tile_vecs) {
            float4 x[8];
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = at[j * tile_vecs];
#pragma unroll
            for (int j = 0; j < 8; j++) { s.x += x[j].x; s.y += x[j].y; s.z += x[j].z; s.w += x[j].w; }
        }
        for (; i < head.y; i++, at += tile_vecs) {
            const float4 x = *at;
            s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
        }
        if (relu) { s.x = fmaxf(s.x, 0.f); s.y = fmaxf(s.y, 0.f); s.z = fmaxf(s.z, 0.f); s.w = fmaxf(s.w, 0.f); }
        const int out_row = row_map ? row_map[w * kWinRows + r] : w * kWinRows + r;
        if (!vec_out) {
            const float x[4] = {s.x, s.y, s.z, s.w};
            for (int j = 0; j < 4 && c + j < n_out; j++) C[(int64_t)out_row * ldc + c + j] = x[j];
            continue;
        }
        *reinterpret_cast<float4*>(C + (int64_t)out_row * ldc + c) = s;
        for (int j = 0; j < n_peer_out; j++) *reinterpret_cast<float4*>(peer_out[j] + peer_col + (int64_t)out_row * ldc + c) = s;
    }
}

static int launch_fixup(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st) {
    if (plan->H > 0) {
        dim3 fgrid((unsigned)plan->H, (unsigned)((kWinRows * (a.N >> 2) + 255) / 256));
        return launch_overlapped(spmm_fixup_kernel, fgrid, 256, 0, st, plan->d_heads, plan->d_frag_win, plan->d_frag_slot, a.scratch, a.C,
                                 a.ldc, a.M, a.N, a.n_out, a.vec_out, a.relu, a.row_map, a.peer_out, a.n_peer_out, a.peer_col);
    }
    return MASK_OK;
}

// 128-column slabs per column block of the persistent kernel for an N-column product
static int sweep_slabs(const mask_plan* plan, int N) {
    int nslab = g_tune_nslab != 0 ? g_tune_nslab : plan->nslab;
    const int fills = N > 256 ? 4 : (N > 128 ? 2 : 1);
    if (nslab != 1 && nslab != 2 && nslab != 4) nslab = fills;
    return nslab < fills ? nslab : fills;
}

// Which kernel: one warp per block (spmm_warp.cu) or the persistent tcgen05 kernel (spmm_sweep.cu).  The tcgen05
// kernel takes up to 512 columns of a tile at once: tile values and ids are read once and every gathered byte goes
// through shared memory once to and once from, so it wins where full-width rows are gathered at the L2's or
// shared memory's rate.  The warp kernel takes at most 128 columns at a time, has no minimum width, spreads small
// matrices over up to 3256 blocks instead of 296, takes long windows first, and re-reads (and rebuilds) the tiles for every
// block of columns.
// It also rounds B where the tcgen05 kernel cuts it off: 2.1 to 3.0e-4 from the exact product (2-norm) against 4.2 to 4.7e-4.
// Measured in turn in bursts of 4 to 8 ms (us, tcgen05 / warp), which the power limit does not reach.  u uniform, g power-law, m
// 27-point stencil, then rows in thousands (T tiles in thousands, groups of the warp kernel per SM):
//   SR-BCRS               N = 64       96           128          192          256          384          448          512
//   u.7   (1.9, .3)       9/8          9/8          9/8          11/8         11/8         17/9         17/9         17/9
//   u6    (9, 2.5)        10/6         11/9         11/9         13/11        13/12        19/12        20/17        19/17
//   u4    (10, 1.7)       9/8          9/9          9/11         12/12        12/13        17/17        17/17        17/17
//   u20   (25, 8.4)       18/10        19/11        19/16        25/18        25/22        39/29        40/37        40/37
//   u8    (39, 3.4)       21/19        22/23        21/21        31/28        30/29        49/46        49/46        48/47
//   u25   (44, 11)        24/13        25/21        25/21        35/31        34/34        55/48        56/61        57/60
//   g60   (98, 25)        74/30        76/38        78/45        92/68        94/81        134/116      140/151      143/152
//   g130  (214, 35)       137/57       139/70       138/84       185/127      184/154      296/226      306/298      323/308
//   u100  (128, 32)       63/31        63/42        65/49        96/82        108/105      189/158      221/211      257/198
//   m43   (54, 18)        29/15        29/16        30/23        42/32        43/42        70/59        73/73        74/74
//   m91   (116, 39)       57/27        58/36        58/45        83/68        85/83        141/124      153/167      157/170
//   m1000 (1290, 422)     557/249      558/338      549/418      816/681      800/844      1325/1275    1393/1645    1477/1695
//   g300  (489, 55)       275/116      279/150      275/172      394/280      396/334      713/499      728/644      728/660
//   g524  (960, 83)       486/208      494/273      488/338      730/533      750/663      1344/993     1367/1281    1387/1319
//   g600  (633, 69)       387/159      394/206      393/259      560/400      590/495      1029/736     1051/934     1070/972
//   g700  (1312, 108)     649/271      658/372      655/460      942/738      987/920      1848/1384    1875/1771    1929/1839
//   g1049 (1973, 148)     967/403      986/568      980/713      1419/1134    1561/1428    2836/2145    2869/2731    2996/2846
//   g2097 (4035, 269)     1871/861     1901/1222    1901/1547    2839/2454    3371/3100    6081/4676    6138/5868    6590/6200
//   ME-TCF (MCO within a tenth where it is not named)
//   u.7   (1.9, .3)       10/15        10/15        10/15        12/16        12/16        18/17        18/17        17/17
//   m3.4  (3.5, 1.4)      7/8          7/8          7/8          8/9          8/9          10/12        10/12        10/12
//   m8    (9.6, 3.4)      11/9         11/11        11/10        15/15        15/14        20/21        21/22        21/20
//   u4    (10, 1.7)       10/16        10/16        10/18        12/19        12/19        17/25        18/25        17/24
//   g7    (11, 4.1)       17/16        17/18        17/17        19/20        19/20        24/29        25/30        25/29
//   g10   (14, 5.7)       21/16        21/18        21/18        24/26        24/27        33/29        34/37        34/37
//   u12   (15, 5.1)       16/11        16/16        16/14        21/19        21/22        30/24        31/32        31/31
//   u16   (16, 6.8)       16/11        16/14        16/14        21/21        22/19        29/29        30/34        31/33
//   m20   (24, 8.3)       18/15        18/14        18/18        26/28        27/29        37/37        40/49        42/48
//   u20   (25, 8.4)       20/14        20/14        20/21        27/28        28/29        40/36        43/47        43/46
//   g20   (29, 12)        31/19        31/24        31/27        35/32        36/37        53/48        57/63        60/62
//   u25   (44, 11)        27/19        27/28        27/33        37/41        38/44        58/61        61/80        62/76
//   u40   (61, 17)        37/27        36/26        35/33        50/44        52/55        81/77        84/101       88/98
//   m43   (54, 18)        33/25        33/25        33/32        52/43        56/53        79/73        83/94        86/94
//   u60   (77, 25)        46/30        46/34        44/36        63/55        65/66        106/94       116/125      128/127
//   u100  (128, 32)       70/43        69/50        69/55        99/89        108/107      190/166      215/229      247/228
//   u200  (255, 42)       133/75       138/100      138/112      208/175      250/217      420/323      492/422      580/427
//   g200  (352, 44)       228/118      232/135      231/163      317/246      325/294      510/428      531/579      544/561
//   g300  (489, 55)       310/148      318/184      316/202      435/334      447/386      794/572      809/780      819/755
//   m1000 (1290, 422)     621/369      629/441      620/510      1025/872     1168/1010    1469/1516    1563/2006    1668/2015
//   g1049 (1973, 148)     1092/528     1124/631     1124/756     1575/1224    1670/1487    3055/2223    3141/3018    3209/2948
// Over the 68 matrices, 3 encodings and 11 to 15 widths of that measurement the choice below takes 0.6 % longer than the better
// kernel would each time (geometric mean; SR-BCRS 0.2 %), at worst 36 % (ME-TCF of an 8^3 stencil, 9 us).  Small bitmap matrices have
// become faster in the warp kernel since (choose_warp_shape): over 512 uniform ones of 60 to 5000 windows and widths 3.5 % longer, at worst
// 75 % (700 windows of 5 tiles, N = 192, 10 us).
static bool use_warp_kernel(const mask_plan* plan, int fmt, int N, bool tf32x3, bool sidx_aligned) {
    if (tf32x3) return true;                    // compensated products: the warp kernel only
    if (!sidx_aligned || g_tune_sweep == 2) return false;
    if (g_tune_async == 0) return false;
    if (g_tune_sweep == 0) return true;
    if (g_tune_tma != 0 && fmt == kFmtSrbcrs && plan->d_vals_tf32 != nullptr) return false;
    const bool dense = fmt == kFmtSrbcrs;
    const int64_t slabs = (N + 127) / 128, T = plan->T, groups = plan->Gw, sms = sm_count();
    const int64_t block = 128 * sweep_slabs(plan, N), padded = (N + block - 1) / block * block;
    const bool pads = 4 * padded >= 5 * (int64_t)N;   // columns that the tcgen05 kernel's blocks would only pad: a quarter of N and more
    const bool wide = N > 256 && !pads;
    // A handful of long groups: one warp takes half a microsecond per tile and twice that for one that it
    // rebuilds, a tcgen05 block an eighth.  With enough columns the warp kernel has more blocks to deal them to, and with very few
    // groups (u.7) neither fills the GPU.
    if (groups < (dense ? 4 : 5) * sms && T > (dense ? 32 : 16) * groups) {
        if (dense) return N > 128 ? groups * slabs <= (N > 256 ? 4 : 2) * sms : (N <= 64 || groups <= sms);
        if (N > 256) return 2 * groups * slabs <= 3 * sms;
        return N <= 96 && groups > 2 * sms && T <= 24 * groups;
    }
    // fewer groups than SMs, all short (ME-TCF, 160 to 256 columns: 9 / 10 on a power-law graph of 500 nodes, 9 / 7 on an 8^3 stencil)
    if (fmt == kFmtMetcf ? 4 * groups <= sms && N > 256 : 4 * groups <= 3 * sms) return true;
    // Tiles that are rebuilt: between the size at which blocks of 64 columns with long steps are all resident (13 an SM) and the one
    // at which blocks of 128 columns fill the GPU (15 an SM) the warp kernel has neither (m20, u20, u25).
    if (N <= 128) return dense || N <= 96 || T <= 18 * groups || 2 * groups <= 13 * sms || groups >= 13 * sms;
    const double served = plan->col_features.hub_share[0];   // gathers of 512-column rows that half the L2 serves with the most gathered ones
    if (dense) {
        // Full-width rows pay where they are read from L2: neighbouring windows share them, or nearly all of B fits.  Not in small matrices.
        if (wide && (plan->local || served >= 0.9)) return T * slabs <= 160000;
        // Two slabs of the tcgen05 kernel remain what the plan table's test multiplies with: 8 to 12 times the L2, 5 to 12 % slower (g524, g700;
        // in a run of seconds 1.53 / 1.48 ms at 2^19 nodes).
        return !(wide && plan->two_slabs_kept);
    }
    if (wide) {   // the same for tiles that are rebuilt, four times as often as the tcgen05 kernel does
        if (!plan->has_col_features) return T > 250000;
        return !plan->local && (plan->nslab == 2 || served < 0.4 || (served < 0.75 && N > 448));
    }
    return groups >= (N > 256 ? 5 : (pads ? 9 : 18)) * sms;   // full rounds of blocks, of two column blocks each up to 256
}

static bool aligned(const void* p, unsigned bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

// The packed arrays as the asynchronous copies read them: 16 bytes at a time, pairs of offsets 8.  Ids are read one by one by both
// kernels; that off 16 bytes they go to the tcgen05 kernel, and compensated products refuse them, is from when the warp kernel
// copied them, and is kept as what the call answers.
static int check_packed_alignment(const SpmmArgs& a) {
    MASK_REQUIRE(aligned(a.val_blk, 16) && aligned(a.coo_idx, 16) && aligned(a.coo_val, 16) && aligned(a.mco_mask, 16),
                 "val_block_val, val_coo_idx, val_coo_val, val_mco_mask and val_mco_val must be 16-byte aligned");
    MASK_REQUIRE(a.mco_mask || aligned(a.coo_off, 8), "val_coo_off must be 8-byte aligned");
    MASK_REQUIRE(!a.tf32x3 || aligned(a.val_sidx, 16), "compensated products need 16-byte aligned val_sidx");
    return MASK_OK;
}

template <int FMT>
static int launch_spmm(const mask_plan* plan, SpmmArgs a, cudaStream_t st) {
    if (plan->G == 0) return MASK_OK;
    // the register-pipelined kernel writes C 16 bytes at a time: rows that are not whole vectors go to the tcgen05 kernel
    const bool registers = g_tune_sweep == 0 && g_tune_async == 0 && !a.tf32x3 && a.vec_out;
    if (!registers && plan->T > 0) {
        const int bad = check_packed_alignment(a);
        if (bad != MASK_OK) return bad;
    }
    a.frag_off = plan->d_frag_off;
    a.frag_win = plan->d_frag_win;
    a.frag_slot = plan->d_frag_slot;
    a.group_off = plan->d_group_off;
    a.row_map = plan->d_row_map;
    a.peer_out = plan->d_peer_out;
    a.n_peer_out = plan->n_peer_out;
    const int N = a.N;
    int rc;
    if (use_warp_kernel(plan, FMT, N, a.tf32x3, aligned(a.val_sidx, 16))) {
        rc = launch_spmm_warp<FMT>(plan, a, st, g_tune_nq);
        return rc != MASK_OK ? rc : launch_fixup(plan, a, st);
    }
    if (g_tune_sweep != 0 && g_tune_tma != 0 && FMT == kFmtSrbcrs && spmm_tma_applies(plan, a)) {
        rc = launch_spmm_tma(plan, a, a.K, st, g_tune_nslab != 0 ? g_tune_nslab : plan->nslab);
        return rc != MASK_OK ? rc : launch_fixup(plan, a, st);
    }
    if (g_tune_sweep != 0 || !a.vec_out) {
        rc = launch_spmm_sweep(plan, a, st, g_tune_nslab != 0 ? g_tune_nslab : plan->nslab);
        return rc != MASK_OK ? rc : launch_fixup(plan, a, st);
    }
    // columns per warp: wide slabs (fewer re-reads of the tile values per column) when N fills
    // four warps of them, else narrower slabs so that small N still spreads over a block
    int nq = N > 256 ? 4 : (N > 128 ? 2 : 1);
    if (g_tune_nq == 1 || g_tune_nq == 2 || g_tune_nq == 4) nq = g_tune_nq;
    const int cols_per_block = 32 * nq * kWarpsPerBlock;
    dim3 grid((unsigned)plan->G, (unsigned)((N + cols_per_block - 1) / cols_per_block));
    dim3 block(kWarpsPerBlock * 32);
    if (grid.y > 65535) return fail(MASK_ERR_INVALID_ARGUMENT, "N too large");
    switch (nq) {
        case 4:
            if (g_tune_min_blocks == 3) spmm_mma_kernel<4, FMT, 3><<<grid, block, 0, st>>>(a);
            else spmm_mma_kernel<4, FMT, 2><<<grid, block, 0, st>>>(a);
            break;
        case 2:
            if (g_tune_min_blocks == 4) spmm_mma_kernel<2, FMT, 4><<<grid, block, 0, st>>>(a);
            else spmm_mma_kernel<2, FMT, 3><<<grid, block, 0, st>>>(a);
            break;
        default: spmm_mma_kernel<1, FMT, 4><<<grid, block, 0, st>>>(a); break;
    }
    MASK_CUDA_TRY(cudaGetLastError());
    return launch_fixup(plan, a, st);
}

static int check_common(const mask_plan* plan, int32_t M, int32_t K, int32_t N, const float* B, int64_t ldb,
                        float* C, int64_t ldc, void* scratch, size_t scratch_bytes, int32_t scratch_columns) {
    MASK_REQUIRE(plan != nullptr, "plan is NULL");
    MASK_REQUIRE(M == plan->M, "M differs from the plan's");
    MASK_REQUIRE(M >= 1 && K >= 1 && N >= 0, "M, K must be positive and N non-negative");
    MASK_REQUIRE(N % 4 == 0, "N must be a multiple of 4");
    if (N == 0) return MASK_OK;
    MASK_REQUIRE(B != nullptr && C != nullptr, "B or C is NULL");
    MASK_REQUIRE(ldb >= N && ldc >= N && ldb % 4 == 0 && ldc % 4 == 0, "ldb/ldc must be >= N and multiples of 4");
    MASK_REQUIRE(ldb < ((int64_t)1 << 30), "ldb too large");
    MASK_REQUIRE((reinterpret_cast<uintptr_t>(B) & 15) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0,
                 "B and C must be 16-byte aligned");
    const size_t need = mask_plan_scratch_bytes(plan, scratch_columns);
    if (need > 0) {
        if (scratch == nullptr || scratch_bytes < need) return fail(MASK_ERR_SCRATCH_TOO_SMALL, "scratch too small for the plan's split windows");
        MASK_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15) == 0, "scratch must be 16-byte aligned");
    }
    return MASK_OK;
}

}  // namespace mask

extern "C" int mask_kernel_revision(void) { return 7; }

extern "C" int mask_spmm_kernel_name(const mask_plan* plan, int format, int32_t N, int epilogue, char* out, size_t capacity) {
    using namespace mask;
    MASK_REQUIRE(plan != nullptr && out != nullptr && capacity > 0, "NULL argument");
    MASK_REQUIRE(format >= kFmtSrbcrs && format <= kFmtMco && N > 0, "bad format or N");
    static const char* const fmt_name[] = {"srbcrs", "metcf", "mco"};
    const bool tf32x3 = format == kFmtSrbcrs && (epilogue & MASK_NUMERICS_TF32X3);
    if (use_warp_kernel(plan, format, N, tf32x3, true)) {
        snprintf(out, capacity, "spmm_warp_kernel<%s>", tf32x3 ? "tf32x3" : fmt_name[format]);
    } else if (g_tune_sweep != 0) {
        const bool tma = g_tune_tma != 0 && format == kFmtSrbcrs && plan->d_vals_tf32 != nullptr;
        snprintf(out, capacity, "%s<nslab=%d,%s>", tma ? "spmm_tma_kernel" : "spmm_sweep_kernel", sweep_slabs(plan, N), fmt_name[format]);
    } else {
        snprintf(out, capacity, "legacy routing (mask_tune sweep=0), %s", fmt_name[format]);
    }
    return MASK_OK;
}

extern "C" int mask_spmm_warp_shape(const mask_plan* plan, int format, int32_t N, int epilogue, int32_t* columns, int32_t* step_tiles) {
    using namespace mask;
    MASK_REQUIRE(plan != nullptr && columns != nullptr && step_tiles != nullptr, "NULL argument");
    MASK_REQUIRE(format >= kFmtSrbcrs && format <= kFmtMco && N > 0, "bad format or N");
    warp_shape(plan, format, N, format == kFmtSrbcrs && (epilogue & MASK_NUMERICS_TF32X3), g_tune_nq, columns, step_tiles);
    return MASK_OK;
}

extern "C" int mask_tune(const char* name, int value) {
    using namespace mask;
    MASK_REQUIRE(name != nullptr, "name is NULL");
    if (!strcmp(name, "nq")) g_tune_nq = value;
    else if (!strcmp(name, "min_blocks")) g_tune_min_blocks = value;
    else if (!strcmp(name, "async")) g_tune_async = value;
    else if (!strcmp(name, "stages")) {}   // the ring depth is fixed
    else if (!strcmp(name, "sweep")) g_tune_sweep = value;
    else if (!strcmp(name, "nslab")) g_tune_nslab = value;
    else if (!strcmp(name, "tma")) g_tune_tma = value;
    else if (!strcmp(name, "session_chunk")) g_session_chunk_cols = value;
    else return fail(MASK_ERR_INVALID_ARGUMENT, "unknown tuning knob");
    return MASK_OK;
}

namespace mask {

// Rows of n floats, any alignment -> rows of n4 floats (n4 = n rounded up to 4, at most 3 zeros at the end).  One
// warp per run of rows; writes are 16 bytes a lane.
__global__ void __launch_bounds__(256) pad_rows_kernel(const float* __restrict__ src, int64_t ld, int32_t rows, int32_t n, int32_t n4,
                                                       float4* __restrict__ dst) {
    let_next_kernel_start();
    wait_for_previous_kernel();
    const int vecs = n4 >> 2;
    const int64_t total = (int64_t)rows * vecs;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int64_t r = i / vecs;
        const int c = (int)(i - r * vecs) << 2;
        const float* at = src + r * ld + c;
        float4 v;
        v.x = __ldg(at);
        v.y = c + 1 < n ? __ldg(at + 1) : 0.f;
        v.z = c + 2 < n ? __ldg(at + 2) : 0.f;
        v.w = c + 3 < n ? __ldg(at + 3) : 0.f;
        dst[i] = v;
    }
}

static bool whole_vectors(const void* p, int64_t ld, int32_t n) {
    return n % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

static int fill_matrix_args(const mask_plan* plan, const mask_matrix* m, SpmmArgs& a) {
    const bool some = plan->T > 0;
    a.val_sidx = m->val_sidx;
    switch (m->format) {
        case kFmtSrbcrs:
            MASK_REQUIRE(!some || (m->val_sidx && m->values), "packed arrays are NULL");
            a.val_blk = static_cast<const float*>(m->values);
            return MASK_OK;
        case kFmtMetcf:
            MASK_REQUIRE(!some || (m->val_sidx && m->offsets && m->index && m->values), "packed arrays are NULL");
            a.coo_off = m->offsets;
            a.coo_idx = static_cast<const int32_t*>(m->index);
            a.coo_val = static_cast<const float*>(m->values);
            return MASK_OK;
        case kFmtMco:
            MASK_REQUIRE(!some || (m->val_sidx && m->offsets && m->index), "packed arrays are NULL");
            MASK_REQUIRE((reinterpret_cast<uintptr_t>(m->index) & 15) == 0 && (reinterpret_cast<uintptr_t>(m->values) & 15) == 0,
                         "val_mco_mask and val_mco_val must be 16-byte aligned");
            a.coo_off = m->offsets;
            a.coo_val = static_cast<const float*>(m->values);
            a.mco_mask = static_cast<const unsigned long long*>(m->index);
            return MASK_OK;
        default: return fail(MASK_ERR_INVALID_ARGUMENT, "unknown format");
    }
}

}  // namespace mask

namespace mask {

// One after the other, products of at most `most` columns.  Column blocks, and rows of partial tiles in the fix-up pass,
// are numbered in the y dimension of a grid (at most 65 535): that many columns are kPieceColumns.
static int launch_pieces(const mask_plan* plan, int format, const SpmmArgs& a, int32_t most, cudaStream_t st) {
    for (int32_t c0 = 0, width; c0 < a.N; c0 += width) {
        SpmmArgs piece = a;
        width = std::min(most, a.N - c0);
        piece.B += c0;
        piece.C += c0;
        piece.peer_col = c0;
        piece.N = width;
        piece.n_out = std::min(width, a.n_out - c0);
        const int rc = format == kFmtSrbcrs ? launch_spmm<kFmtSrbcrs>(plan, piece, st)
                                            : (format == kFmtMetcf ? launch_spmm<kFmtMetcf>(plan, piece, st) : launch_spmm<kFmtMco>(plan, piece, st));
        if (rc != MASK_OK) return rc;
    }
    return MASK_OK;
}

// mask_spmm with scratch for `scratch_columns` columns, in pieces of at most `most`
static int spmm_in_pieces(const mask_plan* plan, const mask_matrix* m, int32_t n, const float* d_B, int64_t ldb, float* d_C, int64_t ldc,
                          float* d_pad, void* d_scratch, size_t scratch_bytes, int epilogue, void* stream, int32_t most, int32_t scratch_columns) {
    MASK_REQUIRE(plan != nullptr && m != nullptr, "plan or matrix is NULL");
    MASK_REQUIRE(n >= 0 && n <= 0x7fffffff - 3, "bad column count");
    if (n == 0) return MASK_OK;
    MASK_REQUIRE(d_B != nullptr && d_C != nullptr && ldb >= n && ldc >= n, "B or C is NULL, or a leading dimension is too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t n4 = (n + 3) & ~3;
    const bool pad = !whole_vectors(d_B, ldb, n), vec_out = whole_vectors(d_C, ldc, n);
    MASK_REQUIRE(!pad || d_pad != nullptr, "B needs padding and the padding buffer is NULL");
    MASK_REQUIRE(vec_out || plan->n_peer_out == 0, "peer outputs need N % 4 == 0, ldc % 4 == 0 and 16-byte aligned C");
    const float* B = pad ? d_pad : d_B;
    const int64_t ld = pad ? n4 : ldb;
    int rc = check_common(plan, m->M, m->K, n4, B, ld, vec_out ? d_C : const_cast<float*>(B), vec_out ? ldc : n4, d_scratch, scratch_bytes,
                          std::min(n4, scratch_columns));
    if (rc != MASK_OK) return rc;
    SpmmArgs a{};
    rc = fill_matrix_args(plan, m, a);
    if (rc != MASK_OK) return rc;
    a.B = B; a.ldb = ld; a.C = d_C; a.ldc = ldc;
    a.scratch = static_cast<float*>(d_scratch);
    a.M = m->M; a.K = m->K; a.N = n4; a.n_out = n; a.vec_out = vec_out;
    a.relu = ((epilogue & 0xff) == MASK_EPILOGUE_RELU);
    a.tf32x3 = (epilogue & MASK_NUMERICS_TF32X3) ? 1 : 0;
    MASK_REQUIRE(!a.tf32x3 || m->format == kFmtSrbcrs, "compensated products are implemented for SR-BCRS only");
    if (pad && plan->T > 0) {
        const int64_t blocks = ((int64_t)m->K * (n4 / 4) + 1023) / 1024;
        rc = launch_overlapped(pad_rows_kernel, dim3((unsigned)std::min<int64_t>(blocks, 8 * sm_count())), 256, 0, st, d_B, ldb, m->K, n, n4,
                               reinterpret_cast<float4*>(d_pad));
        if (rc != MASK_OK) return rc;
    }
    return launch_pieces(plan, m->format, a, std::min(most, kPieceColumns), st);
}

}  // namespace mask

extern "C" int mask_spmm(const mask_plan* plan, const mask_matrix* m, int32_t n, const float* d_B, int64_t ldb, float* d_C, int64_t ldc,
                         float* d_pad, void* d_scratch, size_t scratch_bytes, int epilogue, void* stream) {
    return mask::spmm_in_pieces(plan, m, n, d_B, ldb, d_C, ldc, d_pad, d_scratch, scratch_bytes, epilogue, stream, mask::kPieceColumns, 0x7fffffff);
}

// The entry points that take a matrix array by array.
namespace mask {
int spmm_arrays(const mask_plan* plan, const mask_matrix& m, int32_t N, const float* d_B, int64_t ldb, float* d_C, int64_t ldc, void* d_scratch,
                size_t scratch_bytes, int epilogue, void* stream, int32_t most) {
    const int rc = check_common(plan, m.M, m.K, N, d_B, ldb, d_C, ldc, d_scratch, scratch_bytes, std::min(N, most));
    if (rc != MASK_OK || N == 0) return rc;
    return spmm_in_pieces(plan, &m, N, d_B, ldb, d_C, ldc, nullptr, d_scratch, scratch_bytes, epilogue, stream, most, most);
}
}  // namespace mask

extern "C" int mask_spmm_srbcrs(const mask_plan* plan, const int32_t* d_val_soff, const int32_t* d_val_sidx,
                                const float* d_val_block_val, int32_t M, int32_t K, int32_t N, const float* d_B,
                                int64_t ldb, float* d_C, int64_t ldc, void* d_scratch, size_t scratch_bytes,
                                int epilogue, void* stream) {
    (void)d_val_soff;
    const mask_matrix m{mask::kFmtSrbcrs, M, K, 0, d_val_sidx, nullptr, nullptr, d_val_block_val};
    return mask::spmm_arrays(plan, m, N, d_B, ldb, d_C, ldc, d_scratch, scratch_bytes, epilogue, stream, 0x7fffffff);
}

extern "C" int mask_spmm_metcf(const mask_plan* plan, const int32_t* d_val_soff, const int32_t* d_val_sidx,
                               const int32_t* d_val_coo_off, const int32_t* d_val_coo_idx, const float* d_val_coo_val,
                               int32_t M, int32_t K, int32_t N, const float* d_B, int64_t ldb, float* d_C, int64_t ldc,
                               void* d_scratch, size_t scratch_bytes, int epilogue, void* stream) {
    (void)d_val_soff;
    const mask_matrix m{mask::kFmtMetcf, M, K, 0, d_val_sidx, d_val_coo_off, d_val_coo_idx, d_val_coo_val};
    return mask::spmm_arrays(plan, m, N, d_B, ldb, d_C, ldc, d_scratch, scratch_bytes, epilogue, stream, 0x7fffffff);
}

extern "C" int mask_spmm_mco(const mask_plan* plan, const int32_t* d_val_soff, const int32_t* d_val_sidx,
                             const int32_t* d_val_mco_off, const uint64_t* d_val_mco_mask, const float* d_val_mco_val,
                             int32_t M, int32_t K, int32_t N, const float* d_B, int64_t ldb, float* d_C, int64_t ldc,
                             void* d_scratch, size_t scratch_bytes, int epilogue, void* stream) {
    (void)d_val_soff;
    const mask_matrix m{mask::kFmtMco, M, K, 0, d_val_sidx, d_val_mco_off, d_val_mco_mask, d_val_mco_val};
    return mask::spmm_arrays(plan, m, N, d_B, ldb, d_C, ldc, d_scratch, scratch_bytes, epilogue, stream, 0x7fffffff);
}
