// Pieces shared by the SpMM kernels: launch arguments, the TF32 MMA wrapper and operand rounding.
#pragma once

#include "common.cuh"
#include "launch.cuh"
#include "plan.h"

namespace mask {

struct SpmmArgs {
    const int32_t* frag_off;
    const int32_t* frag_win;
    const int32_t* frag_slot;
    const int32_t* group_off;
    const int32_t* group_tile;  // first tile of every group (+ closing entry): persistent kernel only
    const int4* warp_group;     // warp-level kernel: the plan's d_warp_group and d_warp_first
    const int4* warp_first;
    int32_t n_warp_first;
    int64_t n_frag;             // fragments in the plan (frag_off has n_frag + 1 entries)
    int32_t n_groups;
    int32_t n_col_blocks;       // persistent kernel: column blocks of 128*NSLAB columns
    const int32_t* val_sidx;
    const float* val_blk;      // SR-BCRS
    const int32_t* coo_off;    // ME-TCF: [begin, end) pairs per tile (+ closing entry); MCO: val_mco_off[T+1]
    const int32_t* coo_idx;    // ME-TCF
    const float* coo_val;      // ME-TCF and MCO: the stored values
    const unsigned long long* mco_mask;   // MCO: two 64-bit words per tile, bit Swizzle<1,2,3>(8r+c)
    float* const* peer_out;    // optional: n_peer_out more output bases (peer GPUs' copies of C, same layout)
    int32_t n_peer_out;
    int32_t peer_col;          // column of the peers' copies that column 0 of this launch's C is
    const int32_t* row_map;    // optional: packed row i is output row row_map[i] (row reorder undone on the fly)
    const float* B;
    int64_t ldb;
    float* C;
    int64_t ldc;
    float* scratch;
    int32_t M;
    int32_t K;
    int32_t N;               // columns that are multiplied (a multiple of 4); B and the scratch tiles have them all
    int32_t n_out;           // columns of C that are written: N, or up to 3 fewer
    int32_t vec_out;         // rows of C can be written 16 bytes at a time
    int32_t relu;
    int32_t tf32x3;  // compensated products (MASK_NUMERICS_TF32X3)
    uint32_t ldb_bytes;      // 4 ldb, warp-level kernel only; fills the padding (8 more bytes of arguments: 0.3 us more of the host's time a launch)
};

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t rna_bits(float x) { return __float_as_uint(x) + 0x1000u; }
// Split for compensated products: the rounded value itself (low 13 bits cleared) and the TF32
// operand of what the rounding lost.
__device__ __forceinline__ uint32_t tf32_hi(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
__device__ __forceinline__ uint32_t tf32_lo(float x, uint32_t hi) { return rna_bits(x - __uint_as_float(hi)); }

__device__ __forceinline__ float4 ldg_f4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

constexpr int kWarpsPerBlock = 4;

// Tile encodings the kernels read: dense SR-BCRS tiles, ME-TCF COO runs, MCO bitmaps.
constexpr int kFmtSrbcrs = 0, kFmtMetcf = 1, kFmtMco = 2;

// MCO: the 4 consecutive operand positions 4*lane .. 4*lane+3 of a tile as TF32 operand bits
// (rounded to nearest, ties away), from the tile's two mask words and its compact values
// (values in ascending position order): position p holds value number popcount(mask bits below p).
__device__ __forceinline__ uint4 mco_expand(unsigned long long m0, unsigned long long m1, const uint32_t* vals, int lane) {
    const unsigned long long m = (lane & 16) ? m1 : m0;
    const int sh = 4 * (lane & 15);
    const uint32_t bits = (uint32_t)(m >> sh) & 0xFu;
    int at = ((lane & 16) ? __popcll(m0) : 0) + __popcll(m & ((1ull << sh) - 1ull));
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (bits & 1u) o.x = vals[at++] + 0x1000u;
    if (bits & 2u) o.y = vals[at++] + 0x1000u;
    if (bits & 4u) o.z = vals[at++] + 0x1000u;
    if (bits & 8u) o.w = vals[at] + 0x1000u;
    return o;
}

// x + (-0.0f) == x bit for bit for every x (NaN payloads aside); as opaque assembly it yields a
// fresh register.
__device__ __forceinline__ float detach(float x) {
    float y;
    asm volatile("add.rn.f32 %0, %1, 0f80000000;" : "=f"(y) : "f"(x));
    return y;
}

// Writes (and clears) a warp's accumulators for a fragment of window `win`: straight to C when the fragment is
// its whole window (part < 0), else to partial tile `part` in scratch.  acc[q][j][i]: 32-column group q, MMA j
// (column cb + 4n + j), accumulator register i.  GUARD: there may be fewer than 32 NQ columns.
template <int NQ, bool GUARD>
__device__ __forceinline__ void write_fragment(const SpmmArgs& p, int win, int part, int col_base, int g, int k, float (&acc)[NQ][4][4]) {
    const bool whole = part < 0;
    const int64_t ld = whole ? p.ldc : p.N;
    const int row = win * kWinRows + g, rows_ok = whole ? p.M - win * kWinRows : kWinRows;
    const bool relu = p.relu && whole;
    const bool plain = !whole || (p.vec_out && p.n_peer_out == 0);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const bool in = g + 8 * h < rows_ok;
        float* at = whole ? p.C + (int64_t)(p.row_map && in ? p.row_map[row + 8 * h] : row + 8 * h) * ld
                          : p.scratch + ((int64_t)part * kWinRows + g + 8 * h) * ld;
        at += col_base + 8 * k;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            // A 128-bit store needs its four values in consecutive registers, and so does every
            // MMA accumulator quad -- with a different grouping.  detach() gives the store its own
            // registers, so the unavoidable moves happen here, once per fragment, instead of around
            // every MMA of the main loop.
            float4 v0 = make_float4(detach(acc[q][0][2 * h]), detach(acc[q][1][2 * h]), detach(acc[q][2][2 * h]), detach(acc[q][3][2 * h]));
            float4 v1 = make_float4(detach(acc[q][0][2 * h + 1]), detach(acc[q][1][2 * h + 1]), detach(acc[q][2][2 * h + 1]),
                                    detach(acc[q][3][2 * h + 1]));
            if (relu) {
                v0.x = fmaxf(v0.x, 0.f); v0.y = fmaxf(v0.y, 0.f); v0.z = fmaxf(v0.z, 0.f); v0.w = fmaxf(v0.w, 0.f);
                v1.x = fmaxf(v1.x, 0.f); v1.y = fmaxf(v1.y, 0.f); v1.z = fmaxf(v1.z, 0.f); v1.w = fmaxf(v1.w, 0.f);
            }
            const int left = p.N - (col_base + 8 * k + 32 * q);   // columns from here on
            if (plain) {
                if (in && (!GUARD || left > 0)) *reinterpret_cast<float4*>(at + 32 * q) = v0;
                if (in && (!GUARD || left > 4)) *reinterpret_cast<float4*>(at + 32 * q + 4) = v1;
            } else if (in && !p.vec_out) {   // C with an odd row length (never together with peers' copies)
                const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (left + p.n_out - p.N > i) at[32 * q + i] = v[i];
            } else if (in) {   // the same row into every peer's copy of C (plain stores over NVLink)
                const int64_t off = at + 32 * q - p.C;
                for (int j = -1; j < p.n_peer_out; j++) {
                    float* to = (j < 0 ? p.C : p.peer_out[j] + p.peer_col) + off;
                    if (left > 0) *reinterpret_cast<float4*>(to) = v0;
                    if (left > 4) *reinterpret_cast<float4*>(to + 4) = v1;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[q][j][i] = 0.f;
}

// spmm_mma.cu: the array entry points, in pieces of at most `most` columns.  Scratch for one piece.
int spmm_arrays(const mask_plan* plan, const mask_matrix& m, int32_t N, const float* d_B, int64_t ldb, float* d_C, int64_t ldc, void* d_scratch,
                size_t scratch_bytes, int epilogue, void* stream, int32_t most);
constexpr int32_t kPieceColumns = 1 << 21;

// spmm_sweep.cu: persistent tcgen05 kernel, any N % 4 == 0, groups of any length.  nslab = 128-column
// slabs per column block (1, 2, 4; 0 = by N).
int launch_spmm_sweep(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st, int nslab);

// spmm_tma.cu: persistent tcgen05 kernel fed by the tensor memory accelerator (SR-BCRS with a prepared
// plan, see mask_plan_prepare_values).
bool spmm_tma_applies(const mask_plan* plan, const SpmmArgs& a);
int launch_spmm_tma(const mask_plan* plan, const SpmmArgs& a, int64_t K, cudaStream_t st, int nslab);

// spmm_warp.cu: one warp per block, every encoding.  nq = 32-column groups per warp (1..4; 0 = by N).
template <int FMT>
int launch_spmm_warp(const mask_plan* plan, const SpmmArgs& a, cudaStream_t st, int nq);
void warp_shape(const mask_plan* plan, int fmt, int N, bool comp, int tuned_nq, int* columns, int* step_tiles);   // what it would take

}  // namespace mask
