// Execution plan: fragments of consecutive tiles, grouped per thread block.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "mask_b200.h"

// Fragment f covers tiles [frag_off[f], frag_off[f+1]) of window frag_win[f]; fragments are in
// window order, so tile ranges are contiguous and windows without tiles appear as empty
// fragments (their rows of C must still be written).  frag_slot[f] is -1 when the fragment is
// its whole window (direct store to C) and otherwise the index of its 16xN partial tile in
// scratch.  Thread block g processes fragments [group_off[g], group_off[g+1]); the blocks of the
// warp-level kernel have groups of their own.  heads lists, for the fix-up pass, the first
// fragment of every split window and the number of its pieces.
struct mask_plan {
    int32_t M = 0;
    int32_t W = 0;
    int64_t T = 0;
    int policy = 0;
    int32_t group_tiles = 0;
    int64_t F = 0;  // fragments
    int64_t G = 0;  // groups (thread blocks)
    int64_t Gw = 0; // groups of the warp-level kernel
    int32_t piece_tiles = 0;  // windows of more than 5/4 of this are split
    int64_t P = 0;  // fragments that are part of a split window
    int64_t H = 0;  // split windows
    int64_t P_group = 0;  // P if windows were split into pieces of group_tiles
    int32_t nslab = 0;  // persistent kernel: 128-column slabs per column block (0 = the widest N fills)
    int device = 0;
    std::vector<int32_t> h_frag_off, h_frag_win, h_group_off;   // tables built on the host (every policy but AUTO)
    int32_t* d_tables = nullptr;         // owned: one array that holds all of the following
    int32_t* d_frag_off = nullptr;
    int32_t* d_frag_win = nullptr;
    int32_t* d_frag_slot = nullptr;
    int32_t* d_group_off = nullptr;
    int32_t* d_group_tile = nullptr;  // first tile of every group, then T
    // groups of the warp-level kernel: first fragment, end, first tile, tiles; NULL: it takes the plan's own groups.  The
    // warp_first groups of d_warp_first are taken before the others, among which they are empty.
    const int4* d_warp_group = nullptr;
    const int4* d_warp_first = nullptr;
    int32_t warp_first = 0;
    const int2* d_heads = nullptr;
    int32_t* d_status = nullptr;  // device status word: non-zero after a kernel gave up on a bounded wait
    const int32_t* d_row_map = nullptr;  // optional, not owned: output row of packed row i (a row reorder's order[])
    float* const* d_peer_out = nullptr;  // optional, not owned: device array of n_peer_out extra output bases
    int32_t n_peer_out = 0;
    // what the kernel choice goes by besides the features (choose_plan_parameters; without column features false)
    bool local = false;           // neighbouring windows share the rows of B they gather
    bool two_slabs_kept = false;  // hub-heavy, and B is 8 to 12 times the L2
    mask_column_features col_features = {};   // set by mask_plan_autotune
    int32_t has_col_features = 0;
    float* d_vals_tf32 = nullptr;        // owned: val_block_val rounded to TF32 (mask_plan_prepare_values), for the TMA kernel
    const float* vals_src = nullptr;     // the array d_vals_tf32 was made from
};
