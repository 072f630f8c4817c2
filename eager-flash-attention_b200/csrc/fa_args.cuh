// Kernel arguments of the attention kernel.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>

#include "attention_plan.h"
#include "work_order.h"

namespace efa {

struct FaArgs {
    float*  O32;
    __half* O16;
    float*  O_part;
    float*  m_part;
    float*  l_part;
    int     part_rows;
    int     q_start, q_rows, S, H_local, nsplit, kv_len, causal;
    float   scale_log2e;
    int*    tile_counters;
    int     tile_rows;
    int*    status;
    int     band_blocks;    // 256-row blocks per band of the work order (0 or 1 = strict row order)
    int     counters_sys;   // the tile counters live in host memory: order the rows before the count at system scope
    const short* order_tab; // strict-order launches only: order_tab[k] = the 256-row block taken k-th
                            // (device memory, one entry per block); nullptr = first to last (or last to first, below)
    int     tail_first = -1, tail_total = 0;   // >= 0: the launch covers, as 128-row items, the 256-row items of a launch of tail_total from this one on
    float   rescale_above;  // log2 units by which a row maximum may outgrow the exponent offset in use
    int     group_heads = 0; // > 0 (no counters, causal): longest items first over groups of so many heads (work_order.h)
    int     heavy_first;    // take the row blocks (or bands) from the last to the first; with a causal
                            // mask the last rows sweep the most keys, so the longest items start first
};

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The denominator that goes into the partials of a split. +0 says that the mask leaves nothing of the split for the row: the merge does not read its O. A
// row that has keys there, all of them with a score of -inf, has no sum either, but O is 0 * V, NaN where V is not finite: -0 for that.
__device__ __forceinline__ float partial_sum(float l, bool has_keys)
{
    return has_keys && l == 0.f ? -0.f : l;
}
// ... and how the merge reads it.
__device__ __forceinline__ bool no_keys(float m, float l)
{
    return m == -INFINITY && __float_as_uint(l) == 0u;
}

// Work item `item` of a launch: head, split and first row. tail: 128-row items that are halves of the 256-row ones from a.tail_first on.
__device__ __forceinline__ void pick_item(int item, const FaArgs& a, int items_x, int items_total, int item_rows, bool tail,
                                          int& head, int& split, int& row0)
{
    // Causal and nobody waits for particular rows: longest items first over groups of heads (work_order.h). Else strict
    // row order (heads fastest), which makes every head's K/V stream live at once, far more than the L2 holds, or
    // bands: the blocks of one band of rows are taken head by head, so that the CTAs in flight share a few heads' K/V,
    // and rows still complete band by band, which is all a consumer that handles groups of tiles needs.
    int item_y;
    if (a.group_heads > 0) {
        grouped_item(item, a.H_local, a.nsplit, items_total / items_x, a.group_heads, max(1, a.kv_len / item_rows), head, split, item_y);
    } else {
        const int units = tail ? a.tail_total : items_total, unit = tail ? a.tail_first + item / 2 : item;
        const int items_y = units / items_x;
        const int band_items = a.band_blocks * (item_rows == 128 && !tail ? 2 : 1);
        const int band = band_items > 1 ? min(band_items, items_y) : 1;
        const int per_band = items_x * band;
        const int full = items_y / band;
        int b = unit / per_band, rem = unit - b * per_band, nb = band;
        if (b >= full) { b = full; rem = unit - full * per_band; nb = items_y - full * band; }
        const int item_x = rem / nb;
        item_y = b * band + rem % nb;
        // Longest items first: list scheduling then ends on the shortest items instead of the longest, which
        // is worth up to one item's duration (a fifth of the launch with four heads per GPU at 32k rows).
        if (a.order_tab != nullptr && band == 1) item_y = a.order_tab[item_y];
        else if (a.heavy_first) item_y = items_y - 1 - item_y;
        head  = item_x % a.H_local;
        split = item_x / a.H_local;
    }
    row0 = tail ? item_y * 256 + (item & 1) * 128 : item_y * item_rows;
}

// Warp-specialised kernel (fa_fwd_ws_sm100.cu).
// reserve_sms > 0: persistent grid that leaves that many SMs without an attention CTA.
// K and V maps for it have boxes of fa_ws_kv_box_rows() rows (its stage length); Q maps 128 rows.
int fa_ws_kv_box_rows();
int fa_ws_preload();    // loads the code of every instantiation of the kernel on the current device
FaPlan fa_ws_plan(const FaArgs& a, int d_h, int reserve_sms);
int fa_forward_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a,
                  int d_h, bool out_f16, int reserve_sms, cudaStream_t stream);


// One-tile kernel (fa_fwd_tile_sm100.cu), d_h 16 and 32; the same maps.
int fa_tile_preload();
int fa_forward_tile(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a,
                    int d_h, bool out_f16, cudaStream_t stream);

}  // namespace efa
