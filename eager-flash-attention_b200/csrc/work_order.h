// The order in which a causal attention launch takes its work items where nobody waits for particular rows: longest first,
// over groups of heads. No CUDA in here, so that the CPU tests compile it too.
#pragma once

#ifdef __CUDACC__
#define EFA_HD __host__ __device__ __forceinline__
#else
#define EFA_HD inline
#endif

namespace efa {

// Item `unit` of heads * splits * blocks, taken in groups of `group` heads (the last one may have fewer). Within a group the row blocks
// go from the last to the first and the heads of the group in turn; with splits by how far a block's rows reach past the first
// key of a split, split_blocks = row blocks to the length of a split (at least 1): the items that have all keys of their split, then the
// shorter ones, then those the mask leaves nothing of. Every item comes exactly once, whatever the numbers.
EFA_HD void grouped_item(int unit, int heads, int splits, int blocks, int group, int split_blocks, int& head, int& split, int& block)
{
    const int per_group = group * splits * blocks;
    const int g = unit / per_group;
    int rem = unit - g * per_group;
    const int h0 = g * group, nh = heads - h0 < group ? heads - h0 : group;
    if (splits == 1) {
        const int d = rem / nh;
        head = h0 + (rem - d * nh);
        split = 0;
        block = blocks - 1 - d;
        return;
    }
    // Diagonal d = blocks - 1 - block + split * split_blocks, from 0 on. On it lie the splits lo .. hi; both ends only move at
    // multiples of split_blocks, from 0 and from `blocks` on.
    int pos = 0, lo = 0, hi = 0, next_hi = split_blocks, next_lo = blocks;
    while (true) {
        const bool more = hi < splits - 1;
        const int end = more && next_hi < next_lo ? next_hi : next_lo;
        const int n = (hi - lo + 1) * nh, len = (end - pos) * n;     // hi - lo = -1: a diagonal between two splits' blocks, empty
        if (rem < len || (!more && lo == splits - 1)) {
            const int d = pos + rem / n, r = rem - (d - pos) * n;
            split = lo + r / nh;
            head = h0 + r - (split - lo) * nh;
            block = blocks - 1 - d + split * split_blocks;
            return;
        }
        rem -= len;
        pos = end;
        if (more && end == next_hi) { hi++; next_hi += split_blocks; }
        if (end == next_lo) { lo++; next_lo += split_blocks; }
    }
}

}  // namespace efa
