// The units by which the few-token kernels share their work: plain arithmetic, for the host and the device.
#pragma once
#include "../../include/plora.h"

#ifdef __CUDACC__
#define PLORA_HD __host__ __device__ __forceinline__
#else
#define PLORA_HD inline
#endif

// Units of an item. Shrink: SHR_ROWS rows of the stacked A over one K-split. Expand: what an output column costs. Blocks get
// equal shares of the sum, cut at multiples of 32 columns. The costs are times measured on stretches of every kind, in
// 0.35 us per 1000 columns with two blocks per SM: what a column of B and y takes is not in proportion to its bytes. (With a
// fixed number of columns per unit the slowest blocks took three times as long as the rest, with bytes twice as long.)
#define SHR_ROWS 16
#define EXP_GRAIN 32
PLORA_HD int expand_cost(int r, int cnt) {
    const int b = r <= 32 ? 12 : r <= 64 ? 21 : 21 + 11 * (r - 64) / 64;
    return (cnt > 8 ? 2 * b : b) + (cnt >> 2);
}

// A step's sum of these passes 32 bits (781 full items of rank 256 over 24,576 columns), so it has 64; a block's share of it
// and an item have 32. An item costs at most EXP_ITEM_MAX, or one unit a column where it has more columns than that. That is
// over what 16 tokens of rank 512 cost over 41,000 columns; wider ones share at a coarser scale. With the at most 12,864 items
// that a handle's metadata may hold, the sum stays under 1.08e11 (12,864 tokens' y would not fit the device if an item had
// more columns than EXP_ITEM_MAX) and a share of 64 or more blocks under 2^31.
#define EXP_ITEM_MAX (1 << 23)
#define PLORA_MAX_ITEMS 12864
// ... which limits what a column of a layer this wide may cost (found once, on the host)
inline int expand_most(long long width) { return width < 1 ? EXP_ITEM_MAX : width < EXP_ITEM_MAX ? (int)(EXP_ITEM_MAX / width) : 1; }
PLORA_HD int expand_col_cost(int r, int cnt, int most) {
    const int c = expand_cost(r, cnt);
    return c < most ? c : most;
}
PLORA_HD int expand_item_units(const int* r, const int* rows, int cnt, int most) {
    int units = 0;
    for (int p = 0; p < PLORA_MAX_PARTS; p++)
        if (r[p] > 0 && rows[p] > 0) units += rows[p] * expand_col_cost(r[p], cnt, most);
    return units;
}
PLORA_HD int shrink_item_units(int rank, int nsplit) { return (rank + SHR_ROWS - 1) / SHR_ROWS * nsplit; }

// Both kinds of units in one word, for one scan over the items: a step has at most 12,864 x (4 x 512 / 16 rows x 8 splits) =
// 13.2e6 units of the shrink, under 2^24.
#define UNIT_SHIFT 24
PLORA_HD unsigned long long pack_units(int expand, int shrink) { return ((unsigned long long)expand << UNIT_SHIFT) | (unsigned)shrink; }
PLORA_HD int packed_shrink(unsigned long long at) { return (int)(at & ((1u << UNIT_SHIFT) - 1)); }
PLORA_HD long long packed_expand(unsigned long long at) { return (long long)(at >> UNIT_SHIFT); }

// A layer's unit counts in memory: for the shrink [items, units before item 0, 1, ..., all] in 32 bits, then, from
// unit_expand(rec_cap) on, for the expand [items and, from bit 32 on, blocks; all, units before item 0, 1, ..., all] in 64 bits. In
// 32-bit words:
PLORA_HD int unit_expand(int rec_cap) { return (rec_cap + 2 + 1) & ~1; }
PLORA_HD int unit_words(int rec_cap) { return unit_expand(rec_cap) + 2 * (rec_cap + 3); }

// How many of the grid's blocks share the expand's sum: no less than about 200 columns each. Where all items cost the same
// (first: the units of the first one) and there are at least eight blocks for each, as many as divide by the items (by two each,
// for two parts of one width): a block whose share ends in another item or part starts twice, which the rest then waits for.
// Shrink / expand bracket, two layers: 16 tokens of 16 rank-16 adapters 97 -> 86 us, 256 tokens of 16 145 -> 129, 8 of 8 rank-64
// ones 98 -> 93. (Found by the grouping kernel: the same arithmetic at the head of every block took 0.1 us a launch.)
PLORA_HD int share_blocks(long long total, int items, long long first, int grid) {
    const long long most = total / 2048;
    int blocks = most < 1 ? 1 : most < grid ? (int)most : grid;
    if (items < 1 || total != first * items) return blocks;
    if (16 * items <= blocks) blocks -= blocks % (2 * items);
    else if (8 * items <= blocks) blocks -= blocks % items;
    return blocks;
}
// A block's share of the expand's sum: [share_at(total, b, n), share_at(total, b + 1, n))
PLORA_HD long long share_at(long long total, int block, int blocks) { return total * block / blocks; }
// the units before an item, counted from the block's first unit: exact for the items that meet the share
PLORA_HD int units_from(long long before, long long first) {
    const long long d = before - first;
    return d > 0x7fffffffLL ? 0x7fffffff : d < -0x7fffffffLL ? -0x7fffffff : (int)d;
}

// The block's next stretch: the part of the item that the sum reaches at `local` (into the item), and its columns up to
// `left` further. Returns how much of the sum that is. Both blocks at a cut round it the same way.
PLORA_HD int expand_stretch_at(const int* r, const int* rows, int cnt, int most, int local, int left, int& part, int& c0, int& c1) {
    for (part = 0; part < PLORA_MAX_PARTS; part++) {
        if (r[part] <= 0 || rows[part] <= 0) continue;
        const int each = expand_col_cost(r[part], cnt, most), all = rows[part] * each;
        if (local < all) {
            const int take = left < all - local ? left : all - local;
            const unsigned grain = EXP_GRAIN * (unsigned)each;
            const int lo = (int)(((unsigned)local + grain - 1) / grain * EXP_GRAIN), hi = (int)(((unsigned)local + (unsigned)take + grain - 1) / grain * EXP_GRAIN);
            c0 = lo < rows[part] ? lo : rows[part];
            c1 = take == all - local || hi > rows[part] ? rows[part] : hi;
            return take;
        }
        local -= all;
    }
    part = c0 = c1 = 0;
    return left;
}
