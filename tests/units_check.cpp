// Walks the few-token kernels' shares of a step as their blocks do, and checks that the stretches of columns follow one another
// without a gap or an overlap. Arguments: items, tokens per item, blocks, blocks to walk at each end and in the middle (0: all),
// then rank and columns of every part. Prints the sum of all units.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../pocket-engine_b200/csrc/plora_units.h"

static int fail(const char* what, long long a, long long b) {
    std::printf("%s: %lld %lld\n", what, a, b);
    return 1;
}

int main(int argc, char** argv) {
    const int items = std::atoi(argv[1]), cnt = std::atoi(argv[2]), blocks = std::atoi(argv[3]), walk = std::atoi(argv[4]);
    int r[PLORA_MAX_PARTS] = {}, rows[PLORA_MAX_PARTS] = {}, rank = 0;
    long long width = 0;
    for (int p = 0; 5 + 2 * p < argc; p++) r[p] = std::atoi(argv[5 + 2 * p]), rows[p] = std::atoi(argv[6 + 2 * p]), rank += r[p], width += rows[p];
    const int most = expand_most(width);
    // the grouping kernel's scan
    std::vector<long long> before(items + 1);
    unsigned long long at = 0;
    for (int w = 0; w <= items; w++) {
        before[w] = packed_expand(at);
        if (packed_shrink(at) != w * shrink_item_units(rank, 8)) return fail("shrink units", w, packed_shrink(at));
        if (w < items) at += pack_units(expand_item_units(r, rows, cnt, most), shrink_item_units(rank, 8));
    }
    const long long total = before[items], item = expand_item_units(r, rows, cnt, most);
    if (total != items * item || item > 0x7fffffffLL) return fail("expand units", total, item);
    for (int grid = 1; grid <= 296; grid++) {  // the blocks that a grid gives the step
        const int n = share_blocks(total, items, item, grid);
        if (n < 1 || n > grid || (8 * items <= n && n % items != 0) || n < grid - grid / 8 - 1 - (total / 2048 < grid ? grid : 0)) return fail("blocks", grid, n);
        if (share_blocks(total + 1, items, item, grid) < n) return fail("blocks of unequal items", grid, n);
    }
    int last = -1, part0 = 0, col = 0, next = 0;  // where the block before ended: item, part, column; the block after it
    for (int b = 0; b < blocks; b++) {
        if (walk && b >= walk && b + walk < blocks && (b < blocks / 2 || b >= blocks / 2 + walk)) continue;
        const long long u0 = share_at(total, b, blocks), share = share_at(total, b + 1, blocks) - u0;
        if (share < 0 || share > 0x7fffffffLL) return fail("share", b, share);
        int w = 0;
        while (w + 1 < items && units_from(before[w + 1], u0) <= 0) w++;
        bool first = b != next;  // a block whose predecessor was not walked: its first stretch starts anywhere
        next = b + 1;
        for (int u = 0; u < (int)share;) {
            while (units_from(before[w + 1], u0) <= u) w++;
            const int local = u - units_from(before[w], u0);
            int part, c0, c1;
            const int take = expand_stretch_at(r, rows, cnt, most, local, (int)share - u, part, c0, c1);
            if (local < 0 || take <= 0 || c0 < 0 || c1 < c0 || c1 > rows[part]) return fail("stretch", c0, c1);
            if (first) last = w, part0 = part, col = c0, first = false;
            if (last != w || part0 != part) {  // on to the next part, or the next item's first
                if (last >= 0 && col != rows[part0]) return fail("columns left", col, rows[part0]);
                int p = last == w ? part0 + 1 : 0;
                while (r[p] <= 0 || rows[p] <= 0) p++;
                if ((last >= 0 && w != last && w != last + 1) || p != part) return fail("part", p, part);
                last = w, part0 = part, col = 0;
            }
            if (c0 != col) return fail("gap", col, c0);
            col = c1;
            u += take;
        }
    }
    if (last != items - 1 || col != rows[part0]) return fail("end", last, col);
    std::printf("%lld\n", total);
    return 0;
}
