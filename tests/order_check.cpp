// How launches behind a step's grouping go out: prints nothing and returns 0, or the line that does not hold.
#include <cstdio>

#include "../pocket-engine_b200/csrc/plora_order.h"

#define CHECK(c)                                       \
    do {                                               \
        if (!(c)) {                                    \
            std::printf("%d: %s\n", __LINE__, #c);     \
            return 1;                                  \
        }                                              \
    } while (0)

int main() {
    const LaunchOrder::Stream A = {0, 0}, B = {2, 0}, captured = {2, 7};
    LaunchOrder o;
    auto go = [&](LaunchOrder::Stream s, bool can_wait) {
        const auto l = o.next(s, can_wait);
        o.launched(s);
        return l;
    };
    CHECK(!go(A, true).pdl && go(A, true).pdl);  // nothing known of the stream, then a launch of ours
    // a step on one stream: the first launch waits before it reads, or is a plain one; the ones behind it need not
    o.grouped();
    auto l = go(A, true);
    CHECK(l.pdl && l.late);
    l = go(A, true);
    CHECK(l.pdl && !l.late);
    o.grouped();
    CHECK(!go(A, false).pdl && go(A, false).pdl);
    // rows quantised on another stream in between: the shrink is still the first behind the grouping on its own
    o.grouped();
    go(B, true);
    CHECK(go(A, true).late);
    // a shrink on the side stream, then an apply and an expand on the main one without a join
    o.grouped();
    CHECK(go(B, true).late && go(A, true).late && !go(B, true).late && !go(A, true).late);
    o.grouped();
    CHECK(go(B, true).late && !go(A, false).pdl);
    // what is captured, and what is launched on the same stream behind the capture
    o.grouped();
    CHECK(go(B, true).late && go(captured, true).late && !go(captured, true).late && !go(B, true).late);
    // tile words of the next step: plain launches on every stream
    o.reset();
    CHECK(!go(A, true).pdl && !go(B, true).pdl && go(B, true).pdl);
    // more streams than are kept: the forgotten ones wait again
    o.grouped();
    for (uint64_t s = 100; s < 200; s++) CHECK(go({s, 0}, true).late);
    CHECK(o.next({100, 0}, true).late && !o.next({199, 0}, true).late);
    // the tile shrink beside a cluster kernel that lets it start before its own wait
    CHECK(!tile_shrink_beside(true, false, 0, false));
    CHECK(tile_shrink_beside(true, false, 0, true) && tile_shrink_beside(true, true, 0, false) && tile_shrink_beside(true, false, 1, false));
    CHECK(!tile_shrink_beside(false, true, 1, true));
    return 0;
}
