"""The tile path's expand at the edges of its tiles: more tiles than its grid is deep, every width of the swizzled boxes of
B, column blocks that end inside a box, ranks with two and three accumulators, both output types."""
import pytest

import harness

pytestmark = pytest.mark.gpu

CASES = [
    # runs of 64 to 66 tokens: twice as many tiles as a step of full ones has
    ("many-short-runs", [65, 64, 66] * 10, [16, 32, 48], 256, [("a", 328), ("b", 64)]),
    ("rank-64-and-untargeted", [130, 64, 257], [64, 16], 520, [("a", 72), ("b", 1000)]),
    ("ranks-of-every-box", [200, 70, 64, 128, 129, 91], [16, 32, 48, 64, 96, 128], 1024, [("a", 130)]),
    ("one-column-block", [64], [80], 64, [("a", 8)]),
    # total ranks of 384 and 144 whose rows of A go to several blocks, the last of which has 16; and too many tiles for that
    ("rank-groups", [300, 70], [128, 48], 1032, [("a", 64), ("b", 40), ("c", 8)]),
    # registries with ranks over 64 stage S in another form: four planes of a rank of 96, eight of a rank of 16 (one and two planes above)
    ("planes-of-high-ranks", [200, 90], [96, 16], 4096, [("a", 72)]),
    ("rank-groups-no-room", [128] * 60, [96, 16], 520, [("a", 64), ("b", 40)]),
]


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_tile_expand_edges(pe, case, f32_out):
    from pocket_engine_b200 import workloads
    name, rows, ranks, cols, mods = case
    slots = [1 + i % len(ranks) for i in range(len(rows))]
    wl = workloads.Workload(name, [pe.Site.fused(0, cols, mods)], ranks, 1.0, rows, slots, 19)
    if "untargeted" in name:  # the second adapter leaves the wide part alone
        factors = wl.factors
        wl.factors = lambda i: factors(i)[:1] if i == 1 else factors(i)
    harness.run_and_check(pe, wl, f32_out=f32_out, meta="device", run_min=64)
