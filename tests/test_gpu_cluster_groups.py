"""The cluster kernel of plora_apply over its column groups: steps of few work items take more of them (each loads and multiplies
only the rows of A of the parts its columns meet), with the same bits as in a step of many; ranks that its expand walks 16
and 32 at a time; one to nine tokens of an adapter (groups of four, passes of eight); inputs that end inside a block's share,
inside a step of 32 and inside a warp's round; shares of columns that are no multiple of a step."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu

SITES = [
    (4096, [("q", 4096), ("k", 1024), ("v", 1024)]),
    (1032, [("a", 520), ("b", 136), ("c", 72)]),  # four blocks have inputs, 40 of the last one's
    (5160, [("g", 2056), ("u", 2056)]),
    (17416, [("d", 264)]),                        # more than eight steps of 32 inputs for a warp
    (8, [("t", 40)]),
]


def workload(pe, ranks, rows, slots):
    from pocket_engine_b200 import workloads
    sites = [pe.Site.fused(i, cols, mods) for i, (cols, mods) in enumerate(SITES)]
    return workloads.Workload("groups", sites, ranks, 1.0, rows, slots, 41)


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("ranks", [[16], [32, 16], [48], [64, 24]], ids=str)
def test_groups(pe, ranks, f32_out):
    for n in (1, 2, 4, 5, 8, 9):
        rows = [n] + [1] * (len(ranks) - 1)
        wl = workload(pe, ranks, rows, [1 + i for i in range(len(rows))])
        harness.run_and_check(pe, wl, f32_out=f32_out, meta="device", fused="cluster")


@pytest.mark.parametrize("f32_out", [True, False])
def test_bits_whatever_the_number_of_groups(pe, f32_out):
    ranks = [16, 16, 32, 8]
    rows, slots = [1] * 40, [1 + i % 4 for i in range(40)]
    wl = workload(pe, ranks, rows, slots)
    n = len(SITES)
    xs, ys = [wl.x_bits(i) for i in range(n)], [wl.y_base(i) for i in range(n)]

    def run(first, count):
        w = workload(pe, ranks, rows[first:first + count], slots[first:first + count])
        loras = harness.product_registry(pe, w)
        got = harness.run_gpu(pe, loras, w, f32_out, meta="device", fused="cluster", xs=[x[first:first + count] for x in xs],
                              y_base=[y[first:first + count] for y in ys])
        loras.close()
        return got

    together = run(0, 40)
    for first, count in ((0, 1), (1, 1), (2, 1), (3, 1), (4, 7)):
        for got, all_rows in zip(run(first, count), together):
            assert np.array_equal(got, all_rows[first:first + count]), (first, count)
