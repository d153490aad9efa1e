"""The cluster kernel of plora_apply over layers whose parts are no multiples of 8 wide: rows of y move in pairs of columns there, and which
shares end in one depends on the number of column groups, which may not change a bit. And layers in which it is the slower
kernel for steps of many items: they run as the shrink / expand pair."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu

UNEVEN = [
    (4096, [("a", 4100)]),                        # one to three groups, each of them with an odd last share
    (2048, [("a", 1030), ("b", 2050)]),
    (1024, [("g", 6148), ("u", 6148)]),           # the second part's rows of y start at a multiple of 4
    (5120, [("q", 2054), ("k", 1030), ("v", 518)]),
]


def workload(pe, ranks, rows, slots, which):
    from pocket_engine_b200 import workloads
    sites = [pe.Site.fused(i, cols, mods) for i, (cols, mods) in enumerate(which)]
    return workloads.Workload("uneven", sites, ranks, 1.0, rows, slots, 41)


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("ranks", [[32, 16], [48]], ids=str)
def test_uneven_widths(pe, ranks, f32_out):
    for n in (1, 3, 5, 9):
        rows = [n] + [1] * (len(ranks) - 1)
        wl = workload(pe, ranks, rows, [1 + i for i in range(len(rows))], UNEVEN)
        harness.run_and_check(pe, wl, f32_out=f32_out, meta="device", fused="cluster")


@pytest.mark.parametrize("f32_out", [True, False])
def test_bits_whatever_the_number_of_groups(pe, f32_out):
    ranks = [16, 16, 32, 8]
    rows, slots = [1] * 40, [1 + i % 4 for i in range(40)]
    wl = workload(pe, ranks, rows, slots, UNEVEN)
    n = len(UNEVEN)
    xs, ys = [wl.x_bits(i) for i in range(n)], [wl.y_base(i) for i in range(n)]

    def run(first, count):
        w = workload(pe, ranks, rows[first:first + count], slots[first:first + count], UNEVEN)
        loras = harness.product_registry(pe, w)
        got = harness.run_gpu(pe, loras, w, f32_out, meta="device", fused="cluster", xs=[x[first:first + count] for x in xs],
                              y_base=[y[first:first + count] for y in ys])
        loras.close()
        return got

    together = run(0, 40)
    for first, count in ((0, 1), (1, 1), (2, 1), (3, 1), (4, 7)):
        for got, all_rows in zip(run(first, count), together):
            assert np.array_equal(got, all_rows[first:first + count]), (first, count)


# layers that the cluster kernel could run, in three or four column groups, and in which it is the slower one for steps of many items
BEYOND = [(32, 4096, [("g", 12288), ("u", 12288)]), (48, 2048, [("g", 6144), ("u", 6144)]), (64, 1024, [("g", 3072), ("u", 3072)])]


@pytest.mark.parametrize("rank,cols,mods", BEYOND, ids=lambda v: str(v) if isinstance(v, int) else "")
def test_layers_beyond_the_line_run_as_pairs(pe, rank, cols, mods):
    wl = workload(pe, [rank], [3], [1], [(cols, mods)])
    got = []
    for form in ("cluster", "early"):
        loras = harness.product_registry(pe, wl)
        got.append(harness.run_gpu(pe, loras, wl, True, meta="device", fused=form))
        loras.close()
    assert np.array_equal(got[0][0], got[1][0])
