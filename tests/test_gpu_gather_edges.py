"""The few-token shrink and expand at the edges of their units: every width of the rank, work items of 1, 8, 9 and 16
tokens, input ranges and output columns that end inside a unit, more work items than a block keeps counts for, and the
cluster kernel over steps of fewer and of more adapters than clusters run at once."""
import pytest

import harness

pytestmark = pytest.mark.gpu

CASES = [
    # name, rows of the sequences, ranks, input width, parts
    ("every-rank", [1, 8, 9, 16, 7, 2, 1, 3, 17], [8, 16, 24, 32, 48, 64, 80, 96, 128], 1032, [("a", 520), ("b", 72)]),
    ("ranks-above-128", [5, 1, 16], [144, 200, 256], 544, [("a", 264)]),
    ("outputs-off-16-bytes", [3, 16, 1], [16, 40], 64, [("a", 34), ("b", 6), ("c", 130)]),
    ("narrow-inputs", [9, 1], [32, 8], 8, [("a", 8)]),
    ("many-work-items", [1] * 300, [8] * 300, 128, [("a", 96)]),
    ("untargeted", [1, 1, 1, 2], [16, 8, 16, 16], 2056, [("a", 40), ("b", 1024)]),
]


@pytest.mark.parametrize("form", [False, "early", "cluster"], ids=["bracket", "pair", "apply"])
@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_few_token_edges(pe, case, f32_out, form):
    from pocket_engine_b200 import workloads
    name, rows, ranks, cols, mods = case
    slots = [1 + i % len(ranks) for i in range(len(rows))]
    wl = workloads.Workload(name, [pe.Site.fused(0, cols, mods)], ranks, 1.0, rows, slots, 29)
    if name == "untargeted":  # one adapter targets the narrow part only, one the wide part only
        factors = wl.factors
        wl.factors = lambda i: factors(i)[:1] if i == 1 else factors(i)[1:] if i == 2 else factors(i)
    harness.run_and_check(pe, wl, f32_out=f32_out, meta="device", fused=form)


@pytest.mark.parametrize("adapters", [14, 24, 48])
def test_apply_over_slot_counts(pe, adapters):
    from pocket_engine_b200 import workloads
    rows = [1] * (adapters + 5)
    slots = [i % (adapters + 1) for i in range(len(rows))]
    wl = workloads.Workload("slots-%d" % adapters, [pe.Site.fused(0, 1024, [("a", 1024)]), pe.Site.fused(0, 2048, [("g", 3072), ("u", 3072)])],
                            [16] * adapters, 1.0, rows, slots, 31)
    harness.run_and_check(pe, wl, f32_out=True, meta="device", fused="cluster")
