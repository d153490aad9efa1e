"""The step's grouping runs a thread per tile of as many tiles as the caller says there may be: with more of them it goes over them in
rounds, and the result is the same, as it is beside the order that numpy finds."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_seqs,slots", [(1, 1), (127, 5), (128, 127), (129, 128), (400, 300), (1100, 7)])
def test_rounds(pe, n_seqs, slots):
    from pocket_engine_b200 import workloads
    rng = np.random.default_rng(n_seqs)
    rows = rng.choice([1, 1, 1, 2, 15, 16, 17, 33, 64, 150], n_seqs).tolist()
    which = rng.integers(0, slots + 1, n_seqs).tolist()
    wl = workloads.Workload("rounds", [pe.Site.fused(0, 64, [("a", 64)])] * 2, [8] * slots, 1.0, rows, which, 43)
    loras = harness.product_registry(pe, wl)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    seen = []
    for hint in (loras.max_lora_tiles(), 1, 200):
        seg = harness.SegView(loras, loras.lora_step(hint))
        seen.append([np.array(v).copy() for v in (seg.perm, seg.act, seg.seg_off, seg.mma, seg.work)])
    for other in seen[1:]:
        for a, b in zip(seen[0], other):
            assert np.array_equal(a, b)
    start = np.concatenate([[0], np.cumsum(rows)])
    # runs: neighbours of one slot count as one
    run_of, runs = [], []
    for i, s in enumerate(which):
        if i == 0 or s != which[i - 1] or s == 0:
            runs.append(0)
        runs[-1] += rows[i]
        run_of.append(len(runs) - 1)
    want = [t for slot in range(1, slots + 1) for i in range(n_seqs) if which[i] == slot and runs[run_of[i]] < 64
            for t in range(start[i], start[i + 1])]
    assert np.array_equal(seen[0][0], np.array(want, np.int32))
    loras.device_status()
    loras.close()
