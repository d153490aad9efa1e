"""Which kernels a run takes depends on the run alone, unless the caller draws another line: in steps of every size, and with
the same bits for a prompt alone and in any company."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


def workload(pe, rows, slots):
    from pocket_engine_b200 import workloads
    return workloads.Workload("line", [pe.Site.fused(0, 1032, [("a", 264), ("b", 72)])], [16, 40, 128], 1.0, rows, slots, 37)


@pytest.mark.parametrize("rows", [[64], [63], [256], [257], [1, 255, 64], [64] * 4 + [1], [63, 200]], ids=str)
def test_default_line(pe, rows):
    wl = workload(pe, rows, [1 + i % 3 for i in range(len(rows))])
    loras = harness.product_registry(pe, wl)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    seg = harness.SegView(loras, loras.lora_step(loras.max_lora_tiles()))
    assert sum(int(t[1]) for t in seg.mma) == sum(r for r in rows if r >= 64)
    loras.close()
    for form in (False, "early", "cluster"):
        harness.run_and_check(pe, wl, f32_out=True, meta="device", fused=form)


@pytest.mark.parametrize("form", [False, "early", "cluster"], ids=["bracket", "pair", "apply"])
@pytest.mark.parametrize("f32_out", [True, False])
def test_a_prompt_has_the_same_bits_in_any_company(pe, f32_out, form):
    rows, slots = [64, 1, 200, 30, 129, 300], [1, 2, 3, 1, 2, 1]
    wl = workload(pe, rows, slots)
    x, y = wl.x_bits(0), wl.y_base(0)

    def run(w, first, n):
        loras = harness.product_registry(pe, w)
        got = harness.run_gpu(pe, loras, w, f32_out, meta="device", fused=form, xs=[x[first:first + n]], y_base=[y[first:first + n]])[0]
        loras.close()
        return got

    together = run(wl, 0, sum(rows))
    for i in range(len(rows)):
        first = sum(rows[:i])
        assert np.array_equal(run(workload(pe, [rows[i]], [slots[i]]), first, rows[i]), together[first:first + rows[i]]), i
