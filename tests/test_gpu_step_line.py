"""Steps on both sides of the size from which long runs become tensor-core tiles when the caller has set no line: the
routing, and every form of the path against the oracle."""
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [[256], [257], [1, 255, 64], [64], [64] * 4, [64] * 4 + [1]], ids=str)
def test_default_line(pe, rows):
    from pocket_engine_b200 import workloads
    slots = [1 + i % 3 for i in range(len(rows))]
    wl = workloads.Workload("line", [pe.Site.fused(0, 1032, [("a", 264), ("b", 72)])], [16, 40, 128], 1.0, rows, slots, 37)
    loras = harness.product_registry(pe, wl)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    seg = harness.SegView(loras, loras.lora_step(loras.max_lora_tiles()))
    assert bool(len(seg.mma)) == (sum(rows) > 256)
    loras.close()
    for form in (False, "early", "cluster"):
        harness.run_and_check(pe, wl, f32_out=True, meta="device", fused=form)
