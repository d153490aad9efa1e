"""A step whose calls go to several streams: every kernel reads the launch records of its own step, however the calls interleave."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu

COLS, PARTS, T = 1024, [("a", 512), ("b", 256)], 96


@pytest.mark.parametrize("form", ["quantised-elsewhere", "shrink-elsewhere", "apply-after-a-shrink-elsewhere"])
def test_calls_interleaved_over_streams(pe, form):
    import torch
    from pocket_engine_b200 import workloads
    site = pe.Site.fused(0, COLS, PARTS)
    wl = workloads.Workload("streams", [site], [16, 32, 8, 64], 1.0, [1] * T, [0] * T, 13)
    loras = harness.product_registry(pe, wl)
    loras.set_apply_mode(1)
    hook, N, rng = loras.hook(0), site.width(), np.random.default_rng(2)
    x = harness.to_dev_bf16(wl.x_bits(0), 0)
    base = torch.randn(T, N, device="cuda")
    xq, st = torch.empty(T, COLS, dtype=torch.uint8, device="cuda"), torch.empty(T, device="cuda")
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    m, s = main.cuda_stream, side.cuda_stream
    slots = [torch.from_numpy(rng.integers(0, 5, T).astype(np.int32)).cuda() for _ in range(8)]
    cu = torch.arange(T + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def step(which, y, wait):
        def done():
            if wait:
                torch.cuda.synchronize()
        with torch.cuda.stream(main):
            y.copy_(base)
        loras.meta_build(cu.data_ptr(), slots[which].data_ptr(), T, m)
        step = loras.lora_step(loras.max_lora_tiles(), m, decode=True)
        done()
        if form == "quantised-elsewhere":  # (independent of the step)
            loras.fp8_quant_rows(x.data_ptr(), T, COLS, xq.data_ptr(), st.data_ptr(), s)
            done()
            loras.shrink(hook, step, x.data_ptr(), T, m)
            done()
            loras.expand(hook, step, T, y.data_ptr(), N, True, m)
        else:
            loras.fork(m, s)
            loras.shrink(hook, step, x.data_ptr(), T, s)
            done()
            if form == "shrink-elsewhere":
                loras.join(m, s)
                loras.expand(hook, step, T, y.data_ptr(), N, True, m)
            else:  # the cluster kernel keeps its sums to itself: it needs nothing of the shrink on the other stream
                loras.apply(hook, step, x.data_ptr(), T, y.data_ptr(), N, True, m)
                done()
                loras.join(m, s)
        done()

    want = []
    for k in range(len(slots)):
        want.append(torch.empty(T, N, device="cuda"))
        step(k, want[k], True)
    ys = [torch.empty(T, N, device="cuda") for _ in range(5 * len(slots))]
    torch.cuda.synchronize()
    for i, y in enumerate(ys):
        step(i % len(slots), y, False)
    torch.cuda.synchronize()
    loras.device_status()
    for i, y in enumerate(ys):
        assert torch.equal(y, want[i % len(slots)]), i
    loras.close()
