"""Steps whose gather kernels find no items release their tile kernels at once, which then wait by themselves: x and y written right
before each layer are seen, and S of a layer is not overwritten while the one before reads it. Every iteration has other
inputs; the same calls with the device idle in between give the bits."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["apply", "pair", "bracket"])
@pytest.mark.parametrize("rows", [[199], [700, 64, 130]], ids=str)
def test_prompts_behind_producers(pe, rows, form):
    import torch
    from pocket_engine_b200 import workloads
    sites = [pe.Site.fused(0, 1024, [("a", 1536), ("b", 512)]), pe.Site.fused(0, 2048, [("o", 1024)]), pe.Site.fused(0, 1024, [("c", 4096)])]
    wl = workloads.Workload("prompts", sites, [16, 40], 1.0, rows, [1 + i % 2 for i in range(len(rows))], 47)
    loras = harness.product_registry(pe, wl)
    loras.set_apply_mode(1 if form == "apply" else 0)
    stream = torch.cuda.current_stream().cuda_stream
    T = wl.tokens
    g = torch.Generator(device="cuda").manual_seed(7)
    src = [torch.randn(T, s.cols, device="cuda", generator=g).bfloat16() for s in sites]
    bases = [torch.randn(T, s.width(), device="cuda", generator=g).bfloat16() for s in sites]
    xs, ys = [torch.empty_like(s) for s in src], [torch.empty_like(b) for b in bases]
    words = harness.tiles_of(pe, wl, loras.max_lora_tiles())

    def step(i, idle):
        loras.meta_upload(words, stream)
        st = loras.lora_step(loras.max_lora_tiles(), stream)
        for si in range(len(sites)):
            torch.mul(src[si], 1.0 + 0.25 * (i % 5), out=xs[si])
            torch.mul(bases[si], 0.5 + 0.125 * (i % 3), out=ys[si])
            if idle:
                torch.cuda.synchronize()
            hook, y = loras.hook(si), ys[si]
            if form == "bracket":
                loras.shrink(hook, st, xs[si].data_ptr(), T, stream)
                if idle:
                    torch.cuda.synchronize()
                loras.expand(hook, st, T, y.data_ptr(), y.shape[1], False, stream)
            else:
                loras.apply(hook, st, xs[si].data_ptr(), T, y.data_ptr(), y.shape[1], False, stream)
            if idle:
                torch.cuda.synchronize()
        return [y.clone() for y in ys]

    want = {i: step(i, True) for i in range(15)}
    got = [step(i, False) for i in range(60)]
    torch.cuda.synchronize()
    loras.device_status()
    for i, out in enumerate(got):
        for a, b in zip(out, want[i % 15]):
            assert torch.equal(a, b), i
    loras.close()
