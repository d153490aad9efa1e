"""A step whose expand costs more units than 32 bits hold: every token gets its adapter term."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


def test_prompt_sized_step_above_rank_128(pe):
    import torch
    cols, width, ranks, tokens = 64, 24576, [512, 384], [7000, 1500]  # 438 items of 4.9 M units and 94 of 3.8 M
    site = pe.Site.fused(0, cols, [("gate", width // 2), ("up", width // 2)])
    T = sum(tokens)
    loras = pe.Loras([site], 2, 512, T, 2, device=0)
    rng = np.random.default_rng(5)
    prep, kept = loras.prep(), []
    for i, r in enumerate(ranks):
        f = [pe.Factors(0, p.module, (rng.standard_normal((r, cols)) * 0.1).astype(np.float32), (rng.standard_normal((p.rows, r)) * 0.1).astype(np.float32))
             for p in site.parts]
        loras.upload(1 + i, loras.insert(prep.prepare("a%d" % i, f)))
        kept.append(f)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(T, cols, device="cuda", generator=g).bfloat16()
    y = torch.randn(T, width, device="cuda", generator=g, dtype=torch.bfloat16)
    base = y.clone()
    loras.meta_upload(pe.fill_tiles(np.array(tokens, np.int32), np.array([1, 2], np.int32), loras.max_lora_tiles()))
    step = loras.lora_step(loras.max_lora_tiles())
    lin = pe.Linear(loras, 0)
    lin.forward(x.data_ptr(), T, y.data_ptr(), width, False, lora=step, main=torch.cuda.current_stream().cuda_stream, fused=False)
    torch.cuda.synchronize()
    loras.device_status()
    rows = torch.unique(torch.cat([torch.arange(0, T, 61), torch.tensor([0, 6999, 7000, T - 1])])).cuda()
    for i in range(2):
        mine = rows[(rows >= sum(tokens[:i])) & (rows < sum(tokens[:i + 1]))]
        want = base[mine].double()
        for q, f in enumerate(kept[i]):
            a, b = (torch.from_numpy(m).cuda().bfloat16().double() for m in (f.a, f.b))
            want[:, q * width // 2:(q + 1) * width // 2] += (x[mine].double() @ a.t()) @ b.t()
        got = y[mine].double()
        # one rounding to bf16 (half a step is 2^-9 of the value), and f32 sums of 64 and 512 products before it
        assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()), float((got - want).abs().max())
    loras.close()
