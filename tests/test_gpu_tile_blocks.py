"""Steps whose runs of tokens are twice as many tiles as their rows let the host expect: the kernels take fewer blocks per tile than the
host allowed, each reader of the partial sums the same number, and the bits stay those of one block per tile."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu

# (total ranks 16 to 192, in registries whose rows of A go to several blocks and to one)
CASES = {
    "low-rank": ([16], [64] * 24, [("a", 64)]),
    "rank-groups": ([64, 16, 32], [64, 80] * 13, [("q", 128), ("k", 64), ("v", 64)]),
    "few-tiles": ([64, 16], [64, 200], [("q", 128), ("k", 64), ("v", 64)]),
}


@pytest.mark.parametrize("form", ["bracket", "cluster"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_bits_of_many_short_runs(pe, case, form):
    from pocket_engine_b200 import workloads
    ranks, rows, mods = CASES[case]
    wl = workloads.Workload(case, [pe.Site.fused(0, 4096, mods)], ranks, 1.0, rows, [1 + i % len(ranks) for i in range(len(rows))], 17)
    got = []
    for blocks in (1, 0):
        loras = harness.product_registry(pe, wl)
        loras.set_tile_split(blocks)
        got.append(harness.run_gpu(pe, loras, wl, True, meta="device", fused=False if form == "bracket" else form)[0])
        loras.close()
    assert np.array_equal(got[0], got[1])
    harness.run_and_check(pe, wl, f32_out=True, meta="device", fused=False if form == "bracket" else form, run_min=64)


def test_bits_of_a_layer_in_one_kernel(pe):
    """The same where the planes are added up in place before a one-kernel layer."""
    import torch
    from pocket_engine_b200 import workloads
    wl = workloads.Workload("one-kernel", [pe.Site.fused(0, 4096, [("a", 256)])], [32, 16], 1.0, [64] * 24, [1 + i % 2 for i in range(24)], 19)
    xd = harness.to_dev_bf16(wl.x_bits(0), 0)
    w = torch.randn(256, 4096, device="cuda", generator=torch.Generator("cuda").manual_seed(3)).mul_(1 / 64).bfloat16()
    got = []
    for blocks in (1, 0):
        loras = harness.product_registry(pe, wl)
        loras.set_tile_split(blocks)
        cu, ss = torch.from_numpy(wl.cu()).cuda(), torch.from_numpy(wl.row_slot.copy()).cuda()
        loras.meta_build(cu.data_ptr(), ss.data_ptr(), wl.n_seqs)
        step = loras.lora_step(loras.max_lora_tiles())
        y = torch.empty(wl.tokens, 256, dtype=torch.float32, device="cuda")
        hook = loras.hook(0)
        loras.shrink(hook, step, xd.data_ptr(), wl.tokens)
        loras.linear_bf16_fused(hook, step, xd.data_ptr(), w.data_ptr(), wl.tokens, y.data_ptr(), 256, True)
        torch.cuda.synchronize()
        loras.device_status()
        got.append(y.cpu().numpy())
        loras.close()
    assert np.array_equal(got[0], got[1])
