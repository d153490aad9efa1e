"""The one-kernel layers give a token the same bits on every run and in every company: the adapter passes of a tile are taken
when they happen to be staged, so nothing of y may depend on when that was."""
import pytest

import harness

pytestmark = pytest.mark.gpu

COLS, WIDTHS, RANKS = 4096, [1024, 2048], [64, 16, 128]


def layer(pe, kind, rows, slots, x, w, scales, f32_out, passes=1):
    """The layer's outputs of several runs over the same inputs."""
    import torch
    from pocket_engine_b200 import workloads
    wl = workloads.Workload("bits", [pe.Site.fused(0, COLS, [("p%d" % i, n) for i, n in enumerate(WIDTHS)])], RANKS, 1.0, rows, slots, 29)
    loras = harness.product_registry(pe, wl)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    step, hook, T, N = loras.lora_step(loras.max_lora_tiles()), loras.hook(0), len(x), sum(WIDTHS)
    ys = [torch.full((T, N), float("nan"), dtype=torch.float32 if f32_out else torch.bfloat16, device="cuda") for _ in range(passes)]
    xq = torch.empty(T, COLS, dtype=torch.uint8, device="cuda")
    st = torch.empty(T, device="cuda")
    for y in ys:
        if kind == "fp8":
            loras.fp8_quant_rows(x.data_ptr(), T, COLS, xq.data_ptr(), st.data_ptr())
        loras.shrink(hook, step, x.data_ptr(), T)
        if kind == "fp8":
            loras.linear_fp8_fused(hook, step, xq.data_ptr(), st.data_ptr(), w.data_ptr(), scales.data_ptr(), T, y.data_ptr(), N, f32_out)
        else:
            loras.linear_bf16_fused(hook, step, x.data_ptr(), w.data_ptr(), T, y.data_ptr(), N, f32_out)
    torch.cuda.synchronize()
    loras.device_status()
    loras.close()
    return ys


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_same_bits_on_every_run_and_in_every_company(pe, kind, f32_out):
    import torch
    rows, slots = [1, 520, 300, 1, 2500, 64, 1041, 1], [2, 1, 2, 0, 3, 1, 2, 3]
    g = torch.Generator(device="cuda").manual_seed(17)
    x = torch.randn(sum(rows), COLS, device="cuda", generator=g).bfloat16()
    w = torch.randn(sum(WIDTHS), COLS, device="cuda", generator=g) / COLS ** 0.5
    scales = 0.9 + 0.2 * torch.rand(sum(WIDTHS), device="cuda", generator=g)
    w = w.to(torch.float8_e4m3fn).view(torch.uint8) if kind == "fp8" else w.bfloat16()
    ys = layer(pe, kind, rows, slots, x, w, scales, f32_out, passes=6)
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
    for i in (1, 2, 4, 5, 6):  # a prompt in a step of its own
        at = sum(rows[:i])
        alone = layer(pe, kind, [rows[i]], [slots[i]], x[at:at + rows[i]].contiguous(), w, scales, f32_out)[0]
        assert torch.equal(alone, ys[0][at:at + rows[i]])
