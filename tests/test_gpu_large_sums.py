"""Sums of the shrink at and past the end of the bf16 range, which the few-token expand splits into bf16 terms: what an f32
product chain gives, infinities with their sign included."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [False, "early"], ids=["bracket", "pair"])
@pytest.mark.parametrize("rank,tokens", [(16, 3), (64, 12), (160, 3)])
def test_sums_past_the_bf16_range(pe, rank, tokens, form):
    import torch
    cols, width = 64, 80
    site = pe.Site.fused(0, cols, [("a", width)])
    a, b = np.zeros((rank, cols), np.float32), np.zeros((width, rank), np.float32)
    a[0, :2] = 1.0
    b[:, 0] = np.where(np.arange(width) % 3 == 0, -1, 1) * 2.0 ** -100
    x = np.zeros((tokens, cols), np.float32)
    x[:, 0] = 1.5
    x[0, :2] = 3.38953139e38, 1e36      # a finite f32 whose nearest bf16 is infinite
    x[1, :2] = 3e38, 3e38               # an infinite one
    x[2, :2] = -3e38, -3e38
    loras = pe.Loras([site], 1, rank, tokens, tokens, device=0)
    loras.upload(1, loras.insert(loras.prep().prepare("a", [pe.Factors(0, "a", a, b)])))
    xd = torch.from_numpy(x).bfloat16().cuda()
    y = torch.zeros(tokens, width, device="cuda")
    loras.meta_upload(pe.fill_tiles(np.ones(tokens, np.int32), np.ones(tokens, np.int32), loras.max_lora_tiles()))
    step = loras.lora_step(loras.max_lora_tiles())
    loras.set_apply_mode(0)
    pe.Linear(loras, 0).forward(xd.data_ptr(), tokens, y.data_ptr(), width, True, lora=step, main=torch.cuda.current_stream().cuda_stream, fused=bool(form))
    torch.cuda.synchronize()
    loras.device_status()
    s = (xd[:, 0] .float() + xd[:, 1].float()).cpu().numpy()
    with np.errstate(over="ignore"):
        want = s[:, None] * b[:, 0][None, :]
    assert np.isinf(want[1]).all() and np.isinf(want[2]).all() and np.isfinite(want[0]).all()
    got = y.cpu().numpy()
    assert np.array_equal(np.isinf(want), np.isinf(got)) and np.array_equal(np.sign(want), np.sign(got))
    fin = np.isfinite(want)
    assert np.allclose(got[fin], want[fin], rtol=1e-6, atol=0)
    loras.close()
