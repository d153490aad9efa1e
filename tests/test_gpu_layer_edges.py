"""The one-kernel layers and the row quantisation at the edges of their tiles: both tile widths, steps that end inside a
tile or fill several rounds of block pairs, many runs and ranks over one tile, rows of every length a thread holds."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [8, 264, 512, 4096, 4104, 8192, 8200])
def test_row_quantisation_of_every_row_length(pe, oracle, cols):
    import torch
    rng = np.random.default_rng(cols)
    scale = np.array([1, 1e-3, 30, 1e-36, 3e38, 0], np.float32)[np.arange(19) % 6][:, None]
    x = np.clip(rng.standard_normal((19, cols), dtype=np.float32), -1, 1) * scale
    x[:, ::7] *= np.float32(2.0 ** -9)  # quotients below the normal range of e4m3
    xb = pe.bf16_bits(x).reshape(x.shape)
    loras = pe.Loras([pe.Site.fused(0, cols, [("a", 64)])], 1, 16, 32, device=0)
    xd = harness.to_dev_bf16(xb, 0)
    xq = torch.zeros(19, cols, dtype=torch.uint8, device="cuda")
    st = torch.zeros(19, dtype=torch.float32, device="cuda")
    loras.fp8_quant_rows(xd.data_ptr(), 19, cols, xq.data_ptr(), st.data_ptr())
    torch.cuda.synchronize()
    want_q, want_s = oracle.fp8_quant_rows(xb)
    assert np.array_equal(st.cpu().numpy(), want_s)
    assert np.array_equal(xq.cpu().numpy(), want_q)
    loras.close()


def test_row_quantisation_of_every_mantissa(pe, oracle):
    """Every eight-bit mantissa of an input under every one of a row's maximum, at three scales; inputs of all exponents that
    give a normal, a subnormal and a zero e4m3."""
    import torch
    x = np.zeros((3 * 128, 128 * 20 + 8), np.float32)
    m = (128 + np.arange(128, dtype=np.float32)) / 128
    for i, scale in enumerate([1.0, 2.0 ** 40, 2.0 ** -40]):
        for k in range(128):
            row = np.concatenate([m * np.float32(2.0 ** -e) for e in range(1, 21)]).astype(np.float32)
            row[1::2] *= -1
            x[128 * i + k, :len(row)] = row * np.float32(scale)
            x[128 * i + k, -1] = m[k] * np.float32(scale)  # the maximum
    xb = pe.bf16_bits(x).reshape(x.shape)
    loras = pe.Loras([pe.Site.fused(0, x.shape[1], [("a", 64)])], 1, 16, 384, device=0)
    xd = harness.to_dev_bf16(xb, 0)
    xq = torch.zeros(x.shape, dtype=torch.uint8, device="cuda")
    st = torch.zeros(len(x), dtype=torch.float32, device="cuda")
    loras.fp8_quant_rows(xd.data_ptr(), len(x), x.shape[1], xq.data_ptr(), st.data_ptr())
    torch.cuda.synchronize()
    want_q, want_s = oracle.fp8_quant_rows(xb)
    assert np.array_equal(st.cpu().numpy(), want_s)
    assert np.array_equal(xq.cpu().numpy(), want_q)
    loras.close()


LAYERS = [
    # name, rows of the sequences, ranks, input width, part widths
    ("one-row", [1], [16], 64, [256]),
    ("ends-inside-a-tile", [300, 5], [16, 64], 264, [256, 200]),
    ("many-runs-over-one-tile", [65, 66, 129, 64, 70, 64, 131], [128, 96, 16], 512, [520]),
    ("several-rounds-of-pairs", [2048, 1], [32], 128, [4096]),
    ("narrow-tiles", [256], [64], 192, [9984]),
]


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
def test_bf16_layer_edges(pe, case, f32_out):
    import torch
    from pocket_engine_b200 import workloads
    name, rows, ranks, cols, widths = case
    slots = [1 + i % len(ranks) for i in range(len(rows))]
    wl = workloads.Workload(name, [pe.Site.fused(0, cols, [("p%d" % i, w) for i, w in enumerate(widths)])], ranks, 1.0, rows, slots, 23)
    table, _ = harness.oracle_registry(wl)
    loras = harness.product_registry(pe, wl)
    g = torch.Generator(device="cuda").manual_seed(3)
    w = (torch.randn(wl.sites[0].width(), cols, device="cuda", generator=g) / cols ** 0.5).bfloat16()
    x = harness.to_dev_bf16(wl.x_bits(0), 0)
    base = (x.double() @ w.double().t()).cpu().numpy()
    want = harness.oracle_f64(wl, table, harness.tiles_of(pe, wl), y_base=[base.astype(np.float32)])[0]
    y = torch.full((wl.tokens, wl.sites[0].width()), float("nan"), dtype=torch.float32 if f32_out else torch.bfloat16, device="cuda")
    first = torch.empty_like(y)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    step = loras.lora_step(loras.max_lora_tiles())
    for out in (first, y):  # the second pass finds its barriers and accumulators as the first one left them
        loras.shrink(loras.hook(0), step, x.data_ptr(), wl.tokens)
        loras.linear_bf16_fused(loras.hook(0), step, x.data_ptr(), w.data_ptr(), wl.tokens, out.data_ptr(), y.shape[1], f32_out)
    torch.cuda.synchronize()
    loras.device_status()
    assert torch.equal(first, y)
    got = y.float().cpu().numpy()
    mx, mn = harness.tolerance(got, want)
    assert (mx <= 1e-3 and mn <= 1e-4) if f32_out else (mx <= 4e-2 and mn <= 4e-3), (mx, mn)
    loras.close()


@pytest.mark.parametrize("f32_out", [True, False])
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
@pytest.mark.parametrize("rows,widths", [([1], [19456]), ([70], [9728, 9720]), ([100, 1, 27], [28416]), ([128], [14336, 14344]), ([1] * 65, [37896]),
                                          ([60, 60, 50, 31], [9728, 9720]), ([200, 56], [512, 1000])])
def test_few_tokens_over_a_wide_layer(pe, kind, rows, widths, f32_out):
    """Blocks on their own, with tiles of 192 and of 256 columns, in one round and in more; pairs with tiles of 192 that span parts."""
    import torch
    from pocket_engine_b200 import workloads
    cols = 272 if kind == "fp8" else 264
    wl = workloads.Workload("wide", [pe.Site.fused(0, cols, [("p%d" % i, w) for i, w in enumerate(widths)])], [16, 40], 1.0, rows,
                            [1 + i % 2 for i in range(len(rows))], 41)
    table, _ = harness.oracle_registry(wl)
    loras = harness.product_registry(pe, wl)
    T, N = wl.tokens, wl.sites[0].width()
    g = torch.Generator(device="cuda").manual_seed(5)
    x = harness.to_dev_bf16(wl.x_bits(0), 0)
    w = torch.randn(N, cols, device="cuda", generator=g) / cols ** 0.5
    if kind == "fp8":
        w, xq = w.to(torch.float8_e4m3fn), x.float().to(torch.float8_e4m3fn)
        st = 0.9 + 0.2 * torch.rand(T, device="cuda", generator=g)
        sn = 0.9 + 0.2 * torch.rand(N, device="cuda", generator=g)
        base = (xq.float().double() @ w.float().double().t()) * st.double()[:, None] * sn.double()
    else:
        w = w.bfloat16()
        base = x.double() @ w.double().t()
    want = harness.oracle_f64(wl, table, harness.tiles_of(pe, wl), y_base=[base.cpu().numpy().astype(np.float32)])[0]
    y = torch.full((T, N), float("nan"), dtype=torch.float32 if f32_out else torch.bfloat16, device="cuda")
    loras.set_run_min(1 << 30)  # (a step without long runs; only those take these tiles)
    loras.meta_upload(harness.tiles_of(pe, wl, loras.max_lora_tiles()))
    step = loras.lora_step(loras.max_lora_tiles())
    for _ in range(2):
        loras.shrink(loras.hook(0), step, x.data_ptr(), T)
        if kind == "fp8":
            loras.linear_fp8_fused(loras.hook(0), step, xq.data_ptr(), st.data_ptr(), w.data_ptr(), sn.data_ptr(), T, y.data_ptr(), N, f32_out)
        else:
            loras.linear_bf16_fused(loras.hook(0), step, x.data_ptr(), w.data_ptr(), T, y.data_ptr(), N, f32_out)
    torch.cuda.synchronize()
    loras.device_status()
    got = y.float().cpu().numpy()
    mx, mn = harness.tolerance(got, want)
    assert (mx <= 1e-3 and mn <= 1e-4) if f32_out else (mx <= 4e-2 and mn <= 4e-3), (mx, mn)
    loras.close()
