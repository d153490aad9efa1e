"""Row quantisation of so many rows that a warp takes each (widths up to 2048 and from 3592 to 5120; a block each beyond and between): every
number of pieces a lane may hold, rows that end inside a lane's pieces, an odd number of rows, rows at the edge of the f32 range, all
zeros, infinities and no numbers."""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [8, 264, 2048, 2056, 3592, 4096, 4104, 5120, 5128])
def test_many_rows(pe, oracle, cols):
    import torch
    n = 48 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    rng = np.random.default_rng(cols)
    scale = np.array([1, 1e-3, 30, 1e-36, 3e38, 0, 1e-19], np.float32)[np.arange(n) % 7][:, None]
    x = np.clip(rng.standard_normal((n, cols), dtype=np.float32), -1, 1) * scale
    x[:, ::7] *= np.float32(2.0 ** -9)
    x[5::11, 3] = -0.0
    xb = pe.bf16_bits(x).reshape(x.shape)
    loras = pe.Loras([pe.Site.fused(0, cols, [("a", 64)])], 1, 16, 2048, device=0)

    def run(bits):
        xd = harness.to_dev_bf16(bits, 0)
        xq = torch.zeros(bits.shape, dtype=torch.uint8, device="cuda")
        st = torch.zeros(len(bits), dtype=torch.float32, device="cuda")
        loras.fp8_quant_rows(xd.data_ptr(), len(bits), cols, xq.data_ptr(), st.data_ptr())
        torch.cuda.synchronize()
        return xq.cpu().numpy(), st.cpu().numpy()

    got_q, got_s = run(xb)
    want_q, want_s = oracle.fp8_quant_rows(xb)
    assert np.array_equal(got_s, want_s)
    assert np.array_equal(got_q, want_q)
    # rows with infinities and no numbers: what a step of few rows, a block per row, makes of them
    odd = xb.copy()
    odd[::3, 1] = 0x7f80
    odd[1::3, 2] = 0x7fc1
    odd[2::3, :] = 0xffc0
    many_q, many_s = run(odd)
    few = [run(odd[i:i + 500]) for i in range(0, n, 500)]
    assert np.array_equal(many_q, np.concatenate([f[0] for f in few]))
    assert np.array_equal(many_s, np.concatenate([f[1] for f in few]), equal_nan=True)
    loras.close()
