"""Slabs that are filled by several threads, and pinned buffers that pass from one adapter to the next."""
import numpy as np
import pytest

import harness


def _sites(pe):
    # stretches below and above the size one thread takes at a time, an odd number of rows per stretch
    return [pe.Site.fused(0, 4104, [("q", 4100), ("k", 130)]), pe.Site.fused(0, 64, [("o", 20002)])]


@pytest.mark.parametrize("ranks", [(8, 40), (16, 16), (33, 1)])
def test_slab_bytes_equal_the_oracles(pe, oracle, ranks):
    from pocket_engine_b200 import workloads
    wl = workloads.Workload("slabs", _sites(pe), list(ranks), 2.0, [1], [0], 3)
    loras = pe.Loras(wl.sites, 2, wl.max_rank, 16, device=-1)
    for i in range(2):
        f = wl.factors(i)
        f[0].a[0, 5], f[0].a[0, 6], f[0].b[1, 0] = np.nan, np.inf, -0.0
        got = loras.prep().prepare(f"a{i}", f)
        assert np.array_equal(got.bytes(), oracle.OracleAdapter(wl.sites, f, wl.max_rank).data[:got.len])
        got.drop()
    loras.close()


@pytest.mark.gpu
def test_reused_buffers_reach_the_slots_intact(pe):
    import torch
    from pocket_engine_b200 import workloads
    sites = _sites(pe)
    loras = pe.Loras(sites, 3, 48, 16, device=0)
    prep = loras.prep()
    streams = [torch.cuda.Stream() for _ in range(2)]
    want = {}
    for k in range(12):  # every adapter leaves right behind its upload, so its buffer is wanted while the copy runs
        wl = workloads.Workload("slabs", sites, [(8, 16, 48)[k % 3]], 1.0, [1], [0], k)
        ad = prep.prepare("a", wl.factors(0))
        slot, data = 1 + k % 3, ad.bytes()
        if slot in want:
            torch.cuda.synchronize()  # (the slot's previous content was checked when it was written)
        aid = loras.insert(ad)
        for s in streams[:1 + k % 2]:  # odd ones go to the slot twice, from two streams
            loras.upload(slot, aid, s.cuda_stream)
        loras.retire("a")
        loras.free(aid)
        want[slot] = data
        if k % 3 == 2:
            torch.cuda.synchronize()
            for s, d in want.items():
                assert np.array_equal(harness.dev_read(loras.pool + (s - 1) * loras.slot_bytes, len(d)), d), (k, s)
    loras.close()
