"""The adapter path as a serving program drives it: decode steps replayed from captured graphs, eager steps that mix
prompts and decoding sequences, the FP8 and bf16 one-kernel layers, adapters moving between GPU slots and being
loaded. Sizes are those of the repository's configurations (hidden 4096 / intermediate 12288, hidden 5120 /
intermediate 17408, ranks 8 to 128) and generic ones around them.

A case is one of five kinds:

  graph   a decoding step: sequences of one token each, replayed from graphs.LoraGraphSet (one captured graph per
          batch bucket), with the slot uploads the scheduler queued for the step, if any
  step    an eager step over several layers: tile words, grouping, then every layer's adapter term
  fp8     one FP8 layer: row quantisation, shrink, base product with the adapter term
  bf16    the layers of one block in the one-kernel form: shrink, then base product with the adapter term
  load    an adapter is laid out for the GPU from its f32 factors, registered and uploaded; the one it replaces leaves

`seqs` is the tokens of every sequence of the step: comma-separated counts, "NxM" for N sequences of M tokens.
`ranks` cycles over the adapters. Adapter 0 is the most popular one; how many sequences each adapter has is a
function of the case alone, which sequence gets which is drawn from the seed.
"""
import random

import numpy as np
import torch

import __graft_entry__ as entry

pe = entry.load_package()
from pocket_engine_b200 import graphs, workloads  # noqa: E402

DEV = "cuda:0"
MAX_SEQS = 256  # sequences a serving program is set up for


def listed():
    return [
        # one user chatting: a single token per step through four decoder layers; latency and launches
        dict(name="decode-1", kind="graph", hidden=4096, inter=12288, kv=1024, layers=4, adapters=4, ranks="16",
             seqs="1x1", base=0, popular="even", swaps=0),
        # a small odd batch over adapters of several ranks, two of which the step first brings into GPU slots
        dict(name="decode-13-swap", kind="graph", hidden=4096, inter=12288, kv=1024, layers=4, adapters=8,
             ranks="8,16,32", seqs="13x1", base=2, popular="even", swaps=2),
        # the benchmark's decode mixed batch (64 tokens, 16 rank-16 adapters, a quarter base only), four decoder layers
        dict(name="decode-64", kind="graph", hidden=4096, inter=12288, kv=1024, layers=4, adapters=16, ranks="16",
             seqs="64x1", base=16, popular="even", swaps=0),
        # a full batch over adapters of very different ranks, some far more popular than others
        dict(name="decode-256-hetero", kind="graph", hidden=4096, inter=12288, kv=1024, layers=1, adapters=48,
             ranks="8,16,32,64,128", seqs="256x1", base=26, popular="zipf", swaps=0),
        # one short prompt of one adapter, eager: the first token's latency
        dict(name="prompt-199", kind="step", hidden=4096, inter=12288, kv=1024, layers=2, adapters=1, ranks="16",
             seqs="199", base=0, popular="even", form="apply", f32=False, meta="host"),
        # half prompt chunks, half decoding sequences over the wide layer set (512 tokens, 32 rank-32 adapters)
        dict(name="mixed-512", kind="step", hidden=5120, inter=17408, kv=1024, layers=1, adapters=32, ranks="32",
             seqs="256x1,128,128", base=0, popular="even", form="apply", f32=False, meta="device"),
        # ragged prompts and decoding sequences in the engine's shrink-before / expand-after order, f32 outputs
        dict(name="ragged-bracket-f32", kind="step", hidden=4096, inter=12288, kv=1024, layers=1, adapters=8,
             ranks="16,40,64", seqs="701,1,1,37,1,190,64,1,333,17,1,1,63,1,1,129", base=3, popular="even",
             form="bracket", f32=True, meta="host"),
        # the benchmark's prefill step: eight prompts of 2048 tokens, one rank-64 adapter each
        dict(name="prefill-8x2048", kind="step", hidden=4096, inter=12288, kv=1024, layers=1, adapters=8, ranks="64",
             seqs="8x2048", base=0, popular="even", form="apply", f32=False, meta="device"),
        # the benchmark's FP8 gate + up layer under 256 decoding tokens of many adapters
        dict(name="fp8-256-hetero", kind="fp8", hidden=4096, width=12288, parts=2, adapters=64,
             ranks="8,16,32,64,128", seqs="256x1", base=26, popular="zipf", f32=False),
        # the FP8 layer at a prefill-sized step
        dict(name="fp8-8x2048", kind="fp8", hidden=4096, width=12288, parts=1, adapters=8, ranks="64",
             seqs="8x2048", base=0, popular="even", f32=False),
        # a block's bf16 layers with the adapter term in the same kernel, prompts and a few decoding sequences
        dict(name="bf16-layers-mixed", kind="bf16", hidden=4096, inter=12288, kv=1024, layers=1, adapters=8,
             ranks="16,64", seqs="6x2048,1500,48x1,1041", base=4, popular="even", f32=False),
        # an adapter of an eight-layer model arrives while the program runs and replaces another
        dict(name="load-adapter", kind="load", hidden=4096, inter=12288, kv=1024, layers=8, adapters=1, ranks="16"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _shape(rng, step=64, most=5120):
    hidden = step * _log(rng, 1024 // step, most // step)
    return dict(hidden=hidden, inter=256 * max(hidden // 256, min(68, int(hidden * rng.uniform(2.0, 3.5)) // 256)),
                kv=256 * rng.randint(1, 4))


def _ranks(rng, most=128):
    pick = [r for r in (8, 16, 24, 32, 40, 64, 96, 128) if r <= most]
    return ",".join(str(r) for r in sorted(rng.sample(pick, rng.randint(1, min(3, len(pick))))))


def draw(rng):
    kind = rng.choice(["graph", "graph", "graph", "step", "step", "step", "fp8", "fp8", "bf16", "load"])
    popular = rng.choice(["even", "zipf"])
    if kind == "graph":
        n = _log(rng, 1, MAX_SEQS)
        adapters = min(48, _log(rng, 1, max(2, n)))
        return dict(_shape(rng), kind=kind, layers=rng.randint(1, 2 if adapters > 16 else 4), adapters=adapters,
                    ranks=_ranks(rng, 128 if adapters <= 24 else 64), seqs="%dx1" % n, base=int(n * rng.uniform(0, 0.4)),
                    popular=popular, swaps=rng.choice([0, 0, 1, 2]) if adapters > 2 else 0)
    if kind == "load":
        return dict(_shape(rng), kind=kind, layers=rng.randint(1, 8), adapters=1, ranks=str(rng.choice([8, 16, 32, 64])))
    prompts = [_log(rng, 2, 2048) for _ in range(rng.randint(1, 6 if kind == "bf16" else 8))]
    decode = rng.choice([0, 1, _log(rng, 1, 200)])
    seqs = ",".join(["%d" % p for p in prompts] + (["%dx1" % decode] if decode else []))
    n = len(prompts) + decode
    out = dict(kind=kind, adapters=min(24, _log(rng, 1, n + 1)), ranks=_ranks(rng), seqs=seqs,
               base=int(n * rng.choice([0, 0, rng.uniform(0, 0.4)])), popular=popular, f32=rng.random() < 0.25)
    if kind == "step":
        out.update(_shape(rng), layers=rng.randint(1, 2), form=rng.choice(["apply", "apply", "bracket"]),
                   meta=rng.choice(["host", "device"]))
    elif kind == "bf16":
        out.update(_shape(rng, 256, 4096), layers=1)  # (parts of a one-kernel layer start at multiples of 256 columns)
    else:
        out.update(hidden=128 * _log(rng, 8, 40), width=256 * _log(rng, 4, 64), parts=rng.randint(1, 2))
        if out["hidden"] * out["width"] * out["parts"] > 5120 * 24576:
            out["parts"] = 1
        if rng.random() < 0.4:
            n = _log(rng, 1, MAX_SEQS)
            out.update(seqs="%dx1" % n, base=int(n * rng.uniform(0, 0.3)))
    return out


# ------------------------------------------------------------------------------- shapes and assignment

def _sites(case):
    if case["kind"] == "fp8":
        mods = [("mlp.gate_proj", case["width"]), ("mlp.up_proj", case["width"])][:case["parts"]]
        return [pe.Site.fused(0, case["hidden"], mods)]
    out = []
    for layer in range(case["layers"]):
        out += workloads.block_sites(case["hidden"], case["inter"], case["kv"], layer)
    return out


def _rows(case):
    rows = []
    for piece in case["seqs"].split(","):
        n, _, m = piece.partition("x")
        rows += [int(m)] * int(n) if m else [int(n)]
    return np.array(rows, np.int32)


def _rank(case, i):
    r = [int(v) for v in case["ranks"].split(",")]
    return r[i % len(r)]


def _assignment(case):
    """The adapter of every sequence, -1 for base only: the longest sequences first, popularity as the case says. The
    base-only sequences are the shortest ones."""
    rows = _rows(case)
    order = np.argsort(-rows, kind="stable")
    n_ad, live = case["adapters"], len(rows) - case["base"]
    which = np.full(len(rows), -1, np.int64)
    if case["popular"] == "even":
        which[order[:live]] = np.arange(live) % n_ad
    else:  # Zipf(1.1) shares, every sequence to the adapter furthest behind its share
        share = 1.0 / np.arange(1, n_ad + 1) ** 1.1
        share /= share.sum()
        got = np.zeros(n_ad)
        for k, s in enumerate(order[:live]):
            a = int(np.argmax(share * (k + 1) - got))
            which[s] = a
            got[a] += 1
    return rows, which


def work(case):
    sites = _sites(case)
    if case["kind"] == "load":
        values = sum(_rank(case, 0) * (len(s.parts) * s.cols + sum(p.rows for p in s.parts)) for s in sites)
        return {"bytes": 4 * values + 2 * values + 2 * values, "flops": 0}  # f32 factors in, the slab on both sides
    rows, which = _assignment(case)
    present = sorted(set(int(a) for a in which if a >= 0))
    tokens = {a: int(rows[which == a].sum()) for a in present}
    t_all, t_lora = int(rows.sum()), sum(tokens.values())
    y_el = 4 if case.get("f32") else 2
    by = fl = 0
    for s in sites:
        parts, width = len(s.parts), sum(p.rows for p in s.parts)
        for a in present:
            r = _rank(case, a)
            by += 2 * r * (parts * s.cols + width)
            fl += 2 * tokens[a] * r * (parts * s.cols + width)
        if case["kind"] == "fp8":  # x, e4m3 W and its scales, y once
            by += 2 * t_all * s.cols + s.cols * width + 4 * width + y_el * t_all * width
            fl += 2 * t_all * s.cols * width
        elif case["kind"] == "bf16":
            by += 2 * t_all * s.cols + 2 * s.cols * width + y_el * t_all * width
            fl += 2 * t_all * s.cols * width
        else:  # y is read and written
            by += 2 * t_lora * s.cols + 2 * y_el * t_lora * width
    if case.get("swaps"):  # the slabs that change slots, read on the host and written on the device
        for a in range(case["swaps"]):
            by += 2 * sum(2 * _rank(case, a) * (len(s.parts) * s.cols + sum(p.rows for p in s.parts)) for s in sites)
    return {"bytes": by, "flops": fl}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"
    if case.get("f32"):
        # f32 sums of bf16 products: accumulation order, and about 16 bits of the intermediate on the tensor cores
        return {"rel": 3e-5, "max": 5e-4}
    # bf16 results of f32 sums: a value near a rounding boundary may go to its neighbour
    return {"rel": 5e-3, "max": 2e-2}


# ------------------------------------------------------------------------------- state

class _Device:
    """Device memory of a registry as a tensor (CUDA array interface); the registry lives as long as the tensor."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (int(ptr), False), "version": 2,
                                         "strides": None}


def _factors(case, sites, adapters, gen):
    """f32 factors N(0, 0.02^2) of every adapter: views of one random pool, each module at an offset of its own."""
    need = max(_rank(case, i) for i in range(adapters)) * max(max(s.cols, p.rows) for s in sites for p in s.parts)
    pool = (torch.randn(2 * need + (1 << 20), device=DEV, generator=gen) * 0.02).cpu().numpy()
    at = random.Random(int(torch.randint(1 << 30, (1,), device=DEV, generator=gen)))

    def view(n, m):
        o = at.randrange(len(pool) - n * m)
        return pool[o:o + n * m].reshape(n, m)

    return [[pe.Factors(s.layer, p.module, view(_rank(case, i), s.cols), view(p.rows, _rank(case, i)))
             for s in sites for p in s.parts] for i in range(adapters)]


def _registry(case, sites, tokens, seqs, gen):
    adapters = case["adapters"]
    most = max(_rank(case, i) for i in range(adapters))
    L = pe.Loras(sites, adapters, most, tokens, seqs, device=0)
    prep = L.prep()
    ids = [L.insert(prep.prepare("adapter-%d" % i, f)) for i, f in enumerate(_factors(case, sites, adapters, gen))]
    return L, ids


_streams = []


def _decode_stream():
    """The one stream a serving program runs its decoding steps on, whichever of its states a step uses."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _rand(gen, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device=DEV, generator=gen, dtype=torch.float32).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.default_rng(seed)
    sites = _sites(case)
    if case["kind"] == "load":
        L = pe.Loras(sites, 1, _rank(case, 0), 64, device=0)
        factors = _factors(case, sites, 1, gen)[0]
        prep = L.prep()
        first = prep.prepare("adapter", factors)
        n = first.len
        L.upload(1, L.insert(first))
        slab = torch.as_tensor(_Device(L, L.pool, n), device=DEV)
        return dict(case=case, L=L, prep=prep, factors=factors, slab=slab)
    rows, which = _assignment(case)
    # which sequence of a length runs which adapter, and which slot an adapter sits in, come from the seed
    for n in set(rows.tolist()):
        at = np.nonzero(rows == n)[0]
        which[at] = which[rng.permutation(at)]
    slot_of = np.concatenate([rng.permutation(case["adapters"]) + 1, [0]]).astype(np.int32)  # [-1] is base only
    row_slot = slot_of[which]
    tokens = int(rows.sum())
    f32 = bool(case.get("f32"))
    room = MAX_SEQS if case["kind"] == "graph" else tokens
    L, ids = _registry(case, sites, room, MAX_SEQS if case["kind"] == "graph" else len(rows), gen)
    for i, a in enumerate(ids):
        L.upload(int(slot_of[i]), a)
    xs = [_rand(gen, room, s.cols) for s in sites]
    ys = [_rand(gen, room, s.width(), dtype=torch.float32 if f32 else torch.bfloat16) for s in sites]
    lins = [pe.Linear(L, si) for si in range(len(sites))]
    st = dict(case=case, L=L, rows=rows, row_slot=row_slot, tokens=tokens, f32=f32, xs=xs, ys=ys, lins=lins,
              tiles=L.max_lora_tiles(), decode=int(rows.max()) == 1)
    st["cu"] = torch.from_numpy(np.concatenate([[0], np.cumsum(rows)]).astype(np.int32)).to(DEV)
    st["slots"] = torch.from_numpy(row_slot.copy()).to(DEV)
    if case["kind"] == "graph":
        stream = _decode_stream()

        def body(step, n, s):
            for x, y, lin in zip(xs, ys, lins):
                lin.forward(x.data_ptr(), n, y.data_ptr(), y.shape[1], f32, lora=step, main=s, fused=True)

        torch.cuda.synchronize()
        ybase = [y.clone() for y in ys]
        st["graphs"] = graphs.LoraGraphSet(L, body, MAX_SEQS, stream)
        for y, b in zip(ys, ybase):
            y.copy_(b)
        st["loads"] = [(int(slot_of[i]), ids[i]) for i in range(case["swaps"])]
        st["stream"] = stream
        st["out"] = [y[:tokens] for y in ys]
        torch.cuda.synchronize()
    elif case["kind"] == "fp8":
        k, n = sites[0].cols, sites[0].width()
        st["wq"] = _rand(gen, n, k, dtype=torch.float8_e4m3fn).view(torch.uint8)
        st["sn"] = (torch.rand(n, device=DEV, generator=gen) * 1.5 + 0.5) / 448.0
        st["xq"] = torch.empty(tokens, k, dtype=torch.uint8, device=DEV)
        st["st"] = torch.empty(tokens, dtype=torch.float32, device=DEV)
    elif case["kind"] == "bf16":
        st["ws"] = [_rand(gen, s.width(), s.cols) * s.cols ** -0.5 for s in sites]
    return st


# ------------------------------------------------------------------------------- one pass

def run(st):
    return {"graph": _run_graph, "step": _run_step, "fp8": _run_fp8, "bf16": _run_bf16, "load": _run_load}[
        st["case"]["kind"]](st)


def _run_graph(st):
    L, s = st["L"], st["stream"].cuda_stream
    for slot, adapter in st["loads"]:
        L.upload(slot, adapter, s)
    words = pe.fill_tiles(st["rows"], st["row_slot"], st["tiles"])
    st["graphs"].replay(st["tokens"], words)
    return st["out"]


def _begin(st, s):
    """The step's metadata: tile words from the host, or from the sequence table on the device; then the grouping."""
    L = st["L"]
    if st["case"].get("meta") == "host":
        L.meta_upload(pe.fill_tiles(st["rows"], st["row_slot"], st["tiles"]), s)
    else:
        L.meta_build(st["cu"].data_ptr(), st["slots"].data_ptr(), len(st["rows"]), s)
    return L.lora_step(st["tiles"], s, decode=st["decode"])


def _run_step(st):
    s = torch.cuda.current_stream().cuda_stream
    step = _begin(st, s)
    fused = st["case"]["form"] == "apply"
    for x, y, lin in zip(st["xs"], st["ys"], st["lins"]):
        lin.forward(x.data_ptr(), st["tokens"], y.data_ptr(), y.shape[1], st["f32"], lora=step, main=s, fused=fused)
    return st["ys"]


def _run_fp8(st):
    s = torch.cuda.current_stream().cuda_stream
    L, hook, x, y, t = st["L"], st["lins"][0].lora, st["xs"][0], st["ys"][0], st["tokens"]
    step = _begin(st, s)
    L.fp8_quant_rows(x.data_ptr(), t, x.shape[1], st["xq"].data_ptr(), st["st"].data_ptr(), s)
    L.shrink(hook, step, x.data_ptr(), t, s)
    L.linear_fp8_fused(hook, step, st["xq"].data_ptr(), st["st"].data_ptr(), st["wq"].data_ptr(), st["sn"].data_ptr(), t,
                       y.data_ptr(), y.shape[1], st["f32"], s)
    return [y, st["xq"], st["st"]]


def _run_bf16(st):
    s = torch.cuda.current_stream().cuda_stream
    L, t = st["L"], st["tokens"]
    step = _begin(st, s)
    for x, w, y, lin in zip(st["xs"], st["ws"], st["ys"], st["lins"]):
        L.shrink(lin.lora, step, x.data_ptr(), t, s)
        L.linear_bf16_fused(lin.lora, step, x.data_ptr(), w.data_ptr(), t, y.data_ptr(), y.shape[1], st["f32"], s)
    return st["ys"]


def _run_load(st):
    s = torch.cuda.current_stream().cuda_stream
    L = st["L"]
    old = L.retire("adapter")
    new = L.insert(st["prep"].prepare("adapter", st["factors"]))
    L.upload(1, new, s)
    L.free(old)
    return st["slab"]
