"""The work this package is used for, as cases to be timed.

Each case is one call (or the few calls that belong together) of the public entry points on the GPU:

  decode    fused attention of one new token per sequence over the compressed cache (fp16 or 2-/4-bit codes)
  prefill   prune + compression of a prompt's K and V into the arenas the decode path reads
  append    the 256 oldest window tokens of every sequence joining the compressed cache during decode
  convert   the reference-shaped compression of already pruned K and V (model prefill through the module names
            that ``compat.install()`` registers)
  ops       the reference-shaped pair of products over a compact compressed cache (q.K^T, P.V)
  step      what runs in one decoder layer per token besides the GEMMs: norm, RoPE + window append (with or without
            the per-step prune), attention with device-resident lengths, residual add + norm, SiLU * up

Inputs are synthetic with the statistics of the benchmark: K and V ~ N(0, 1), four K channels per head ten times
larger, per-token magnitude pruning at 50-80 %.
"""
import math

import torch

from mustafar_b200 import compression as comp
from mustafar_b200 import compression_quant as cq
from mustafar_b200 import ops, ops_quant, step_ops

D = 128
DEV = "cuda"


def listed():
    return [
        # one sequence, 4k context: the interactive single-user call; latency and host time count
        dict(name="decode b1 4k", what="decode", batch=1, kv_heads=8, group=4, tokens=4096, window=128, sparsity=0.7, bits=16,
             qgroup=64),
        # a handful of sequences of an odd length, 8 query heads per kv head, half of the values kept, ragged window
        dict(name="decode b7 10k g8", what="decode", batch=7, kv_heads=8, group=8, tokens=10176, window=217, sparsity=0.5,
             bits=16, qgroup=64),
        # the benchmark's headline: a full serving batch at 32k context
        dict(name="decode b64 32k", what="decode", batch=64, kv_heads=8, group=4, tokens=32768, window=128, sparsity=0.7, bits=16,
             qgroup=64),
        # the quantised model's cache (2-bit codes, one scale per tile) under a serving batch
        dict(name="decode 2-bit b32 16k", what="decode", batch=32, kv_heads=8, group=4, tokens=16384, window=128, sparsity=0.7,
             bits=2, qgroup=64),
        # 4-bit codes with a scale per 32 nonzeros, smaller batch
        dict(name="decode 4-bit b8 4k g32", what="decode", batch=8, kv_heads=8, group=4, tokens=4096, window=128, sparsity=0.5,
             bits=4, qgroup=32),
        # a layer's prompt of 8 sequences x 8k tokens going into the fp16 arenas
        dict(name="prefill b8 8k", what="prefill", batch=8, kv_heads=8, tokens=8192, sparsity=0.7, bits=16),
        # the same for the quantised cache, an odd prompt length
        dict(name="prefill 2-bit b4 5k", what="prefill", batch=4, kv_heads=8, tokens=4928, sparsity=0.7, bits=2),
        # every 256 decode steps: one block of every sequence moves from the window to the cache
        dict(name="append b32 at 4k", what="append", batch=32, kv_heads=8, tokens=4096, sparsity=0.7),
        # the reference's own model code at prefill: one prompt, already pruned tensors, lists of packed values back
        dict(name="convert b1 3k", what="convert", heads=8, tokens=3840, sparsity=0.7),
        # the reference's own model code at decode: the two products with 8-row padded operands
        dict(name="ops b8 16k", what="ops", batch=8, kv_heads=8, group=4, tokens=16384, sparsity=0.7, bits=16),
        # ... and its quantised counterpart at a moderate length
        dict(name="ops 2-bit b4 7k", what="ops", batch=4, kv_heads=8, group=4, tokens=6912, sparsity=0.7, bits=2),
        # the non-GEMM launches of one layer of a decode step, small batch: launches and host time count
        dict(name="step b4 2k", what="step", batch=4, kv_heads=8, group=4, tokens=2048, window=201, sparsity=0.7,
             hidden=4096, ffn=14336, prune=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tokens(rng, lo, hi, heads, limit):
    """A multiple of 64 (the block the formats are made of), spread over its logarithm, heads * tokens <= limit."""
    hi = max(lo, min(hi, limit // heads))
    return 64 * max(1, _log_int(rng, lo / 64, hi / 64))


def draw(rng):
    what = rng.choice(["decode", "decode", "decode", "prefill", "append", "convert", "ops", "step"])
    s = rng.choice([0.5, 0.6, 0.7, 0.8])
    if what == "decode":
        b, h, g = _log_int(rng, 1, 64), rng.choice([1, 2, 4, 8, 8]), rng.choice([1, 2, 4, 4, 8])
        bits = rng.choice([16, 16, 2, 4])
        t = _tokens(rng, 256, 32768, b * h, 1 << 22)
        return dict(what=what, batch=b, kv_heads=h, group=g, tokens=t, window=rng.randint(1, 383), sparsity=s, bits=bits,
                    qgroup=64 if bits == 16 else rng.choice([64, 32]))
    if what == "prefill":
        b, h = _log_int(rng, 1, 16), rng.choice([1, 4, 8])
        return dict(what=what, batch=b, kv_heads=h, tokens=_tokens(rng, 256, 16384, b * h, 1 << 19), sparsity=s,
                    bits=rng.choice([16, 2, 4]))
    if what == "append":
        b, h = _log_int(rng, 1, 64), rng.choice([1, 4, 8])
        return dict(what=what, batch=b, kv_heads=h, tokens=256 * max(1, _tokens(rng, 256, 8192, b * h, 1 << 20) // 256), sparsity=s)
    if what == "convert":
        h = rng.randint(1, 16)
        return dict(what=what, heads=h, tokens=_tokens(rng, 64, 8192, h, 1 << 16), sparsity=s)
    if what == "ops":
        b, h, g = _log_int(rng, 1, 16), rng.choice([1, 4, 8]), rng.choice([1, 2, 4, 8])
        return dict(what=what, batch=b, kv_heads=h, group=g, tokens=_tokens(rng, 256, 16384, b * h, 1 << 20), sparsity=s,
                    bits=rng.choice([16, 16, 2, 4]))
    h, g = rng.choice([1, 4, 8]), 4
    return dict(what=what, batch=_log_int(rng, 1, 32), kv_heads=h, group=g, tokens=256 * rng.randint(1, 16),
                window=rng.randint(130, 383), sparsity=s, hidden=rng.choice([2048, 4096, 5120]), ffn=rng.choice([5632, 11008, 14336]),
                prune=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ inputs
def _kv(gen, heads, n, scale=None):
    x = torch.randn(heads, n, D, generator=gen, device=DEV)
    return (x if scale is None else x * scale).half()


def _k_scale(gen, heads):
    """Four of the 128 channels of every K head are ten times larger."""
    ch = torch.rand(heads, D, generator=gen, device=DEV).argsort(dim=1)[:, :4]
    return torch.ones(heads, 1, D, device=DEV).scatter_(2, ch[:, None, :], 10.0)


def _stores(case, heads, max_tokens):
    bits = case.get("bits", 16)
    if bits == 16:
        cap = int(max_tokens * D * min(1.0, 1.25 - case["sparsity"])) // 8 * 8
        k, v = (comp.SparseStore(heads, max_tokens, kind, DEV, nz_capacity=cap) for kind in (comp.KEY, comp.VALUE))
        k.nz.zero_(), v.nz.zero_()            # what no value is written to stays zero
    else:
        k, v = (cq.QuantStore(heads, max_tokens, kind, DEV, bits, case.get("qgroup", 64)) for kind in (comp.KEY, comp.VALUE))
        k.packed.zero_(), v.packed.zero_()
    return k, v


def _fill(gen, case, k, v, tokens, scale):
    rank = comp.keep_rank(case["sparsity"])
    step = max(64, (1 << 27) // (k.n_heads * D) // 64 * 64)
    for t0 in range(0, tokens, step):
        n = min(step, tokens - t0)
        k.append(_kv(gen, k.n_heads, n, scale), rank)
        v.append(_kv(gen, k.n_heads, n), rank)


def _compact(store):
    """An arena's contents in the reference's compact layout: bitmaps, packed values, offsets, head offsets."""
    lens = store.packed_lengths().tolist()
    idx = store.accum.clone()
    off = torch.zeros(store.n_heads, dtype=torch.int32, device=DEV)
    off[1:] = torch.cumsum(idx[:-1, -1] // 4, dim=0).to(torch.int32)
    return store.bitmaps.clone(), torch.cat([store.nz[h, :n] for h, n in enumerate(lens)]), idx, off


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    what, sp = case["what"], case["sparsity"]
    st = dict(case=case, rank=comp.keep_rank(sp))
    if what == "decode":
        heads = case["batch"] * case["kv_heads"]
        scale = _k_scale(gen, heads)
        st["k"], st["v"] = _stores(case, heads, case["tokens"])
        _fill(gen, case, st["k"], st["v"], case["tokens"], scale)
        st["kw"], st["vw"] = _kv(gen, heads, case["window"], scale), _kv(gen, heads, case["window"])
        st["q"] = _kv(gen, heads * case["group"], 1)[:, 0]
    elif what == "prefill":
        # what a fused q|k|v projection leaves: [batch, token, kv head, 128], read in place
        b, h, t = case["batch"], case["kv_heads"], case["tokens"]
        x = torch.randn(2, b, t, h, D, generator=gen, device=DEV).half()
        x[0] *= _k_scale(gen, h).view(1, 1, h, D).half()
        st["x"] = [y.transpose(1, 2) for y in x]
        st["k"], st["v"] = _stores(case, b * h, t)
    elif what == "append":
        heads = case["batch"] * case["kv_heads"]
        scale = _k_scale(gen, heads)
        st["k"], st["v"] = _stores(case, heads, case["tokens"] + 256)
        _fill(gen, case, st["k"], st["v"], case["tokens"], scale)
        st["kw"], st["vw"] = _kv(gen, heads, 384, scale), _kv(gen, heads, 384)
    elif what == "convert":
        h, t = case["heads"], case["tokens"]
        st["x"] = [comp.prune(_kv(gen, h, t, _k_scale(gen, h)), sp), comp.prune(_kv(gen, h, t), sp)]
        st["nz"] = [torch.zeros(h * t * D, dtype=torch.float16, device=DEV) for _ in range(2)]
    elif what == "ops":
        b, h, g, t = case["batch"], case["kv_heads"], case["group"], case["tokens"]
        if case["bits"] == 16:
            k, v = _stores(case, b * h, t)
            _fill(gen, case, k, v, t, _k_scale(gen, b * h))
            st["k"], st["v"] = _compact(k), _compact(v)
        else:
            st["k"] = cq.compress_quant(_kv(gen, b * h, t, _k_scale(gen, b * h)), comp.KEY, st["rank"], case["bits"])
            st["v"] = cq.compress_quant(_kv(gen, b * h, t), comp.VALUE, st["rank"], case["bits"])
        q = _kv(gen, b * h * g, 1)
        p = torch.softmax(2 * torch.randn(b * h * g, 1, t, generator=gen, device=DEV), -1).half()
        st["q8"], st["p8"] = (torch.nn.functional.pad(y, (0, 0, 0, 7)) for y in (q, p))
        st["ws"] = torch.zeros(1, dtype=torch.float16, device=DEV)
    else:
        b, h, g, t, w = case["batch"], case["kv_heads"], case["group"], case["tokens"], case["window"]
        heads, hid, ffn = b * h, case["hidden"], case["ffn"]
        scale = _k_scale(gen, heads)
        st["k"], st["v"] = _stores(case, heads, t + 1024)       # room for blocks still to come
        _fill(gen, case, st["k"], st["v"], t, scale)
        st["kw"], st["vw"] = _kv(gen, heads, 384, scale), _kv(gen, heads, 384)
        rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV).half()  # noqa: E731
        st["embed"], st["ids"] = rnd(1000, hid), torch.randint(0, 1000, (b,), generator=gen, device=DEV)
        st["qkv"], st["delta"], st["gu"] = rnd(b, (g + 2) * h * D), rnd(b, hid), rnd(b, 2 * ffn)
        st["w1"], st["w2"] = 1 + 0.1 * rnd(hid), 1 + 0.1 * rnd(hid)
        st["inv"] = step_ops.rope_inv_freq(500000.0, DEV)
        st["qbuf"] = torch.empty(heads * g, D, dtype=torch.float16, device=DEV)
        # position, window slot, window length, compressed length: read by the kernels on the device
        st["state"] = torch.tensor([t + w - 1, w - 1, w, t], dtype=torch.int32, device=DEV)
        st["stage"] = min(8192, 64 * (D - st["rank"] + 4) + 896)
        st["ws"] = ops.new_workspace(st["qbuf"].device, ops.plan(heads, t + 1024, 384, g)[1])
    return st


# ------------------------------------------------------------------------------------------------ one pass
def _cache(*stores):
    if isinstance(stores[0], comp.SparseStore):
        return [(s.bitmaps, s.accum, s.nz, s.stats) for s in stores]
    return [(s.bitmaps, s.tile_offsets, s.counts, s.units, s.scales, s.zeros, s.packed, s.head_tail, s.stats) for s in stores]


def run(st):
    case = st["case"]
    what = case["what"]
    if what == "decode":
        if case["bits"] == 16:
            return ops.decode_attention(st["q"], st["k"], st["v"], st["kw"], st["vw"], case["group"])
        return ops_quant.decode_attention_quant(st["q"], st["k"].as_dict(), st["v"].as_dict(), case["tokens"], st["kw"], st["vw"],
                                                case["group"], case["bits"])
    if what == "prefill":
        for s, x in zip((st["k"], st["v"]), st["x"]):
            s.reset()
            s.append(x, st["rank"])
        return _cache(st["k"], st["v"])
    if what == "append":
        for s, w in ((st["k"], st["kw"]), (st["v"], st["vw"])):
            s.tokens = case["tokens"]                # the same block again, behind the same cache
            s.append(w[:, :256], st["rank"])
        return _cache(st["k"], st["v"])
    if what == "convert":
        got = []
        for fn, x, nz in zip((comp.convert_key_batched, comp.convert_value_batched), st["x"], st["nz"]):
            bitmaps, accum, packed = fn(x)
            # the per-head values back to back, as the model code keeps them (here in a buffer for the longest case)
            torch.cat(packed, out=nz[:sum(p.numel() for p in packed)])
            got.append((bitmaps, accum, nz))
        return got
    if what == "ops":
        t, g, bq = case["tokens"], case["group"], case["batch"] * case["kv_heads"] * case["group"]
        if case["bits"] == 16:
            (kb, kn, ki, ko), (vb, vn, vi, vo) = st["k"], st["v"]
            return (ops.mustafar_key_formulation(kb, kn, ki, ko, st["q8"], t, D, bq, g),
                    ops.mustafar_value_formulation(vb, vn, vi, vo, st["p8"], st["ws"], D, t, bq, g))
        k, v, bits = st["k"], st["v"], case["bits"]
        return (ops_quant.mustafar_key_formulation_quant(k["bitmaps"], k["packed"], k["tile_offsets"], k["scales"], k["zeros"],
                                                         st["q8"], t, D, bq, g, bits, 32 // bits),
                ops_quant.mustafar_value_formulation_quant(v["bitmaps"], v["packed"], v["tile_offsets"], v["counts"], v["units"],
                                                           v["scales"], v["zeros"], st["p8"], st["ws"], D, t, bq, g, bits,
                                                           32 // bits))
    g, h, s = case["group"], case["kv_heads"], st["state"]
    prune = dict(prune_rank=st["rank"], prune_back=128) if case["prune"] else {}
    x = st["embed"].index_select(0, st["ids"])
    h1 = step_ops.add_rmsnorm(x, None, st["w1"], 1e-5)
    step_ops.rope_append(st["qkv"], st["inv"], s[0:1], s[1:2], g * h, h, st["qbuf"], st["kw"], st["vw"], **prune)
    att = ops.decode_attention(st["qbuf"], st["k"], st["v"], st["kw"], st["vw"], g, stage_halves=st["stage"],
                               window_len=s[2:3], n_tokens=s[3:4], workspace=st["ws"])
    h2 = step_ops.add_rmsnorm(x, st["delta"], st["w2"], 1e-5)
    return x, h1, st["qbuf"], st["kw"], st["vw"], att, h2, step_ops.silu_mul(st["gu"])


# ------------------------------------------------------------------------------------------------ bounds
def _cache_bytes(case, heads, tokens):
    """K and V of the compressed cache as stored: bitmaps, offsets, values (kept ones, padded per tile on average)."""
    kept = D - comp.keep_rank(case["sparsity"]) + 1
    tiles, bits = 2 * 2 * tokens * heads, case.get("bits", 16)
    if bits == 16:
        return tiles * (8 + 4 + 2 * (kept / 2 + 3.5))
    ng = 64 // case.get("qgroup", 64)
    return tiles * (8 + 4 + 4 * ng + 4 * (kept / 2 * bits / 32 + 0.5))


def work(case):
    what = case["what"]
    kept = D - comp.keep_rank(case["sparsity"]) + 1
    if what in ("decode", "step"):
        heads, g = case["batch"] * case["kv_heads"], case["group"]
        nbytes = _cache_bytes(case, heads, case["tokens"]) + 2 * 2 * heads * case["window"] * D + 2 * 2 * heads * g * D
        flops = 4.0 * heads * g * (case["tokens"] * kept + case["window"] * D)
        if what == "step":
            b, hid = case["batch"], case["hidden"]
            nbytes += 2 * (b * 2 * (g + 2) * case["kv_heads"] * D + b * 5 * hid + 2 * hid + b * 3 * case["ffn"])
            flops += b * (10 * hid + 6 * case["ffn"])
        return dict(bytes=nbytes, flops=flops)
    if what == "ops":
        heads, g, t = case["batch"] * case["kv_heads"], case["group"], case["tokens"]
        # read the cache, the query and the probabilities (row 0 of the padded operands), write the padded results
        return dict(bytes=_cache_bytes(case, heads, t) + heads * g * (2 * D + 2 * t + 16 * t + 16 * D),
                    flops=4.0 * heads * g * t * kept)
    heads = case["heads"] if what == "convert" else case["batch"] * case["kv_heads"]
    n = 256 if what == "append" else case["tokens"]
    out = _cache_bytes(case, heads, n)
    if case.get("bits", 16) != 16:
        out += 2 * 2 * n * heads * 8                 # counts and units per tile
    return dict(bytes=2 * 2 * heads * n * D + out, flops=2.0 * 2 * heads * n * D)


def tolerance(case):
    if case["what"] in ("prefill", "append", "convert"):
        return "exact"                               # bitmaps, offsets, packed values and codes are defined bit for bit
    # fp16 results, probabilities and dequantised values rounded to fp16, fp32 sums
    return {"rel": 2e-3, "max": 0.05}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _prune(x, rank):
    size = x.abs().float()
    return x * (size >= size.kthvalue(rank, dim=-1, keepdim=True).values)


def _stored(x, kind, bits, qgroup):
    """Pruned values as a cache of ``bits``-bit codes stands for them: (code - zero) * scale of each tile's groups."""
    if bits == 16:
        return x
    heads, n, _ = x.shape
    tiles = (x.view(heads, n // 64, 64, D).transpose(2, 3) if kind == comp.KEY else x.view(heads, n, 2, 64)).float()
    there, out = tiles != 0, torch.zeros_like(tiles)
    nth = there.cumsum(-1, dtype=torch.int16) - 1
    for g in range(64 // qgroup):
        mine = there & (nth >= g * qgroup) & (nth < (g + 1) * qgroup)
        lo = tiles.masked_fill(~mine, math.inf).amin(-1, keepdim=True)
        hi = tiles.masked_fill(~mine, -math.inf).amax(-1, keepdim=True)
        # tensors divided by tensors: a scalar divisor may be turned into a product with its reciprocal
        scale = (hi - lo) / torch.full_like(lo, 2 ** bits - 1)
        scale = torch.where(scale == 0, torch.ones_like(scale), scale)
        zero = torch.floor(-lo / scale + 0.5).half().float()
        scale = scale.half().float()
        code = (torch.floor(tiles / torch.where(scale == 0, torch.ones_like(scale), scale) + 0.5) + zero).clamp(0, 2 ** bits - 1)
        out = torch.where(mine, (code - zero) * scale, out)
    return (out.transpose(2, 3) if kind == comp.KEY else out).reshape(heads, n, D)


class _Dense:
    """Takes a store's place in ``_fill`` and keeps the values its cache would stand for."""

    def __init__(self, heads, kind, bits, qgroup):
        self.n_heads, self.kind, self.bits, self.qgroup, self.parts = heads, kind, bits, qgroup, []

    def append(self, x, rank):
        step = max(1, (1 << 25) // (x.shape[1] * D))
        self.parts.append(torch.cat([_stored(_prune(y, rank), self.kind, self.bits, self.qgroup) for y in x.split(step)]))

    def heads(self, lo, hi):
        return torch.cat([p[lo:hi] for p in self.parts], dim=1).double()


def _pair(case, heads):
    return [_Dense(heads, kind, case.get("bits", 16), case.get("qgroup", 64)) for kind in (comp.KEY, comp.VALUE)]


def _attend(k, v, kw, vw, q, group):
    out, n = [], sum(p.shape[1] for p in k.parts)
    step = max(1, (1 << 26) // (n * D))
    for lo in range(0, k.n_heads, step):
        hi = min(k.n_heads, lo + step)
        ks, vs = (torch.cat([s.heads(lo, hi), w[lo:hi].double()], 1) for s, w in ((k, kw), (v, vw)))
        s = q[lo * group:hi * group].double().view(hi - lo, group, D) @ ks.transpose(1, 2) / math.sqrt(D)
        out.append((s.softmax(-1) @ vs).view(-1, D))
    return torch.cat(out)


def _rmsnorm(x, w):
    return x * (x.square().mean(-1, keepdim=True) + 1e-5).rsqrt() * w


def _rotate(x, angle):
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def exact(case, seed):
    what = case["what"]
    if what not in ("decode", "ops", "step"):
        return None                                  # nothing but values taken over as they are, and integers
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rank, g = comp.keep_rank(case["sparsity"]), case["group"]
    heads, t = case["batch"] * case["kv_heads"], case["tokens"]
    k, v = _pair(case, heads)
    if what == "ops":
        if case["bits"] == 16:
            _fill(gen, case, k, v, t, _k_scale(gen, heads))
        else:
            k.append(_kv(gen, heads, t, _k_scale(gen, heads)), rank)
            v.append(_kv(gen, heads, t), rank)
        q = _kv(gen, heads * g, 1)
        p = torch.softmax(2 * torch.randn(heads * g, 1, t, generator=gen, device=DEV), -1).half()
        got = [torch.zeros(heads * g, 8, n, dtype=torch.float64, device=DEV) for n in (t, D)]
        step = max(1, (1 << 26) // (t * D))
        for lo in range(0, heads, step):
            hi = min(heads, lo + step)
            rows = slice(lo * g, hi * g)
            got[0][rows, 0] = (q[rows].double().view(hi - lo, g, D) @ k.heads(lo, hi).transpose(1, 2)).view(-1, t)
            got[1][rows, 0] = (p[rows].double().view(hi - lo, g, t) @ v.heads(lo, hi)).view(-1, D)
        return tuple(got)
    scale = _k_scale(gen, heads)
    _fill(gen, case, k, v, t, scale)
    w = case["window"]
    if what == "decode":
        kw, vw = _kv(gen, heads, w, scale), _kv(gen, heads, w)
        return _attend(k, v, kw, vw, _kv(gen, heads * g, 1)[:, 0], g)
    b, h, hid, ffn = case["batch"], case["kv_heads"], case["hidden"], case["ffn"]
    kw, vw = _kv(gen, heads, 384, scale), _kv(gen, heads, 384)
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV).half()  # noqa: E731
    embed, ids = rnd(1000, hid), torch.randint(0, 1000, (b,), generator=gen, device=DEV)
    qkv, delta, gu = rnd(b, (g + 2) * h * D).double(), rnd(b, hid).double(), rnd(b, 2 * ffn).double()
    w1, w2 = 1 + 0.1 * rnd(hid), 1 + 0.1 * rnd(hid)
    angle = (t + w - 1) * 500000.0 ** -(torch.arange(D // 2, dtype=torch.float64, device=DEV) / (D // 2))
    kw, vw = kw.double(), vw.double()
    qn, kn, vn = qkv.view(b, (g + 2) * h, D).split([g * h, h, h], dim=1)
    q = _rotate(qn, angle).reshape(-1, D)
    kw[:, w - 1], vw[:, w - 1] = _rotate(kn, angle).reshape(-1, D), vn.reshape(-1, D)
    if case["prune"]:
        for win in (kw, vw):
            win[:, w - 130] = _prune(win[:, w - 130], rank)
    x = embed[ids].double()
    y = x + delta
    gate, up = gu.chunk(2, -1)
    att = _attend(k, v, kw[:, :w], vw[:, :w], q, g)
    return y, _rmsnorm(x, w1.double()), q, kw, vw, att, _rmsnorm(y, w2.double()), gate * gate.sigmoid() * up
