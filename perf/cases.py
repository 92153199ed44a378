"""Performance cases of the attention library: what its users call, over the sizes they call it with.

A case is a dict of plain values.  Its `kind` picks the entry point:

  dense    flash_attn_func            equal or unequal lengths, forward or forward + backward
  packed   flash_attn_qkvpacked_func  one (batch, seq, 3, heads, dim) tensor, forward + backward
  varlen   flash_attn_varlen_func     packed sequences of different lengths
  cache    flash_attn_with_kvcache    append to a paged or contiguous cache, then attend to it
  int8     attention_int8             INT8 Q K^T forward

Sequence lengths of a batch belong to the case (`lens_seed`), the values of the tensors to the seed
of prepare().
"""
import math
import random

import numpy as np
import torch

import flash_attn_triton_b200 as fa

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _dense(name, **kw):
    c = dict(name=name, kind="dense", dtype="fp16", batch=1, seq_q=128, seq_k=128, heads=16, heads_kv=16, dim=128,
             causal=True, train=True)
    c.update(kw)
    return c


def _packed(name, **kw):
    c = dict(name=name, kind="packed", dtype="bf16", batch=8, seq=512, heads=16, dim=64, causal=False, dropout=0.1)
    c.update(kw)
    return c


def _varlen(name, **kw):
    c = dict(name=name, kind="varlen", dtype="fp16", sequences=32, shortest=256, longest=4096, multiple=64, heads=32,
             heads_kv=32, dim=128, causal=True, window=-1, alibi=False, softcap=0.0, train=True, lens_seed=3)
    c.update(kw)
    return c


def _cache(name, **kw):
    c = dict(name=name, kind="cache", dtype="fp16", batch=64, shortest=1024, longest=32768, new=1, page=256, heads=32,
             heads_kv=8, dim=128, rotary=True, lens_seed=1)
    c.update(kw)
    return c


def _int8(name, **kw):
    c = dict(name=name, kind="int8", dtype="fp16", batch=8, heads=32, seq=8192, dim=128, causal=True, train=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest training call (unit tests, tiny models): all latency and launches
        _dense("train_tiny", batch=2, seq_q=128, seq_k=128, heads=4, heads_kv=4, dim=64),
        # the headline training step: long causal sequences, a full device
        _dense("train_long", batch=16, seq_q=4096, seq_k=4096, heads=16, heads_kv=16, dim=128),
        # encoder-decoder cross attention in training: narrow heads, no mask, key length no multiple of a tile
        _dense("train_cross", batch=4, seq_q=1024, seq_k=1531, heads=32, heads_kv=32, dim=64, causal=False),
        # prompt processing of one request with grouped query heads, an odd prompt length
        _dense("prefill_gqa", dtype="bf16", batch=1, seq_q=4001, seq_k=4001, heads=32, heads_kv=8, train=False),
        # prompt processing with the widest heads
        _dense("prefill_d256", dtype="bf16", batch=2, seq_q=1999, seq_k=1999, heads=16, heads_kv=8, dim=256, train=False),
        # encoder training on packed qkv with attention dropout
        _packed("train_dropout"),
        # training on packed documents with every score option: window, ALiBi, soft cap
        _varlen("varlen_train", window=1024, alibi=True, softcap=30.0),
        # a batch of prompts of very different lengths packed together
        _varlen("varlen_prefill", dtype="bf16", sequences=24, shortest=17, longest=2048, multiple=1, heads_kv=8, train=False,
                lens_seed=5),
        # one decode step of a large serving batch over a paged cache
        _cache("decode_batch"),
        # one decode step of a single conversation over a contiguous cache: latency
        _cache("decode_single", dtype="bf16", batch=1, shortest=1900, longest=1900, page=0),
        # a chunk of a long prompt appended to, and attending to, a paged cache
        _cache("cache_chunk", dtype="bf16", batch=4, shortest=1024, longest=8192, new=256, page=64, lens_seed=7),
        # INT8 scores over long sequences
        _int8("int8_long"),
    ]


def _log_int(rng, low, high, odd=0.5):
    """Log-uniform whole number; half of them as drawn, the others rounded to a multiple of 64 where that fits."""
    x = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if rng.random() >= odd and x >= 64:
        x = x // 64 * 64
    return max(low, min(high, x))


def draw(rng):
    kind = rng.choice(("train", "train", "prefill", "packed", "varlen", "varlen", "decode", "decode", "chunk", "int8"))
    dtype = rng.choice(("fp16", "bf16"))
    c = None
    while c is None or _cost(c) > _LIMIT[kind]:
        dim = rng.choice((64, 128))
        if kind == "train":
            seq = _log_int(rng, 64, 8192)
            cross = rng.random() < 0.25
            heads = rng.choice((4, 8, 16, 32))
            c = _dense("", dtype=dtype, batch=_log_int(rng, 1, 16, 1.0), seq_q=seq, seq_k=_log_int(rng, 64, 4096) if cross else seq,
                       heads=heads, heads_kv=heads // rng.choice((1, 1, 2, 4)), dim=dim, causal=not cross and rng.random() < 0.7)
        elif kind == "prefill":
            seq = _log_int(rng, 16, 16384)
            heads = rng.choice((8, 16, 32))
            c = _dense("", dtype=dtype, batch=_log_int(rng, 1, 8, 1.0), seq_q=seq, seq_k=seq, heads=heads,
                       heads_kv=heads // rng.choice((1, 2, 4, 8)), dim=rng.choice((64, 128, 128, 256)), train=False)
        elif kind == "packed":
            c = _packed("", dtype=dtype, batch=_log_int(rng, 1, 32, 1.0), seq=_log_int(rng, 64, 2048),
                        heads=rng.choice((8, 12, 16)), dim=dim, causal=rng.random() < 0.3, dropout=rng.choice((0.1, 0.1, 0.2, 0.0)))
        elif kind == "varlen":
            longest = _log_int(rng, 64, 4096)
            heads = rng.choice((8, 16, 32))
            options = rng.random() < 0.4
            c = _varlen("", dtype=dtype, sequences=_log_int(rng, 2, 48, 1.0), shortest=max(1, longest // rng.choice((2, 8, 32))),
                        longest=longest, multiple=rng.choice((1, 1, 64)), heads=heads, heads_kv=heads // rng.choice((1, 1, 4)),
                        dim=dim, window=rng.choice((-1, 256, 1024)) if options else -1, alibi=options and rng.random() < 0.5,
                        softcap=30.0 if options and rng.random() < 0.5 else 0.0, train=rng.random() < 0.5,
                        lens_seed=rng.randrange(1 << 20))
        elif kind in ("decode", "chunk"):
            longest = _log_int(rng, 128, 32768)
            kv = rng.choice((2, 4, 8))
            c = _cache("", dtype=dtype, batch=_log_int(rng, 1, 64, 1.0), shortest=max(1, longest // rng.choice((1, 4, 32))), longest=longest,
                       new=rng.choice((1, 1, 1, 2, 4)) if kind == "decode" else _log_int(rng, 16, 1024),
                       page=rng.choice((0, 16, 64, 128, 256)), heads=kv * rng.choice((1, 4, 8)), heads_kv=kv, dim=dim,
                       rotary=rng.random() < 0.7, lens_seed=rng.randrange(1 << 20))
        else:
            c = _int8("", batch=_log_int(rng, 1, 8, 1.0), heads=rng.choice((8, 16, 32)), seq=64 * _log_int(rng, 2, 128, 1.0),
                      dim=rng.choice((64, 128, 128)), causal=rng.random() < 0.5, train=rng.random() < 0.3)
    del c["name"]
    return c


# the most one drawn case of a kind may cost, in the units of _cost: below the largest listed cases in time
_LIMIT = {"train": 77e9, "prefill": 10e9, "packed": 3e9, "varlen": 20e9, "decode": 8.7e9, "chunk": 2e9, "int8": 60e9}


def _cost(c):
    w = work(c)
    return max(w["bytes"], w["flops"] / 50)


def _lens(c):
    """Lengths of a batch: the packed sequences, or the tokens already in a cache."""
    rng = np.random.default_rng(c["lens_seed"])
    n = c["sequences"] if c["kind"] == "varlen" else c["batch"]
    m = c.get("multiple", 1)
    low = max(1, c["shortest"] // m)
    return (m * rng.integers(low, max(low, c["longest"] // m) + 1, size=n)).tolist()


def _randn(gen, dtype, *shape):
    return torch.randn(*shape, device="cuda", dtype=dtype, generator=gen)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[c["dtype"]]
    s = dict(case=c, kind=c["kind"])
    if c["kind"] == "dense":
        q = _randn(gen, dt, c["batch"], c["seq_q"], c["heads"], c["dim"])
        k = _randn(gen, dt, c["batch"], c["seq_k"], c["heads_kv"], c["dim"])
        v = _randn(gen, dt, c["batch"], c["seq_k"], c["heads_kv"], c["dim"])
        s.update(q=q, k=k, v=v)
        if c["train"]:
            s["dout"] = _randn(gen, dt, *q.shape)
    elif c["kind"] == "packed":
        s["qkv"] = _randn(gen, dt, c["batch"], c["seq"], 3, c["heads"], c["dim"]).requires_grad_()
        s["dout"] = _randn(gen, dt, c["batch"], c["seq"], c["heads"], c["dim"])
        s["random_seed"] = seed
    elif c["kind"] == "varlen":
        lens = _lens(c)
        total = sum(lens)
        q = _randn(gen, dt, total, c["heads"], c["dim"])
        k = _randn(gen, dt, total, c["heads_kv"], c["dim"])
        v = _randn(gen, dt, total, c["heads_kv"], c["dim"])
        s.update(q=q, k=k, v=v, longest=max(lens),
                 cu_seqlens=torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda"))
        s["slopes"] = None
        if c["alibi"]:
            s["slopes"] = torch.tensor([2.0 ** (-8 * (i + 1) / c["heads"]) for i in range(c["heads"])], device="cuda")
        if c["train"]:
            s["dout"] = _randn(gen, dt, *q.shape)
    elif c["kind"] == "cache":
        lens, new, D, Hkv = _lens(c), c["new"], c["dim"], c["heads_kv"]
        most = max(lens) + new
        if c["page"]:
            # pages handed out from a shuffled pool; a row of the table ends in copies of its first page
            need = [-(-(n + new) // c["page"]) for n in lens]
            order = np.random.default_rng(c["lens_seed"] + 1).permutation(sum(need))
            table = np.zeros((c["batch"], max(need)), dtype=np.int32)
            at = 0
            for b, n in enumerate(need):
                table[b, :n] = order[at:at + n]
                table[b, n:] = order[at]
                at += n
            s["block_table"] = torch.from_numpy(table).cuda()
            shape = (sum(need), c["page"], Hkv, D)
        else:
            s["block_table"] = None
            shape = (c["batch"], most, Hkv, D)
        s["k_cache"], s["v_cache"] = _randn(gen, dt, *shape), _randn(gen, dt, *shape)
        s["q"] = _randn(gen, dt, c["batch"], new, c["heads"], D)
        s["k"], s["v"] = _randn(gen, dt, c["batch"], new, Hkv, D), _randn(gen, dt, c["batch"], new, Hkv, D)
        s["cache_seqlens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        s["cos"] = s["sin"] = None
        if c["rotary"]:
            inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, dtype=torch.float32, device="cuda") / D))
            angle = torch.arange(most, dtype=torch.float32, device="cuda")[:, None] * inv[None, :]
            s["cos"], s["sin"] = torch.cos(angle).to(dt), torch.sin(angle).to(dt)
    else:
        shape = (c["batch"], c["heads"], c["seq"], c["dim"])
        q, k, v = (_randn(gen, dt, *shape) for _ in range(3))
        k *= 1 + 7 * (torch.rand(*shape, device="cuda", generator=gen) < 0.01)      # outliers, as activations have them
        s.update(q=q, k=k, v=v)
        if c["train"]:
            s["dout"] = _randn(gen, dt, *shape)
    if c.get("train"):
        for t in (s["q"], s["k"], s["v"]):
            t.requires_grad_()
    return s


def run(state):
    s, c = state, state["case"]
    if s["kind"] == "dense":
        out = fa.flash_attn_func(s["q"], s["k"], s["v"], causal=c["causal"])
    elif s["kind"] == "packed":
        random.seed(s["random_seed"])       # a reproducible training step: the dropout seed is drawn from here
        out = fa.flash_attn_qkvpacked_func(s["qkv"], dropout_p=c["dropout"], causal=c["causal"])
        return (out,) + torch.autograd.grad(out, (s["qkv"],), s["dout"])
    elif s["kind"] == "varlen":
        out = fa.flash_attn_varlen_func(s["q"], s["k"], s["v"], s["cu_seqlens"], s["cu_seqlens"], s["longest"], s["longest"],
                                        causal=c["causal"], window_size=(c["window"], 0 if c["window"] >= 0 else -1),
                                        softcap=c["softcap"], alibi_slopes=s["slopes"])
    elif s["kind"] == "cache":
        out = fa.flash_attn_with_kvcache(s["q"], s["k_cache"], s["v_cache"], s["k"], s["v"], s["cos"], s["sin"],
                                         cache_seqlens=s["cache_seqlens"], block_table=s["block_table"], causal=True,
                                         rotary_interleaved=False)
        return out, s["k_cache"], s["v_cache"]
    else:
        out = fa.attention_int8(s["q"], s["k"], s["v"], causal=c["causal"])
    if c["train"]:
        return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    return out


def _pairs(n, m, causal, window=-1, start=0):
    """(query, key) pairs that see each other: query i sits at start + i and has m keys before it or around it."""
    i = np.arange(start, start + n, dtype=np.int64)
    last = np.minimum(i, m - 1) if causal else np.full(n, m - 1, dtype=np.int64)
    first = np.maximum(i - window, 0) if window >= 0 else np.zeros(n, dtype=np.int64)
    return int(np.maximum(last - first + 1, 0).sum())


def work(case):
    """Bytes: inputs read once, outputs written once.  FLOPs: two products per visible pair and head in the
    forward, five in the backward."""
    c = case
    D, H = c["dim"], c["heads"]
    train = c["kind"] == "packed" or bool(c.get("train"))
    if c["kind"] == "dense":
        q = c["batch"] * c["seq_q"] * H * D
        kv = c["batch"] * c["seq_k"] * c["heads_kv"] * D
        pairs = c["batch"] * H * _pairs(c["seq_q"], c["seq_k"], c["causal"])
    elif c["kind"] == "varlen":
        lens = _lens(c)
        q, kv = sum(lens) * H * D, sum(lens) * c["heads_kv"] * D
        pairs = H * sum(_pairs(n, n, c["causal"], c["window"]) for n in lens)
    elif c["kind"] == "cache":
        lens, new, Hkv = _lens(c), c["new"], c["heads_kv"]
        q, knew = c["batch"] * new * H * D, c["batch"] * new * Hkv * D
        pairs = H * sum(_pairs(new, n + new, True, start=n) for n in lens)
        # the cached keys and values, the new ones read and written, q and the output
        return {"bytes": 2.0 * (2 * sum(lens) * Hkv * D + 4 * knew + 2 * q), "flops": 4.0 * D * pairs}
    else:
        q = kv = c["batch"] * c["seq"] * H * D
        pairs = c["batch"] * H * _pairs(c["seq"], c["seq"], c["causal"])
    elements = 2 * q + 2 * kv + ((2 * q + 2 * kv) if train else 0)
    return {"bytes": 2.0 * elements, "flops": 4.0 * D * pairs * (3.5 if train else 1.0)}


def tolerance(case):
    """Probabilities and score gradients are rounded to the tensors' type before they are multiplied, results
    when they are stored: a few units of 2^-11 (fp16) or 2^-9 (bf16).  With a soft cap the tanh carries the same
    relative error into the exponent, which grows with the score."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}
    return {"rel": 5e-3 if case.get("softcap") else 3e-3}
