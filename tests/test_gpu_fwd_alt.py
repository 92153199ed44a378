"""The one-tile forward kernel (fwd_alt_sm100.cu): head_dim 256, and chunks of tokens against a KV cache."""
import numpy as np
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu


def dev(t):
    return None if t is None else t.to(DEV)


@pytest.mark.parametrize("Sq,Sk,Hq,Hkv,kw", [
    (256, 256, 2, 2, dict(causal=True)),                       # two key tiles: one per softmax group
    (129, 257, 2, 1, dict()),                                  # a tile of one row, a tile of one key
    (700, 900, 4, 2, dict(causal=True)),                       # odd number of tiles
    (300, 1500, 2, 1, dict(window=(200, 100))),                # tiles skipped on both sides
    (400, 400, 2, 2, dict(causal=True, softcap=20.0, alibi=True)),
    (640, 320, 1, 1, dict(causal=True, window=(64, -1))),      # query tiles that see no key
])
def test_d256_vs_oracle(Sq, Sk, Hq, Hkv, kw):
    from flash_attn_triton_b200 import _native as N, _ops
    q, k, v, _ = cases.dense_case(Sq + Sk, 2, Sq, Sk, Hq, Hkv, 256)
    sl = torch.tensor([0.5 ** (i + 1) for i in range(Hq)]) if kw.get("alibi") else None
    wl, wr = kw.get("window", (-1, -1))
    alibi = None if sl is None else dev(sl).unsqueeze(0).expand(2, -1).contiguous()
    o, lse, _ = _ops.dense_forward(dev(q), dev(k), dev(v), 1 / 16, kw.get("causal", False), wl, wr, kw.get("softcap", 0.0),
                                   alibi, 0, N.IMPL_TCGEN05, "bshd", True)
    ro, rl = orc.attention_ref(q, k, v, softmax_scale=1 / 16, causal=kw.get("causal", False), window=(wl, wr),
                               softcap=kw.get("softcap", 0.0), alibi_slopes=sl)
    assert maxdiff(o, ro) <= util.FWD_TOL
    assert maxdiff(lse * util.LN2, rl) <= util.FWD_TOL
    assert N.lib().fa_device_wait_status(0) == 0


def test_d256_packed_keeps_neighbours_out():
    """Packed sequences whose lengths end inside a tile, next to a sequence of NaN and infinities."""
    import flash_attn_triton_b200 as fa
    lens = [300, 131, 257]
    q, k, v, _, cu, _ = cases.varlen_case(5, lens, lens, 2, 1, 256)
    k[300:431] = float("nan")
    v[300:431] = float("inf")
    out = fa.flash_attn_varlen_func(dev(q), dev(k), dev(v), dev(cu), dev(cu), 300, 300, causal=True)
    for a, b in ((0, 300), (431, 688)):
        ro, _ = orc.attention_ref(q[None, a:b], k[None, a:b], v[None, a:b], causal=True)
        assert maxdiff(out[a:b], ro[0]) <= util.FWD_TOL


CHUNKS = [
    # Hq, Hkv, D, page (0: contiguous), tokens in the cache, new tokens, options
    (8, 2, 128, 64, [500, 0, 131], 96, dict(causal=True, rotary=128)),
    (8, 2, 128, 16, [77, 1000], 33, dict(causal=True, rotary=64, interleaved=True)),
    (4, 4, 64, 256, [3, 700], 17, dict(causal=True)),                         # just past the decode kernel
    (6, 2, 64, 128, [260, 129], 40, dict(causal=True, rotary=32)),            # groups of three: no packing
    (16, 1, 128, 0, [2100], 20, dict(causal=True, rotary=128)),               # few units: keys in pieces
    (4, 1, 256, 32, [300, 10], 130, dict(causal=True, rotary=256)),
    (4, 2, 128, 0, [200, 90], 64, dict(window=(50, 20))),
    (4, 2, 128, 0, [5, 128], 40, dict(causal=True, alibi=True, leftpad=[7, 0])),
    (8, 2, 64, 64, [640, 64], 0, dict(causal=True, queries=64)),              # nothing appended
]


@pytest.mark.parametrize("case", range(len(CHUNKS)))
def test_cache_chunk_vs_oracle(case):
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    Hq, Hkv, D, page, lens, new, kw = CHUNKS[case]
    rng = np.random.default_rng(700 + case)
    B, pads = len(lens), kw.get("leftpad")
    Sq = kw.get("queries", new)
    most = max(n + new + (pads[b] if pads else 0) for b, n in enumerate(lens))
    q = cases.randn16(rng, B, Sq, Hq, D)
    kn, vn = (cases.randn16(rng, B, new, Hkv, D) for _ in range(2))
    bt = None
    if page:
        need = [-(-(n + new) // page) for n in lens]
        table = np.zeros((B, max(need) + 1), dtype=np.int32)
        order, at = rng.permutation(sum(need) + 2), 0
        for b, n in enumerate(need):
            table[b, :n] = order[at:at + n]
            table[b, n:] = order[at]
            at += n
        bt = torch.from_numpy(table)
        shape = (sum(need) + 2, page, Hkv, D)
    else:
        shape = (B, most + 3, Hkv, D)
    kc, vc = cases.randn16(rng, *shape), cases.randn16(rng, *shape)
    # rows past the cached tokens hold what an earlier user left there: not finite
    used = torch.zeros(shape[:2], dtype=torch.bool)
    for b, n in enumerate(lens):
        for t in range(n):
            pos = t + (pads[b] if pads else 0)
            used[(int(bt[b, pos // page]), pos % page) if page else (b, pos)] = True
    kc[~used], vc[~used] = float("nan"), float("inf")
    cos = sin = None
    if "rotary" in kw:
        cos, sin = cases.rotary_tables(most + 5, kw["rotary"])
    sl = torch.tensor([0.5 ** (i + 1) for i in range(Hq)]) if kw.get("alibi") else None
    pad = torch.tensor(pads, dtype=torch.int32) if pads else None
    cl = torch.tensor(lens, dtype=torch.int32)
    common = dict(causal=kw.get("causal", False), rotary_interleaved=kw.get("interleaved", False))
    ro, rkc, rvc = orc.kvcache_ref(q, kc, vc, kn if new else None, vn if new else None, cos, sin, cache_seqlens=cl,
                                   cache_leftpad=pad, block_table=bt, window=kw.get("window", (-1, -1)), alibi_slopes=sl, **common)
    kcd, vcd = dev(kc), dev(vc)
    for _ in range(2):                   # the second call appends the same tokens again
        out = fa.flash_attn_with_kvcache(dev(q), kcd, vcd, dev(kn) if new else None, dev(vn) if new else None, dev(cos), dev(sin),
                                         cache_seqlens=dev(cl), cache_leftpad=dev(pad), block_table=dev(bt),
                                         window_size=kw.get("window", (-1, -1)), alibi_slopes=dev(sl), **common)
        assert maxdiff(out, ro) <= util.FWD_TOL
    for got, want in ((kcd, rkc), (vcd, rvc)):
        got, want = got.cpu(), want
        same = torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))
        assert same and torch.equal(got.isnan(), want.isnan())
    with pytest.raises(ValueError):      # the checks run ahead of the append: nothing is written
        bad = cl.clone()
        bad[0] = 1 << 20
        fa.flash_attn_with_kvcache(dev(q), kcd, vcd, dev(kn) if new else None, dev(vn) if new else None, dev(cos), dev(sin),
                                   cache_seqlens=dev(bad), cache_leftpad=dev(pad), block_table=dev(bt), **common)
    assert torch.equal(torch.nan_to_num(kcd.cpu(), nan=7.0), torch.nan_to_num(rkc, nan=7.0))
    assert N.lib().fa_device_wait_status(0) == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,causal,window", [
    (1, 128, 128, 2, 1, True, (-1, -1)),          # one tile
    (2, 129, 385, 2, 2, False, (-1, -1)),         # a row and a key past the tiles
    (1, 640, 300, 4, 1, True, (-1, -1)),          # query tiles past the last key
    (1, 700, 700, 2, 2, True, (150, -1)),         # tiles skipped, rows that see part of two tiles
    (1, 2100, 2100, 12, 3, True, (-1, -1)),       # more CTAs than SMs
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dense_routes(monkeypatch, B, Sq, Sk, Hq, Hkv, causal, window, D, dtype):
    """The three dense forward kernels against the oracle on the same problem, rows past it untouched."""
    from flash_attn_triton_b200 import _native as N, _ops
    q, k, v, _ = (t.to(dtype) for t in cases.dense_case(Sq + Sk + D, B, Sq, Sk, Hq, Hkv, D))
    ro, rl = orc.attention_ref(q, k, v, causal=causal, window=window)
    for route in (None, "0", "1"):                # by the rule (the one-tile kernel here), two-tile, persistent
        if route is None:
            monkeypatch.delenv("FA_B200_FWD_PERSISTENT_FROM", raising=False)
        else:
            monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", route)
        o, lse, _ = _ops.dense_forward(dev(q), dev(k), dev(v), D ** -0.5, causal, *window, 0.0, None, 0, N.IMPL_TCGEN05,
                                       "bshd", True)
        assert maxdiff(o, ro) <= util.tols(dtype)[0], route
        assert maxdiff(lse * util.LN2, rl) <= util.tols(dtype)[0], route
    assert N.lib().fa_device_wait_status(0) == 0


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal,window", [
    (16, 16, 2048, 2048, 128, True, None),     # one entry: one-tile kernel, all: persistent
    (16, 16, 4096, 4096, 64, True, None),
    (16, 16, 2048, 2048, 128, False, None),    # ... with part of the exponentials on the FMA pipe
    (16, 16, 2049, 2175, 64, False, None),
    (20, 16, 2048, 1930, 128, False, None),    # as many key tiles, but below the persistent kernel's first length
    (24, 8, 8192, 8192, 128, True, None),
    (16, 16, 1024, 1024, 64, False, None),     # one entry: one-tile kernel, all: two-tile
    (32, 16, 300, 500, 128, False, None),
    (32, 16, 384, 384, 64, True, None),
    (32, 16, 700, 700, 128, False, (200, 60)),
    (16, 16, 2500, 2500, 64, False, (300, -1)),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_an_entry_has_the_same_result_in_any_batch(B, H, Sq, Sk, D, causal, window, dtype):
    """The kernel depends on the number of tiles of the call; the results (and the LSE) do not."""
    from flash_attn_triton_b200 import _native as N, _ops
    g = torch.Generator(DEV).manual_seed(Sk)
    q, k, v = (2 * torch.randn(B, s, H, D, device=DEV, dtype=dtype, generator=g) for s in (Sq, Sk, Sk))
    wl, wr = window or (-1, -1)

    def run(n):
        o, lse, _ = _ops.dense_forward(q[:n], k[:n], v[:n], D ** -0.5, causal, wl, wr, 0.0, None, 0, N.IMPL_AUTO, "bshd", True)
        return o, lse

    whole = run(B)
    for n in (1, 2):
        for a, b in zip(run(n), whole):
            assert torch.equal(a, b[:n])


def _exact_chunk(q, k, v, start):
    """float64 attention of the tokens at start.. over all keys, causal; (tokens, heads, dim) each"""
    g = q.shape[1] // k.shape[1]
    k, v = (t.double().repeat_interleave(g, 1) for t in (k, v))
    s = torch.einsum("ihd,jhd->hij", q.double(), k) / q.shape[-1] ** 0.5
    i = torch.arange(q.shape[0], device=q.device)[:, None] + start
    return torch.einsum("hij,jhd->ihd", s.masked_fill(torch.arange(k.shape[0], device=q.device) > i, -torch.inf).softmax(-1), v)


@pytest.mark.parametrize("tokens,length,Hq,Hkv,D,size", [(40, 300, 8, 2, 64, 1.0), (100, 3000, 16, 4, 128, 1.0), (100, 3000, 16, 4, 128, 4.0),
                                                         (20, 900, 8, 8, 256, 1.0), (130, 127, 8, 8, 128, 2.0)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_cache_chunk_is_as_exact_as_decode(tokens, length, Hq, Hkv, D, size, dtype):
    """Against float64, not above the decode kernel (which an explicit number of pieces takes), whose probabilities are rounded
    once and relative to finer maxima.  Both round the output; in two parts P adds next to nothing to that."""
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(length)
    mk = lambda *s, f=1.0: (torch.randn(*s, device=DEV, generator=g) * f).to(dtype)
    q, kc, vc = mk(2, tokens, Hq, D, f=size), mk(2, length + tokens, Hkv, D), mk(2, length + tokens, Hkv, D)
    lens = torch.full((2,), length + tokens, dtype=torch.int32, device=DEV)
    err = []
    for splits in (0, 1):
        out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=splits)
        ref = torch.stack([_exact_chunk(q[b], kc[b], vc[b], length) for b in range(2)])
        err.append(((out.double() - ref).norm() / ref.norm()).item())
    assert err[0] <= err[1], err


def test_cache_chunk_keeps_infinite_values():
    """An infinite value of a visible key makes its column infinite and no other, not NaN, for every row that sees the key."""
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(1)
    q, kc, vc = (torch.randn(1, n, h, 64, device=DEV, dtype=torch.half, generator=g) for n, h in ((64, 8), (500, 2), (500, 2)))
    vc[0, 70, 1, 5], vc[0, 333, 0, 9] = float("inf"), float("-inf")
    kc[0, 333, 0] = 8 * q[0, 10, 2] / q[0, 10, 2].norm()            # close to the whole weight of one row
    lens = torch.tensor([500], dtype=torch.int32, device=DEV)
    out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True)
    want = torch.zeros_like(out)
    want[0, :, 4:, 5], want[0, :, :4, 9] = float("inf"), float("-inf")
    assert torch.equal(out.isinf(), want.isinf()) and torch.equal(out[out.isinf()], want[want.isinf()])
    assert torch.isfinite(out[~out.isinf()]).all()
