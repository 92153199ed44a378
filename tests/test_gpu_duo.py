"""The forward with two CTAs per SM against the two-tile kernel: bit for bit the same, whatever the options, head groups,
ragged ends and strides, dense and packed."""
import random

import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu

OPTIONS = [
    dict(causal=True), dict(), dict(window_size=(150, 0)), dict(window_size=(60, 90)),
    dict(causal=True, softcap=20.0), dict(alibi=True), dict(causal=True, alibi=True, window_size=(200, -1)),
]


def enough_tiles(tiles, heads):
    """More than 2.5 CTAs per SM: the calls that the rule of the kernel takes."""
    return 2 * tiles * heads > 5 * torch.cuda.get_device_properties(0).multi_processor_count


def slopes(kw):
    kw = dict(kw)
    if kw.pop("alibi", False):
        kw["alibi_slopes"] = torch.tensor([0.5 ** (i + 1) for i in range(16)], device=DEV)
    return kw


@pytest.mark.parametrize("kw", OPTIONS + [dict(causal=True, dropout_p=0.2), dict(dropout_p=0.1)], ids=str)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,Hkv", [(400, 400, 16), (385, 640, 4)])
def test_two_ctas_against_two_tiles(monkeypatch, kw, D, Sq, Sk, Hkv):
    import flash_attn_triton_b200 as fa
    assert enough_tiles(10 * -(-Sq // 128), 16)
    kw = slopes(kw)
    g = torch.Generator(DEV).manual_seed(D)
    q = torch.randn(10, Sq, 16, D, device=DEV, dtype=torch.half, generator=g)
    kv = torch.randn(10, Sk, 2, Hkv, D, device=DEV, dtype=torch.half, generator=g)      # k and v: slices of one tensor
    k, v = kv[:, :, 0], kv[:, :, 1]

    def run():
        random.seed(3)                                                                   # the dropout mask
        return fa.flash_attn_func(q, k, v, **kw)

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())


@pytest.mark.parametrize("kw", OPTIONS, ids=str)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_packed_two_ctas(monkeypatch, kw, D, dtype):
    """Empty and one-token sequences, ends inside and on the edge of a tile, and a neighbour full of NaN and infinities."""
    import flash_attn_triton_b200 as fa
    lens = [400, 0, 1, 385, 130, 300, 129, 256, 17, 511] * 3
    assert enough_tiles(sum(lens) // 128 + len(lens) // 2, 16)
    q, k, v, _, cu, _ = cases.varlen_case(7 + D, lens, lens, 16, 4, D)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    opts = slopes(kw)
    run = lambda k, v: fa.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), cu.to(DEV), max(lens), max(lens), **opts)
    got = run(k, v)
    bad = slice(int(cu[4]), int(cu[5]))                                                  # the 130 tokens after the 385
    kb, vb = k.clone(), v.clone()
    kb[bad], vb[bad] = float("nan"), float("inf")
    beside = run(kb, vb)
    assert torch.equal(beside[:bad.start], got[:bad.start]) and torch.equal(beside[bad.stop:], got[bad.stop:])
    ref = dict(kw)
    ref["window"] = ref.pop("window_size", (-1, -1))
    ref["alibi_slopes"] = opts["alibi_slopes"].cpu() if ref.pop("alibi", False) else None
    for b in range(len(lens) // 3):
        if lens[b]:
            r = slice(int(cu[b]), int(cu[b + 1]))
            want, _ = orc.attention_ref(q[None, r], k[None, r], v[None, r], **ref)
            assert maxdiff(got[r], want[0]) <= util.tols(dtype)[0], b
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run(k, v))


@pytest.mark.parametrize("S,D,kw", [(1537, 128, dict(causal=True)), (1920, 128, dict(causal=True)), (1921, 128, dict(causal=True)),
                                    (1600, 128, dict(causal=True, dropout_p=0.2)), (1920, 128, dict()), (1921, 128, dict()),
                                    (1600, 128, dict(causal=True, softcap=20.0)), (2047, 64, dict(causal=True, alibi=True)),
                                    (1530, 64, dict(softcap=20.0))], ids=str)
def test_below_the_persistent_kernel(monkeypatch, S, D, kw):
    """Lengths on both sides of the rule where the two-tile kernel is the alternative: equal to it bit for bit."""
    import random
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(S)
    q, k, v = (torch.randn(2, S, 16, D, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    assert enough_tiles(2 * -(-S // 128), 16)
    opts = slopes(kw)

    def run():
        random.seed(3)                               # the dropout mask
        return fa.flash_attn_func(q, k, v, **opts)

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())


@pytest.mark.parametrize("S,kw", [(128, dict()), (129, dict()), (128, dict(causal=True)), (256, dict(causal=True)), (257, dict(causal=True)),
                                  (256, dict(causal=True, softcap=20.0)), (257, dict(causal=True, alibi=True)), (128, dict(dropout_p=0.2)),
                                  (256, dict(causal=True, dropout_p=0.2)), (400, dict(causal=True, window_size=(255, 0))),
                                  (400, dict(causal=True, window_size=(256, 0))), (640, dict(window_size=(100, 155))),
                                  (640, dict(window_size=(128, 128), softcap=20.0)), (640, dict(window_size=(0, 255), alibi=True))], ids=str)
@pytest.mark.parametrize("packed", [False, True])
def test_short_rows(monkeypatch, S, kw, packed):
    """head_dim 64 on both sides of the rule for P over S: equal to the two-tile kernel bit for bit.  Packed: S on average and longest, the
    rule has another line there."""
    import flash_attn_triton_b200 as fa
    kw = slopes(kw)
    if packed and "dropout_p" in kw:
        pytest.skip("packed calls with dropout have another kernel")
    g = torch.Generator(DEV).manual_seed(S)
    B, half = 24, 50 if packed else 0
    assert enough_tiles(B * -(-S // 128), 16)
    lens = [S - half, S + half] * (B // 2)
    q, k, v = (torch.randn(sum(lens), 16, 64, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)

    def run():
        random.seed(3)                               # the dropout mask
        if packed:
            return fa.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), **kw)
        return fa.flash_attn_func(*(t.view(B, S, 16, 64) for t in (q, k, v)), **kw)

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())


@pytest.mark.parametrize("B,Sq,S,H,D,kw", [
    (8, 1030, 1030, 8, 128, dict()), (6, 1536, 1536, 8, 128, dict()), (8, 1030, 1030, 8, 64, dict(softcap=20.0)),
    (4, 1700, 1792, 16, 128, dict(alibi=True)), (7, 1000, 1900, 8, 128, dict(dropout_p=0.1)), (5, 1100, 1700, 16, 128, dict(causal=True)),
    (5, 1300, 1900, 16, 128, dict(causal=True, softcap=20.0)), (5, 1664, 1664, 16, 64, dict(causal=True, alibi=True)),
    (5, 1664, 1664, 16, 128, dict(causal=True, dropout_p=0.1)), (-14, 900, 900, 16, 128, dict()), (-14, 1900, 1900, 8, 128, dict(softcap=20.0)),
    (-14, 1900, 1900, 8, 64, dict(alibi=True))], ids=str)
def test_longer_rows(monkeypatch, B, Sq, S, H, D, kw):
    """Seven to fifteen key tiles, on both sides of the rule that goes by the waves of the two kernels, rows and keys of different
    lengths and (B < 0) packed: equal to the two-tile kernel bit for bit."""
    import flash_attn_triton_b200 as fa
    packed, B = B < 0, abs(B)
    g = torch.Generator(DEV).manual_seed(S)
    mk = lambda n: torch.randn(n, H, D, device=DEV, dtype=torch.half, generator=g)
    kw = dict(kw)
    if kw.pop("alibi", False):
        kw["alibi_slopes"] = torch.tensor([0.5 ** (i + 1) for i in range(H)], device=DEV)
    lens = [S - 300 * (i % 2) for i in range(B)] if packed else [S] * B
    rows = lens if packed else [Sq] * B
    q, k, v = mk(sum(rows)), mk(sum(lens)), mk(sum(lens))
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)

    def run():
        random.seed(3)                               # the dropout mask
        if packed:
            return fa.flash_attn_varlen_func(q, k, v, cu, cu, S, S, **kw)
        return fa.flash_attn_func(q.view(B, Sq, H, D), k.view(B, S, H, D), v.view(B, S, H, D), **kw)

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())


@pytest.mark.parametrize("kw", [dict(), dict(causal=True), dict(softcap=20.0), dict(window_size=(40, 0))], ids=str)
@pytest.mark.parametrize("D", [64, 128])
def test_items_one_behind_the_other(monkeypatch, kw, D):
    """Several items per CTA, of no, one and a few key tiles in turn, whole and ragged: everything is handed on from item to item.  Launches
    one behind the other find the queue as the first one did."""
    import flash_attn_triton_b200 as fa
    rows = [128, 130, 1, 257, 300, 64, 128, 129] * 8
    keys = [0, 128, 129, 0, 1, 300, 256, 17] * 8
    assert enough_tiles(sum(-(-n // 128) for n in rows) // 2, 16)
    g = torch.Generator(DEV).manual_seed(D)
    mk = lambda n, h: torch.randn(n, h, D, device=DEV, dtype=torch.half, generator=g)
    q, k, v = mk(sum(rows), 16), mk(sum(keys), 4), mk(sum(keys), 4)
    cq, ck = (torch.tensor([0] + x, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32) for x in (rows, keys))
    run = lambda: fa.flash_attn_varlen_func(q, k, v, cq, ck, max(rows), max(keys), **kw)
    got = [run() for _ in range(3)]
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    want = run()
    for o in got:
        assert torch.equal(o, want)


@pytest.mark.parametrize("n", [3, 32, 33, 70])
@pytest.mark.parametrize("kw", [dict(causal=True), dict(window_size=(200, 30)), dict(window_size=(100, -1)), dict(window_size=(-1, 60))], ids=str)
def test_order_by_weight(monkeypatch, n, kw):
    """Packed batches on both sides of 32 sequences, empty and short ones among them, heads in one group and in several (keys and values above
    32 MB): every tile is worked on once, whatever the order."""
    import flash_attn_triton_b200 as fa
    lens = [(0, 1, 129, 700, 128, 383, 64)[i * i % 7] for i in range(n)]
    lens[0] = 2000 if n > 3 else 6000
    H, Hk = (16, 4) if n > 3 else (32, 32)
    g = torch.Generator(DEV).manual_seed(n)
    mk = lambda h: torch.randn(sum(lens), h, 128, device=DEV, dtype=torch.half, generator=g)
    q, k, v = mk(H), mk(Hk), mk(Hk)
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)
    run = lambda: fa.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), **kw)
    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())


# With 16 heads on 148 SMs: up to two items per CTA, some of the first ones no tiles (as a list of tiles; with three grid dimensions; short and empty
# sequences first, last and in between)
UNEVEN = [[256, 512, 384, 640, 128, 768, 256, 512], [128] * 12 + [256] * 6, [30] * 2 + [252] * 10, [0] + [256] * 12, [256] * 12 + [0, 0, 1],
          [300, 0, 1, 640, 129, 0, 511, 250, 128, 128, 30, 700]]


@pytest.mark.parametrize("kw", [dict(), dict(alibi=True), dict(softcap=20.0), dict(wl=100, wr=60), dict(wl=0, wr=200, softcap=20.0)], ids=str)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lens", UNEVEN, ids=len)
def test_two_items_per_cta_with_gaps(monkeypatch, lens, D, kw):
    """Every row of O and every LSE is written, as by the two-tile kernel, into buffers that were full of NaN."""
    import ctypes as C
    from flash_attn_triton_b200 import _native as N, _ops
    kw = dict(kw)
    H, grid = 16, 2 * torch.cuda.get_device_properties(0).multi_processor_count
    entries, per = sum(lens) // 128 + len(lens), -(-max(lens) // 128)
    assert grid < min(entries, per * len(lens)) * H <= 2 * grid and enough_tiles(sum(lens) // 128 + len(lens) // 2, H)
    g = torch.Generator(DEV).manual_seed(D)
    mk = lambda h: torch.randn(sum(lens), h, D, device=DEV, dtype=torch.half, generator=g)
    q, k, v = mk(H), mk(4), mk(4)
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)
    sl = torch.full((len(lens), H), 0.125, device=DEV) if kw.get("alibi") else None

    def run():
        o, lse = torch.full_like(q, float("nan")), torch.full((H, sum(lens)), float("nan"), device=DEV)
        a = N.AttnArgs()
        _ops._fill_common(a, q, k, v, o, _ops._THD, _ops._THD, batch=len(lens), sq=max(lens), sk=max(lens), hq=H, hkv=4, d=D, scale=D ** -0.5,
                          causal=False, wl=kw.get("wl", -1), wr=kw.get("wr", -1), softcap=kw.get("softcap", 0.0), alibi=sl, q_pos_offset=0,
                          impl=N.IMPL_AUTO, cu_q=cu, cu_k=cu)
        a.lse2 = lse.data_ptr()
        a.lse_stride = N._I64x3(0, 1, sum(lens))
        N.check(N.lib().fa_varlen_fwd(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "fa_varlen_fwd")
        return o, lse

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    want = run()
    for x, y in zip(got, want):
        assert not torch.isnan(y).any() and torch.equal(x, y)


def test_gradients_of_uneven_sequences():
    """The unpadded batch of an encoder: no mask, sequences of unequal length."""
    import flash_attn_triton_b200 as fa
    lens, H, D = UNEVEN[1], 16, 64
    q, k, v, do, cu, _ = cases.varlen_case(5, lens, lens, H, H, D)
    ts = [t.to(DEV).requires_grad_() for t in (q, k, v)]
    out = fa.flash_attn_varlen_func(*ts, cu.to(DEV), cu.to(DEV), max(lens), max(lens))
    grads = torch.autograd.grad(out, ts, do.to(DEV))
    for b in range(0, len(lens), 3):
        r = slice(int(cu[b]), int(cu[b + 1]))
        ro, _, *rg = orc.attention_grads_ref(q[None, r], k[None, r], v[None, r], do[None, r])
        assert maxdiff(out[r], ro[0]) <= util.FWD_TOL
        for a, w in zip(grads, rg):
            assert maxdiff(a[r], w[0]) <= util.GRAD_TOL


def test_rows_before_the_first_sequence():
    """With the value checks off a first sequence may start behind row 0: the rows before it belong to nobody."""
    import flash_attn_triton_b200 as fa
    first, lens, H = 700, [500] * 16, 16
    assert enough_tiles(len(lens) * 4, H)
    g = torch.Generator(DEV).manual_seed(1)
    q, k, v = (torch.randn(first + sum(lens), H, 64, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)
    run = lambda q, k, v, cu: fa.flash_attn_varlen_func(q, k, v, cu, cu, 500, 500, causal=True)
    want = run(*(t[first:].contiguous() for t in (q, k, v)), cu)
    fa.set_validation(False)
    try:
        got = run(q, k, v, cu + first)
    finally:
        fa.set_validation(True)
    assert torch.equal(got[first:], want)


@pytest.mark.parametrize("kw", [dict(causal=True), dict(window_size=(200, -1)), dict(window_size=(-1, 60)), dict(causal=True, softcap=20.0)], ids=str)
@pytest.mark.parametrize("D,H", [(64, 32), (128, 16)])
def test_order_by_weight_in_groups_of_heads(monkeypatch, D, H, kw):
    """Keys and values above 32 MB, so that the heads come in groups, in sequences too short for the persistent kernel: every tile is worked
    on once."""
    import flash_attn_triton_b200 as fa
    lens = [1500, 0, 1, 1900, 700, 128, 1031, 64]
    assert 4 * sum(lens) * H * D > 32 << 20 and max(lens) < 2048 and enough_tiles(sum(lens) // 128, H)
    g = torch.Generator(DEV).manual_seed(D)
    q, k, v = (torch.randn(sum(lens), H, D, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    cu = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32)
    run = lambda: fa.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), **kw)
    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())
