"""Packed variable-length attention parity (forward and backward)."""
import numpy as np
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, LN2, maxdiff

pytestmark = pytest.mark.gpu


def fa():
    import flash_attn_triton_b200 as m
    return m


def run_varlen(q, k, v, do, cu_q, cu_k, max_q, max_k, **kw):
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    out = fa().flash_attn_varlen_func(qd, kd, vd, cu_q.to(DEV), cu_k.to(DEV), max_q, max_k, **kw)
    dq, dk, dv = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    return out.detach().cpu(), dq.cpu(), dk.cpu(), dv.cpu()


def test_golden_varlen_all(golden):
    """3 sequences, GQA 4/2, causal + window + ALiBi + softcap: reference output, base-2
    LSE and gradients."""
    from flash_attn_triton_b200 import _native as N, _ops
    g = golden("varlen_all")
    ql, kl = g["q_lens"].tolist(), g["k_lens"].tolist()
    q, k, v, do, cu_q, cu_k = cases.varlen_case(7, ql, kl, 4, 2, 64)
    assert cases.checksum(q, k, v, do) == str(g["checksum"])
    sl = torch.from_numpy(g["slopes"])
    out, dq, dk, dv = run_varlen(q, k, v, do, cu_q, cu_k, 130, 130, softmax_scale=0.125,
                                 causal=True, window_size=(48, 0), softcap=30.0,
                                 alibi_slopes=sl.to(DEV))
    assert maxdiff(out, g["out"]) <= util.FWD_TOL
    for n, t in (("dq", dq), ("dk", dk), ("dv", dv)):
        assert maxdiff(t, g[n]) <= util.GRAD_TOL, n
    al = sl[None].expand(3, -1).contiguous().to(DEV)
    _, lse, _ = _ops.varlen_forward(q.to(DEV), k.to(DEV), v.to(DEV), cu_q.to(DEV), cu_k.to(DEV),
                                    130, 130, 0.125, True, 48, 0, 30.0, al, N.IMPL_AUTO, True)
    assert maxdiff(lse.transpose(0, 1), g["lse2"]) <= util.FWD_TOL


def test_golden_varlen_rect(golden):
    g = golden("varlen_rect")
    q, k, v, do, cu_q, cu_k = cases.varlen_case(8, [3, 5], [4, 6], 2, 2, 16)
    out = fa().flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu_q.to(DEV), cu_k.to(DEV),
                                      5, 6, causal=True)
    assert maxdiff(out, g["out"]) <= util.FWD_TOL


CASES = [
    # q_lens, k_lens, Hq, Hkv, D, kwargs
    ([5, 70, 1, 130], [5, 70, 1, 130], 4, 4, 64, dict(causal=True)),
    ([64, 0, 33], [64, 0, 33], 2, 1, 128, dict(causal=True)),
    ([10, 20, 30], [40, 5, 64], 4, 2, 32, dict()),
    ([10, 20], [0, 7], 2, 2, 64, dict(causal=True)),
    ([200, 129], [200, 129], 8, 2, 128, dict(causal=True, window_size=(50, 0), softcap=30.0,
                                              alibi="heads")),
    ([17, 260], [17, 260], 2, 2, 256, dict(window_size=(7, 9))),
    ([33], [33], 2, 2, 16, dict(causal=True)),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_varlen_vs_oracle(case):
    ql, kl, Hq, Hkv, D, kw = CASES[case]
    kw = dict(kw)
    q, k, v, do, cu_q, cu_k = cases.varlen_case(50 + case, ql, kl, Hq, Hkv, D)
    okw = dict(causal=kw.get("causal", False), window=kw.get("window_size", (-1, -1)),
               softcap=kw.get("softcap", 0.0))
    if kw.pop("alibi", None):
        sl = torch.tensor([2.0 ** (-8 * (i + 1) / Hq) for i in range(Hq)])
        kw["alibi_slopes"] = sl.to(DEV)
        okw["alibi_slopes"] = sl
    out, dq, dk, dv = run_varlen(q, k, v, do, cu_q, cu_k, max(ql), max(kl), **kw)
    ro, _, rdq, rdk, rdv = orc.varlen_attention_grads_ref(q, k, v, do, cu_q, cu_k, **okw)
    assert maxdiff(out, ro) <= util.FWD_TOL
    assert maxdiff(dq, rdq) <= util.GRAD_TOL
    assert maxdiff(dk, rdk) <= util.GRAD_TOL
    assert maxdiff(dv, rdv) <= util.GRAD_TOL


def test_packed_variants_and_options():
    m = fa()
    ql = [12, 40]
    q, k, v, do, cu, _ = cases.varlen_case(70, ql, ql, 2, 2, 64)
    ro, _ = orc.varlen_attention_ref(q, k, v, cu, cu, causal=True)
    qkv = torch.stack((q, k, v), dim=1).to(DEV)
    assert maxdiff(m.flash_attn_varlen_qkvpacked_func(qkv, cu.to(DEV), 40, causal=True), ro) <= util.FWD_TOL
    kv = torch.stack((k, v), dim=1).to(DEV)
    assert maxdiff(m.flash_attn_varlen_kvpacked_func(q.to(DEV), kv, cu.to(DEV), cu.to(DEV), 40, 40,
                                                     causal=True), ro) <= util.FWD_TOL
    # deterministic=True is the same computation
    o2 = m.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), cu.to(DEV), 40, 40,
                                  causal=True, deterministic=True)
    assert maxdiff(o2, ro) <= util.FWD_TOL
    # return_attn_probs: natural-log lse padded with -inf
    o3, lse, probs = m.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV),
                                              cu.to(DEV), 40, 40, causal=True, return_attn_probs=True)
    assert maxdiff(o3, ro) <= util.FWD_TOL and lse.shape == (2, 2, 40) and torch.isinf(lse[0, :, 12:]).all()
    # seqused_k trims each sequence's keys
    o4 = m.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), cu.to(DEV), 40, 40,
                                  seqused_k=[6, 20])
    kk = torch.cat([k[0:6], k[12:32]])
    vv = torch.cat([v[0:6], v[12:32]])
    r4, _ = orc.varlen_attention_ref(q, kk, vv, cu, torch.tensor([0, 6, 26]))
    assert maxdiff(o4, r4) <= util.FWD_TOL
    # paged k/v
    page = 16
    pool_k = torch.zeros(8, page, 2, 64, dtype=torch.float16)
    pool_v = torch.zeros(8, page, 2, 64, dtype=torch.float16)
    table = torch.tensor([[5, 0, 0], [2, 7, 1]], dtype=torch.int32)
    for b, (s, e) in enumerate(((0, 12), (12, 52))):
        for t in range(s, e):
            pg = table[b, (t - s) // page]
            pool_k[pg, (t - s) % page] = k[t]
            pool_v[pg, (t - s) % page] = v[t]
    o5 = m.flash_attn_varlen_func(q.to(DEV), pool_k.to(DEV), pool_v.to(DEV), cu.to(DEV), cu.to(DEV),
                                  40, 40, causal=True, block_table=table.to(DEV))
    assert maxdiff(o5, ro) <= util.FWD_TOL
    # value errors
    with pytest.raises(ValueError):
        m.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), cu.to(DEV), 10, 40)
    bad = torch.tensor([0, 30, 20], dtype=torch.int32, device=DEV)
    with pytest.raises(ValueError):
        m.flash_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), bad, bad, 40, 40)
    z = m.flash_attn_varlen_func(q[:0].to(DEV), k[:0].to(DEV), v[:0].to(DEV),
                                 torch.zeros(3, dtype=torch.int32, device=DEV),
                                 torch.zeros(3, dtype=torch.int32, device=DEV), 0, 0)
    assert z.shape == (0, 2, 64)


def test_config3_shape_reduced_and_full():
    """32 sequences, H32 D128, causal + window 1024 + ALiBi + softcap 30.  The oracle checks
    two whole sequences of a reduced-head run; the full-size run is checked through
    properties (finite, rows of V=1 give 1, agreement of the shared sequences)."""
    m = fa()
    rng = np.random.default_rng(3)
    lens = (64 * rng.integers(4, 65, size=32)).tolist()
    H, D = 32, 128
    T = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(3)
    q = torch.randn(T, H, D, device=DEV, dtype=torch.float16, generator=g)
    k = torch.randn(T, H, D, device=DEV, dtype=torch.float16, generator=g)
    v = torch.randn(T, H, D, device=DEV, dtype=torch.float16, generator=g)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=DEV)
    sl = torch.tensor([2.0 ** (-8 * (i + 1) / H) for i in range(H)], device=DEV)
    kw = dict(causal=True, window_size=(1024, 0), alibi_slopes=sl, softcap=30.0)
    do = torch.randn(T, H, D, device=DEV, dtype=torch.float16, generator=g)
    qg, kg, vg = (t.detach().requires_grad_() for t in (q, k, v))
    out = m.flash_attn_varlen_func(qg, kg, vg, cu, cu, max(lens), max(lens), **kw)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), do)
    out = out.detach()
    assert torch.isfinite(out).all() and all(torch.isfinite(t).all() for t in (dq, dk, dv))
    ones = m.flash_attn_varlen_func(q, k, torch.ones_like(v), cu, cu, max(lens), max(lens), **kw)
    assert (ones.float() - 1).abs().max().item() <= 2e-3
    # shortest, longest, first and last sequence against the oracle, 2 heads: output and gradients
    # (every head has its own K/V here, so a head's slice of the gradients is self-contained)
    for b in sorted({int(np.argmin(lens)), int(np.argmax(lens)), 0, len(lens) - 1}):
        s, e = int(cu[b]), int(cu[b + 1])
        hs = [0, H - 1]
        ro, _, rdq, rdk, rdv = orc.attention_grads_ref(
            q[s:e, hs].cpu()[None], k[s:e, hs].cpu()[None], v[s:e, hs].cpu()[None], do[s:e, hs].cpu()[None],
            causal=True, window=(1024, 0), softcap=30.0, alibi_slopes=sl[hs].cpu())
        assert maxdiff(out[s:e, hs], ro[0]) <= util.FWD_TOL, b
        for n, a, r in (("dq", dq, rdq), ("dk", dk, rdk), ("dv", dv, rdv)):
            assert maxdiff(a[s:e, hs], r[0]) <= util.GRAD_TOL, (b, n)


@pytest.mark.parametrize("batch", [1, 128, 129, 1024, 2500])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_values_of_cu_seqlens_are_checked(batch, dtype):
    """Every value check, at the first, a middle and the last sequence, in both arrays; with dropout they are made by themselves.
    What is refused in several ways is refused for the first of them, and the call after a refused one works."""
    total, H, D = 4 * batch, 1, 16
    q, k, v = (torch.randn(total, H, D, device=DEV, dtype=torch.half) for _ in range(3))
    good = torch.arange(0, total + 1, 4, dtype=dtype, device=DEV)

    def call(cu_q, cu_k, max_q=4, max_k=4, **kw):
        return fa().flash_attn_varlen_func(q, k, v, cu_q, cu_k, max_q, max_k, **kw)

    def refused(text, *args, **kw):
        for more in (dict(), dict(dropout_p=0.5)):
            with pytest.raises(ValueError, match=text):
                call(*args, **kw, **more)

    want = call(good, good)
    for which in (0, 1):
        def bad(i, x):
            cu = good.clone()
            cu[i] = x
            return (cu, good) if which == 0 else (good, cu)
        refused("start at zero", *bad(0, 1))
        refused("cover the packed", *bad(batch, total + 1), max_q=9, max_k=9)
        for i in {1, batch // 2, batch - 1} - {0, batch}:
            refused("non-decreasing", *bad(i, total + 7))
            refused("cover every packed sequence", *bad(i, 4 * i + 1))
    refused("cover every packed sequence", good, good, max_q=3)
    refused("cover every packed sequence", good, good, max_k=3)
    if batch > 1:
        both = good.clone()
        both[0], both[1] = 1, 0
        refused("start at zero", both, good, max_q=1)
    assert torch.equal(call(good, good), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert torch.equal(call(good, good), want)
        refused("cover every packed sequence", good, good, max_q=3)
    torch.cuda.current_stream().wait_stream(side)


def test_what_the_values_are_refused_for_comes_first():
    """Calls that are wrong in two ways: cu_seqlens, and something that is looked at behind them."""
    import torch.autograd.forward_ad as fwad
    q = torch.randn(64, 2, 64, device=DEV, dtype=torch.half)
    good = torch.tensor([0, 30, 64], dtype=torch.int32, device=DEV)
    bad = torch.tensor([1, 30, 64], dtype=torch.int32, device=DEV)
    call = lambda cu, x=q, **kw: fa().flash_attn_varlen_func(x, q, q, cu, good, 34, 34, **kw)
    want = call(good)
    slopes = torch.ones(3, device=DEV)
    for kw, own in ((dict(alibi_slopes=slopes), ValueError), (dict(window_size=(3,)), IndexError), (dict(window_size=("a", 1)), TypeError),
                    (dict(softmax_scale="a"), TypeError)):
        with pytest.raises(ValueError, match="start at zero"):
            call(bad, **kw)
        with pytest.raises(own) as e:
            call(good, **kw)
        assert "start at zero" not in str(e.value)
    with fwad.dual_level():
        x = fwad.make_dual(q, torch.ones_like(q))
        with pytest.raises(ValueError, match="start at zero"):
            call(bad, x)
        with pytest.raises(NotImplementedError):
            call(good, x)
    assert torch.equal(call(good), want)


@pytest.mark.parametrize("where", ["cpu", DEV])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.int16])
def test_longest_sequence_as_a_tensor(dtype, where):
    """max_seqlen as `(cu[1:] - cu[:-1]).max()` leaves it: one that is too small is refused in any type, with dropout too."""
    q = torch.randn(64, 2, 64, device=DEV, dtype=torch.half)
    cu = torch.tensor([0, 30, 64], dtype=torch.int32, device=DEV)
    n = lambda x: torch.tensor(x, dtype=dtype, device=where)
    want = fa().flash_attn_varlen_func(q, q, q, cu, cu, 34, 34)
    assert torch.equal(fa().flash_attn_varlen_func(q, q, q, cu, cu, n(34), n(34)), want)
    for more in (dict(), dict(dropout_p=0.5)):
        for lengths in ((n(33), n(34)), (n(34), n(33)), (33, n(34))):
            with pytest.raises(ValueError, match="cover every packed sequence"):
                fa().flash_attn_varlen_func(q, q, q, cu, cu, *lengths, **more)


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_value_checks_are_refused_under_capture():
    q = torch.randn(64, 2, 64, device=DEV, dtype=torch.half)
    cu = torch.tensor([0, 30, 64], dtype=torch.int32, device=DEV)
    call = lambda: fa().flash_attn_varlen_func(q, q, q, cu, cu, 34, 34)
    want = call()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            call()
    assert torch.equal(call(), want)
    fa().set_validation(False)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = call()
        graph.replay()
    finally:
        fa().set_validation(True)
    assert torch.equal(out, want)


def test_tickets_of_value_checks():
    """As many tickets as there are: the next check is not taken, calls go on, and a ticket is handed in once."""
    import ctypes as C
    from flash_attn_triton_b200 import _native as N
    lib, cu, out = N.lib(), torch.tensor([0, 30, 64], dtype=torch.int32, device=DEV), []
    q = torch.randn(64, 2, 64, device=DEV, dtype=torch.half)
    ticket, failed, stream = C.c_int32(), C.c_uint32(), N.stream_ptr(q.device)
    want = fa().flash_attn_varlen_func(q, q, q, cu, cu, 34, 34)

    def issue(longest):
        return lib.fa_varlen_check(cu.data_ptr(), cu.data_ptr(), 2, 64, 64, 0, longest, 34, 0, C.byref(ticket), stream)

    for i in range(128):
        assert issue(34 - i % 2) == 0
        out.append(ticket.value)
    assert issue(34) == -2                               # FA_ERR_UNSUPPORTED, without a wait
    assert torch.equal(fa().flash_attn_varlen_func(q, q, q, cu, cu, 34, 34), want)
    with pytest.raises(ValueError, match="cover every packed sequence"):
        fa().flash_attn_varlen_func(q, q, q, cu, cu, 34, 33)
    lens = torch.tensor([5], dtype=torch.int32, device=DEV)
    cache = torch.zeros(1, 64, 2, 64, device=DEV, dtype=torch.half)
    fa().flash_attn_with_kvcache(q[None, :1], cache, cache.clone(), cache_seqlens=lens)      # a call with a word of its own
    for i, t in enumerate(out):
        assert lib.fa_check_result(t, C.byref(failed), stream) == 0
        assert failed.value == (8 if i % 2 else 0)       # FA_VARLEN_LONGEST
    for t in out:
        assert lib.fa_check_result(t, C.byref(failed), stream) == -1
    assert issue(34) == 0
    assert lib.fa_check_result(ticket.value, C.byref(failed), stream) == 0 and failed.value == 0
