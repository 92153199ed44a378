"""Hand-over between the work items of the persistent backward kernels: items of one, two and a few tiles, many per CTA,
with every resource (K, V, ring slots, tensor memory, staged results) passed on from item to item."""
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,kw", [
    (40, 128, 128, 8, 8, dict(causal=True)),                   # one tile per item, three items per CTA
    (12, 200, 300, 8, 8, dict()),                              # two query tiles, three key tiles with a ragged end
    (6, 384, 384, 16, 16, dict(causal=True)),                  # items of three, two and one tile in turn
    (5, 130, 520, 16, 4, dict(causal=True)),                   # groups of four heads; key blocks that no query sees
    (4, 700, 700, 8, 8, dict(wl=100, wr=0)),                   # window: items of two tiles
])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_short_items(B, Sq, Sk, Hq, Hkv, kw, D, dtype):
    from flash_attn_triton_b200 import _native as N, _ops
    q, k, v, do = (t.to(dtype) for t in cases.dense_case(Sq + Sk + D, B, Sq, Sk, Hq, Hkv, D))
    causal, wl, wr = kw.get("causal", False), kw.get("wl", -1), kw.get("wr", -1)
    args = (D ** -0.5, causal, wl, wr, 0.0, None, 0)
    qd, kd, vd, dod = (t.to(DEV) for t in (q, k, v, do))
    o, lse, _ = _ops.dense_forward(qd, kd, vd, *args, N.IMPL_TCGEN05, "bshd", True)
    got = _ops.dense_backward(qd, kd, vd, o, lse, dod, *args, N.IMPL_TCGEN05, "bshd")
    again = _ops.dense_backward(qd, kd, vd, o, lse, dod, *args, N.IMPL_TCGEN05, "bshd")
    assert N.lib().fa_device_wait_status(0) == 0
    want = orc.attention_grads_ref(q, k, v, do, softmax_scale=D ** -0.5, causal=causal, window=(wl, wr))[2:]
    for a, b, r in zip(got, again, want):
        assert torch.equal(a, b)
        assert maxdiff(a, r) <= util.tols(dtype)[1]


@pytest.mark.parametrize("softcap,alibi", [(0.0, False), (0.0, True), (20.0, False), (20.0, True)])
@pytest.mark.parametrize("D", [64, 128])
def test_packed_items_with_options(softcap, alibi, D):
    """Packed sequences of one key to a few tiles, ends inside tiles, more items than CTAs; each set of score options is a
    kernel of its own."""
    import flash_attn_triton_b200 as fa
    lens = [1, 300, 128, 513, 64, 257, 400, 129, 700, 31, 256, 512]
    H = 8
    q, k, v, do, cu, _ = cases.varlen_case(11 + D, lens, lens, H, H, D)
    sl = torch.tensor([0.5 ** (i + 1) for i in range(H)]) if alibi else None
    ts = [t.to(DEV).requires_grad_() for t in (q, k, v)]
    out = fa.flash_attn_varlen_func(*ts, cu.to(DEV), cu.to(DEV), max(lens), max(lens), causal=True, softcap=softcap,
                                    alibi_slopes=None if sl is None else sl.to(DEV))
    grads = torch.autograd.grad(out, ts, do.to(DEV))
    for b in range(len(lens)):
        r = slice(int(cu[b]), int(cu[b + 1]))
        ro, _, *rg = orc.attention_grads_ref(q[None, r], k[None, r], v[None, r], do[None, r], causal=True, softcap=softcap,
                                             alibi_slopes=sl)
        assert maxdiff(out[r], ro[0]) <= util.FWD_TOL
        for a, w in zip(grads, rg):
            assert maxdiff(a[r], w[0]) <= util.GRAD_TOL


@pytest.mark.parametrize("wl", [0, 31, 32, 95, 127, 161])
@pytest.mark.parametrize("softcap,alibi", [(20.0, True), (0.0, True), (0.0, False)])
@pytest.mark.parametrize("D", [64, 128])
def test_masks_that_end_in_each_column_group(wl, softcap, alibi, D):
    """Windows and a diagonal that cross the columns of every element-wise thread (64 of a tile, 32 with score options)."""
    from flash_attn_triton_b200 import _native as N, _ops
    B, S, H = 2, 417, 2
    q, k, v, do = cases.dense_case(wl + D, B, S, S, H, H, D)
    sl = torch.tensor([0.25, 0.0625]) if alibi else None
    args = (D ** -0.5, True, wl, -1, softcap, None if sl is None else sl.to(DEV).repeat(B, 1), 0)
    qd, kd, vd, dod = (t.to(DEV) for t in (q, k, v, do))
    o, lse, _ = _ops.dense_forward(qd, kd, vd, *args, N.IMPL_TCGEN05, "bshd", True)
    got = _ops.dense_backward(qd, kd, vd, o, lse, dod, *args, N.IMPL_TCGEN05, "bshd")
    assert N.lib().fa_device_wait_status(0) == 0
    want = orc.attention_grads_ref(q, k, v, do, softmax_scale=D ** -0.5, causal=True, window=(wl, -1), softcap=softcap,
                                   alibi_slopes=sl)[2:]
    for a, r in zip(got, want):
        assert maxdiff(a, r) <= util.GRAD_TOL
