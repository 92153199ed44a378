"""Problems of less than a tile, and just around one, through the automatic choice of kernels."""
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,Hq,Hkv,causal", [
    (1, 1, 2, 2, True), (1, 130, 2, 1, False), (17, 3, 2, 2, True), (16, 16, 4, 1, True), (127, 127, 2, 2, False),
    (128, 128, 2, 1, True), (129, 129, 2, 2, True), (200, 255, 2, 2, False)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dense(Sq, Sk, Hq, Hkv, causal, D, dtype):
    import flash_attn_triton_b200 as fa
    q, k, v, do = (t.to(dtype) for t in cases.dense_case(Sq + Sk, 2, Sq, Sk, Hq, Hkv, D))
    out, dq, dk, dv = util.run_dense(fa.flash_attn_func, q, k, v, do, causal=causal)
    ro, _, rdq, rdk, rdv = orc.attention_grads_ref(q, k, v, do, causal=causal)
    f, g = util.tols(dtype)
    assert maxdiff(out, ro) <= f
    for n, a, b in (("dq", dq, rdq), ("dk", dk, rdk), ("dv", dv, rdv)):
        assert maxdiff(a, b) <= g, n


def test_packed_short_sequences():
    import flash_attn_triton_b200 as fa
    lens = [1, 40, 0, 127, 3]
    q, k, v, do, cu, _ = cases.varlen_case(9, lens, lens, 4, 2, 64)
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    sl = torch.tensor([0.5, 0.25, 0.125, 0.0625])
    out = fa.flash_attn_varlen_func(qd, kd, vd, cu.to(DEV), cu.to(DEV), 127, 127, causal=True, softcap=10.0,
                                    alibi_slopes=sl.to(DEV))
    got = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    for b, n in enumerate(lens):
        if n == 0:
            continue
        a = sum(lens[:b])
        ref = orc.attention_grads_ref(*(t[None, a:a + n] for t in (q, k, v, do)), causal=True, softcap=10.0, alibi_slopes=sl)
        assert maxdiff(out[a:a + n], ref[0][0]) <= util.FWD_TOL
        for name, x, y in zip(("dq", "dk", "dv"), got, ref[2:]):
            assert maxdiff(x[a:a + n], y[0]) <= util.GRAD_TOL, name
