"""Dropout on the tcgen05 kernels: the mask drawn once as bits (dropout_bits.cu) and read by the forward, dQ and
dK/dV kernels."""
import ctypes as C
import random

import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu


def bits_of(words, rows, cols):
    """(rows, words) int32 -> bool (rows, cols)"""
    b = (words.view(rows, -1, 1) >> torch.arange(32, dtype=torch.int32)) & 1
    return b.reshape(rows, -1)[:, :cols].bool()


@pytest.mark.parametrize("Sq,Sk,p", [(128, 256, 0.1), (129, 257, 0.5), (300, 900, 0.2), (640, 321, 0.999)])
def test_bits_are_the_reference_stream(Sq, Sk, p):
    from flash_attn_triton_b200 import _native as N
    t = torch.zeros(1, max(Sq, Sk), 1, 64, dtype=torch.half, device=DEV)
    a = N.AttnArgs()
    a.batch, a.seqlen_q, a.seqlen_k, a.heads_q, a.heads_kv, a.head_dim = 1, Sq, Sk, 1, 1, 64
    a.q = a.k = a.v = a.o = t.data_ptr()
    a.softmax_scale, a.window_left, a.window_right = 0.125, -1, -1
    a.dropout_p, a.dropout_seed, a.dropout_row_stride = p, (5 << 32) | 1234567, 960
    n = N.lib().fa_dropout_bits_bytes(C.byref(a), 0)
    mt, nt = -(-Sq // 128), -(-Sk // 128)
    assert n == 2 * mt * nt * 128 * 128 // 8
    buf = torch.zeros(n // 4, dtype=torch.int32, device=DEV)
    N.check(N.lib().fa_dropout_bits(C.byref(a), buf.data_ptr(), N.stream_ptr(buf.device)), "fa_dropout_bits")
    rows, cols = buf.cpu().chunk(2)
    keep = orc.dropout_keep_ref(Sq, Sk, p, (5 << 32) | 1234567, 960)
    assert torch.equal(bits_of(rows, mt * 128, Sk)[:Sq], keep)
    assert torch.equal(bits_of(cols, nt * 128, Sq)[:Sk], keep.T)


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,D,kw", [
    (2, 128, 256, 2, 2, 64, dict()),                                  # the smallest the rule takes
    (1, 257, 257, 2, 1, 128, dict(causal=True)),                      # one row, one key past the tiles
    (1, 300, 1000, 4, 2, 64, dict(causal=True)),
    (1, 700, 321, 2, 2, 128, dict(causal=True, window=(130, -1))),    # query tiles that see few keys
    (1, 70, 513, 2, 2, 64, dict()),                                   # one short query tile
    (2, 100, 90, 4, 2, 128, dict(causal=True)),                       # forward drawn per score, backward on bits
    (1, 2200, 2100, 1, 1, 64, dict(window=(300, 200))),               # longer than the persistent forward starts at
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dropout_on_tcgen05_vs_oracle(B, Sq, Sk, Hq, Hkv, D, kw, dtype):
    import flash_attn_triton_b200 as fa
    q, k, v, do = (t.to(dtype) for t in cases.dense_case(Sq + Sk, B, Sq, Sk, Hq, Hkv, D))
    call = dict(causal=kw.get("causal", False), window_size=kw.get("window", (-1, -1)))
    random.seed(11)
    seed = random.randrange(2 ** 31 - 1)
    random.seed(11)
    out, dq, dk, dv = util.run_dense(fa.flash_attn_func, q, k, v, do, dropout_p=0.25, **call)
    ro, _, _, rdq, rdk, rdv = orc.attention_dropout_ref(q, k, v, do, dropout_p=0.25, seed=seed, **kw)
    f, g = util.tols(dtype)
    amp = 1.0 / 0.75              # kept entries, and their rounding errors, are scaled by this
    assert maxdiff(out, ro) <= f * amp
    for n, a, b in (("dq", dq, rdq), ("dk", dk, rdk), ("dv", dv, rdv)):
        assert maxdiff(a, b) <= g * amp, n


@pytest.mark.parametrize("D", [64, 128])
def test_every_probability_meets_its_own_bit(D):
    """Equal scores and one-hot values: the output is the mask itself, key by key."""
    import flash_attn_triton_b200 as fa
    Sq, Sk = 260, 384
    q = torch.zeros(1, Sq, 1, D, dtype=torch.half, device=DEV)
    k = torch.zeros(1, Sk, 1, D, dtype=torch.half, device=DEV)
    for k0 in range(0, Sk, D):
        v = torch.zeros(1, Sk, 1, D, dtype=torch.half, device=DEV)
        v[0, k0:k0 + D, 0] = torch.eye(D, dtype=torch.half, device=DEV)
        random.seed(3)
        seed = random.randrange(2 ** 31 - 1)
        random.seed(3)
        out = fa.flash_attn_func(q, k, v, dropout_p=0.3)
        keep = orc.dropout_keep_ref(Sq, Sk, 0.3, seed, 384)[:, k0:k0 + D]
        assert torch.equal(out[0, :, 0].cpu() > 0, keep)
