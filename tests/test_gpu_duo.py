"""The forward with two CTAs per SM against the two-tile kernel: bit for bit the same, whatever the options, head groups,
ragged ends and strides."""
import random

import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(causal=True), dict(), dict(window_size=(150, 0)), dict(window_size=(60, 90)),
    dict(causal=True, softcap=20.0), dict(alibi=True), dict(causal=True, alibi=True, window_size=(200, -1)),
    dict(causal=True, dropout_p=0.2), dict(dropout_p=0.1),
], ids=str)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,Hkv,packed", [(400, 400, 16, True), (385, 640, 4, False)])
def test_two_ctas_against_two_tiles(monkeypatch, kw, D, Sq, Sk, Hkv, packed):
    import flash_attn_triton_b200 as fa
    kw = dict(kw)
    g = torch.Generator(DEV).manual_seed(D)
    q = torch.randn(10, Sq, 16, D, device=DEV, dtype=torch.half, generator=g)
    kv = torch.randn(10, Sk, 2, Hkv, D, device=DEV, dtype=torch.half, generator=g)      # k and v: slices of one tensor
    k, v = kv[:, :, 0], kv[:, :, 1]
    if kw.pop("alibi", False):
        kw["alibi_slopes"] = torch.tensor([0.5 ** (i + 1) for i in range(16)], device=DEV)

    def run():
        random.seed(3)                                                                   # the dropout mask
        return fa.flash_attn_func(q, k, v, **kw)

    got = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")
    assert torch.equal(got, run())
