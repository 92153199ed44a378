"""The persistent forward over packed sequences of one or two query tiles: items whose second stream has no tile, or whose
group is far behind the other, hand their output entries on all the same."""
import numpy as np
import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("longest", [256, 2100])      # 2100: by the rule on lengths, among the short ones
def test_short_items_of_the_persistent_forward(monkeypatch, D, causal, longest):
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    lens = np.random.default_rng(1).integers(1, 257, size=64).tolist() + [longest]
    g = torch.Generator(DEV).manual_seed(D)
    q, k, v = (torch.randn(sum(lens), 16, D, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=DEV)
    run = lambda: fa.flash_attn_varlen_func(q, k, v, cu, cu, longest, longest, causal=causal)
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "0")         # one CTA per item
    want = run()
    monkeypatch.setenv("FA_B200_FWD_PERSISTENT_FROM", "1")
    for _ in range(20):
        assert torch.equal(run(), want)
    assert N.lib().fa_device_wait_status(0) == 0
