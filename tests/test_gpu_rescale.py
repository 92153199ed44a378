"""The one-tile forward where every key tile raises the row maxima, and each asks for the accumulator to be rescaled."""
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("Sk", [200, 1100])          # up to 255 keys, and at head_dim 256, every growth counts
def test_growing_maxima(D, Sk):
    from flash_attn_triton_b200 import _native as N, _ops
    q, k, v, _ = cases.dense_case(77, 1, 384, Sk, 2, 2, D)
    k = (k.float() * torch.linspace(3.0, 0.1, Sk)[None, :, None, None]).half()      # key tiles are visited from the last
    o, lse, _ = _ops.dense_forward(q.to(DEV), k.to(DEV), v.to(DEV), D ** -0.5, False, -1, -1, 0.0, None, 0, N.IMPL_TCGEN05,
                                   "bshd", True)
    ro, rl = orc.attention_ref(q, k, v)
    assert maxdiff(o, ro) <= util.FWD_TOL and maxdiff(lse * util.LN2, rl) <= util.FWD_TOL
    assert N.lib().fa_device_wait_status(0) == 0
