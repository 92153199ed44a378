"""Packed forwards whose grid is a list of tiles: more sequences than lanes of a warp, empty ones, ends inside and on
the edge of a tile."""
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu

LENS = {
    "one": [130],
    "empty": [0, 256, 0, 0, 129, 1, 0],
    "many": [(37 * i * i) % 300 for i in range(70)],       # the search takes three sequences per lane, then one; some without a tile
    "long_last": [1] * 33 + [513],
    "same_length": [128] * 40,                              # an entry for each: nothing to search
    "two_steps": [(7 * i) % 40 for i in range(1100)] + [300, 0, 129],
}


@pytest.mark.parametrize("name", list(LENS))
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_tiles(name, D, causal):
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    lens = LENS[name]
    q, k, v, _, cu, _ = cases.varlen_case(3 + D, lens, lens, 2, 1, D)
    out = fa.flash_attn_varlen_func(*(t.to(DEV) for t in (q, k, v)), cu.to(DEV), cu.to(DEV), max(lens), max(lens), causal=causal)
    assert N.lib().fa_device_wait_status(0) == 0
    for b, n in enumerate(lens):
        if n:
            r = slice(int(cu[b]), int(cu[b + 1]))
            ro, _ = orc.attention_ref(q[None, r], k[None, r], v[None, r], causal=causal)
            assert maxdiff(out[r], ro[0]) <= util.FWD_TOL, (b, n)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_packed_sequence_has_the_result_of_a_dense_call(D, dtype):
    """The kernel of a packed call follows from its lengths together; the result of a sequence does not."""
    import flash_attn_triton_b200 as fa
    lens = [700, 256, 1500, 300, 129]
    q, k, v, _, cu, _ = cases.varlen_case(19, lens, lens, 4, 2, D)
    q, k, v = (2 * t.to(DEV, dtype) for t in (q, k, v))
    out = fa.flash_attn_varlen_func(q, k, v, cu.to(DEV), cu.to(DEV), max(lens), max(lens), causal=True)
    for b, n in enumerate(lens):
        if n >= 256:                 # shorter dense calls rescale at every growth of a maximum
            r = slice(int(cu[b]), int(cu[b + 1]))
            assert torch.equal(out[r], fa.flash_attn_func(q[None, r], k[None, r], v[None, r], causal=True)[0])
