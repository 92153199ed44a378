"""Row statistics of the tcgen05 dK/dV kernels (bwd_stats.cuh): as exact as the fp32 of the mma.sync kernels, at any size."""
import math

import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def grads(q, k, v, do, scale, causal, feat=None, softcap=0.0):
    """Gradients by (the automatic choice, the mma.sync kernels), from one forward."""
    from flash_attn_triton_b200 import _native as N, _ops
    args = (scale, causal, -1, -1, softcap, None, 0)
    o, lse, _ = _ops.dense_forward(q, k, v, *args, N.IMPL_AUTO, "bshd", True, feat)
    return [_ops.dense_backward(q, k, v, o, lse, do, *args, impl, "bshd", feat) for impl in (N.IMPL_AUTO, N.IMPL_MMA)], (o, lse)


SHAPES = [(64, 64), (127, 250), (300, 300), (1024, 1024)]


@pytest.mark.parametrize("Sq,Sk", SHAPES)
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("variant", ["plain", "dropout", "softcap"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_delta_beyond_sixteen_bits(Sq, Sk, D, variant, dtype):
    """Values with a common offset and gradients as loss scaling leaves them: delta is far above 65504, and dP with it;
    their difference is not.  Both kernels round P and dS to 16 bits once (2^-12 or 2^-9 at most, half of that on
    average); where dP and delta cancel, fp32 leaves 2^-24 of 4e5 in each, against differences of some hundred."""
    from flash_attn_triton_b200 import _ops
    g = torch.Generator(DEV).manual_seed(Sq)
    mk = lambda s: torch.randn(2, s, 2, D, device=DEV, dtype=dtype, generator=g)
    q, k, v, do = mk(Sq), mk(Sk), mk(Sk) * 8 + 200, mk(Sq).abs() * 8 + 8
    feat = _ops.Features(dropout_p=0.25, seed=5, row_stride=1024) if variant == "dropout" else None
    # dropout without a mask: with only a few keys the share of them that is kept is far from 1 - p, and dS of a row, which
    # grows with the values' offset, passes 65504 in either kernel
    (got, want), (o, _) = grads(q, k, v, do, D ** -0.5, variant != "dropout", feat, 30.0 if variant == "softcap" else 0.0)
    assert (o.double() * do.double()).sum(-1).abs().max() > 1.5 * 65504
    tol = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    if variant == "softcap":
        tol += 2.0 ** -8           # the two tanh differ by up to 2^-11 of the score
    for a, b in zip(got, want):
        assert torch.isfinite(a).all() and rel(a, b) <= tol


@pytest.mark.parametrize("Sq,Sk", SHAPES)
@pytest.mark.parametrize("scale,size", [(None, 1.0), (None, 16.0), (1e-4, 300.0), (3.0, 1.0)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_errors_are_those_of_fp32_statistics(Sq, Sk, scale, size, dtype):
    """Large and small LSE, scales far from the usual one: against float64, not above the mma.sync kernels by more than what
    another order of the same sums moves it (under 0.1 % over seeds; the bound is 0.5 %)."""
    D = 128
    scale = scale or D ** -0.5
    g = torch.Generator(DEV).manual_seed(Sk)
    mk = lambda s, f=1.0: (torch.randn(2, s, 4, D, device=DEV, generator=g) * f).to(dtype)
    q, k, v, do = mk(Sq, size), mk(Sk), mk(Sk), mk(Sq)
    (got, want), _ = grads(q, k, v, do, scale, True)
    x = [t.double().requires_grad_() for t in (q, k, v)]
    s = torch.einsum("bihd,bjhd->bhij", x[0], x[1]) * scale
    s = s.masked_fill(torch.arange(Sk, device=DEV) > torch.arange(Sq, device=DEV)[:, None], -math.inf)
    ref = torch.autograd.grad(torch.einsum("bhij,bjhd->bihd", s.softmax(-1), x[2]), x, do.double())
    for a, b, r in zip(got, want, ref):
        assert rel(a, r) <= 1.005 * rel(b, r)


def test_a_delta_that_is_not_finite_stays_in_its_gradient():
    """It reaches dQ and dK, as fp32 arithmetic has it, and leaves dV (of the same row) finite."""
    from flash_attn_triton_b200 import _native as N, _ops
    g = torch.Generator(DEV).manual_seed(0)
    q, k, v, do = (torch.randn(1, 300, 1, 64, device=DEV, dtype=torch.half, generator=g) for _ in range(4))
    args = (0.125, True, -1, -1, 0.0, None, 0)
    o, lse, _ = _ops.dense_forward(q, k, v, *args, N.IMPL_AUTO, "bshd", True)
    o = o.clone()
    o[0, 150, 0, 0] = float("inf")
    for impl in (N.IMPL_AUTO, N.IMPL_MMA):
        dq, dk, dv = _ops.dense_backward(q, k, v, o, lse, do, *args, impl, "bshd")
        assert not torch.isfinite(dk[0, :151]).any() and torch.isfinite(dv).all() and not torch.isfinite(dq[0, 150]).any()
