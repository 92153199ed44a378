"""Packed q/k/v and k/v: read in place, gradients written into packed tensors."""
import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


def fa():
    import flash_attn_triton_b200 as m
    return m


def placed(shape, how):
    """A random leaf-to-be of this shape: dense, off a 16-byte boundary, or with padded or odd strides."""
    n = torch.Size(shape).numel()
    if how == "dense":
        return torch.randn(shape, device=DEV, dtype=torch.half)
    if how == "misaligned":
        return torch.randn(n + 1, device=DEV, dtype=torch.half)[1:].view(shape)
    if how == "padded":          # rows of head_dim inside wider ones, still multiples of 8
        return torch.randn(*shape[:-1], shape[-1] + 8, device=DEV, dtype=torch.half)[..., :shape[-1]]
    if how == "odd":             # a pitch that is no multiple of 8
        return torch.randn(*shape[:-1], shape[-1] + 1, device=DEV, dtype=torch.half)[..., :shape[-1]]
    if how == "heads_first":     # (batch, heads, packed, rows, dim) in memory
        b, s, p, h, d = shape
        return torch.randn(b, h, p, s, d, device=DEV, dtype=torch.half).permute(0, 3, 2, 1, 4)
    raise ValueError(how)


@pytest.mark.parametrize("how", ["dense", "misaligned", "padded", "odd", "heads_first"])
@pytest.mark.parametrize("B,S,H,D", [(2, 200, 4, 64), (1, 300, 2, 128), (2, 64, 3, 32), (1, 2, 2, 64)])
@pytest.mark.parametrize("packing", ["qkv", "kv"])
def test_same_as_separate_tensors(packing, B, S, H, D, how):
    torch.manual_seed(S)
    P = 3 if packing == "qkv" else 2
    x = placed((B, S, P, H, D), how).requires_grad_()
    q = torch.randn(B, S, H, D, device=DEV, dtype=torch.half, requires_grad=True)
    do = torch.randn(B, S, H, D, device=DEV, dtype=torch.half)
    if packing == "qkv":
        out, wrt = fa().flash_attn_qkvpacked_func(x, causal=True), (x,)
    else:
        out, wrt = fa().flash_attn_kvpacked_func(q, x, causal=True), (q, x)
    got = torch.autograd.grad(out, wrt, do)
    parts = [t.contiguous().clone().detach().requires_grad_() for t in x.unbind(2)]
    if packing == "kv":
        parts.insert(0, q)
    want_out = fa().flash_attn_func(*parts, causal=True)
    want = torch.autograd.grad(want_out, parts, do)
    assert torch.equal(out, want_out)
    assert torch.equal(got[-1], torch.stack(want[-P:], dim=2))
    if packing == "kv":
        assert torch.equal(got[0], want[0])
