"""The autograd node of the attention calls (csrc/host_ext.cpp) under what PyTorch does with nodes."""
import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


def mk(*s, seed=0):
    g = torch.Generator(DEV).manual_seed(seed + sum(s))
    return torch.randn(*s, device=DEV, dtype=torch.half, generator=g)


def fa():
    import flash_attn_triton_b200 as m
    return m


def varlen(q, k, v, cu, **kw):
    return fa().flash_attn_varlen_func(q, k, v, cu, cu, 156, 156, **kw)


@pytest.mark.parametrize("side", ["cu_seqlens", "alibi", "used"])
def test_side_tensor_changed_in_place_is_refused(side):
    q, k, v = (mk(256, 4, 64, seed=i).requires_grad_() for i in range(3))
    cu = torch.tensor([0, 100, 256], dtype=torch.int32, device=DEV)
    used = torch.tensor([90, 156], dtype=torch.int32, device=DEV)
    slopes = torch.rand(2, 4, device=DEV)
    out = varlen(q, k, v, cu, alibi_slopes=slopes, seqused_k=used if side == "used" else None)
    changed = dict(cu_seqlens=cu, alibi=slopes, used=used)[side]
    changed[1:2] += 1
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.float().sum().backward()


def test_hooks_see_every_saved_tensor():
    q, k, v = (mk(256, 4, 64, seed=i).requires_grad_() for i in range(3))
    cu = torch.tensor([0, 100, 256], dtype=torch.int32, device=DEV)
    slopes = torch.rand(4, device=DEV)
    want = torch.autograd.grad(varlen(q, k, v, cu, alibi_slopes=slopes).float().sum(), (q, k, v))
    seen = []

    def pack(t):
        seen.append(tuple(t.shape))
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.to(DEV)):
        out = varlen(q, k, v, cu, alibi_slopes=slopes)
    assert sorted(seen) == sorted([(256, 4, 64)] * 4 + [(4, 256), (3,), (3,), (2, 4)])      # inputs, output, LSE, lengths, slopes
    for a, b in zip(torch.autograd.grad(out.float().sum(), (q, k, v)), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("call", ["dense", "packed", "varlen", "int8"])
def test_checkpointed_region_that_ends_in_attention(call):
    """projection -> attention -> reshape: the backward of the attention node is what runs the region again."""
    from torch.utils.checkpoint import checkpoint
    torch.manual_seed(0)
    proj = torch.nn.Linear(64, 192, device=DEV, dtype=torch.half)
    x = mk(2, 256, 4, 64).requires_grad_()
    cu = torch.tensor([0, 256, 512], dtype=torch.int32, device=DEV)

    def region(x):
        y = proj(x)
        q, k, v = y.split(64, -1)
        if call == "dense":
            out = fa().flash_attn_func(q, k, v, causal=True)
        elif call == "packed":
            out = fa().flash_attn_qkvpacked_func(y.view(2, 256, 4, 3, 64).transpose(2, 3), causal=True)
        elif call == "varlen":
            out = fa().flash_attn_varlen_func(*(t.reshape(512, 4, 64) for t in (q, k, v)), cu, cu, 256, 256, causal=True)
        else:
            out = fa().attention_int8(*(t.transpose(1, 2).contiguous() for t in (q, k, v)), causal=True)
        return out.reshape(2, -1)

    wrt = (x, proj.weight)
    want = torch.autograd.grad(region(x).float().sum(), wrt)
    got = torch.autograd.grad(checkpoint(region, x, use_reentrant=False).float().sum(), wrt)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("call", ["dense", "packed", "varlen", "int8"])
def test_forward_mode_is_refused(call):
    import torch.autograd.forward_ad as fw
    cu = torch.tensor([0, 256], dtype=torch.int32, device=DEV)
    shape = dict(dense=(1, 256, 4, 64), packed=(1, 256, 3, 4, 64), varlen=(256, 4, 64), int8=(1, 4, 256, 64))[call]
    x = mk(*shape)
    run = dict(dense=lambda t: fa().flash_attn_func(x, t, x), packed=lambda t: fa().flash_attn_qkvpacked_func(t),
               varlen=lambda t: fa().flash_attn_varlen_func(x, x, t, cu, cu, 256, 256),
               int8=lambda t: fa().attention_int8(t, x, x))[call]
    with fw.dual_level():
        run(x)
        with pytest.raises(NotImplementedError):
            run(fw.make_dual(x, torch.ones_like(x)))


def test_output_without_a_gradient_gives_zeros():
    class Dropped(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, grad):
            return None

    q, k, v = (mk(1, 256, 4, 64, seed=i).requires_grad_() for i in range(3))
    w = mk(1, 256, 4, 64, seed=3).requires_grad_()
    (Dropped.apply(fa().flash_attn_func(q, k, v)) * w).sum().backward()
    for t in (q, k, v):
        assert t.grad is not None and not t.grad.any()


def test_backward_of_one_graph_from_several_threads():
    import threading
    q, k, v = (mk(1, 256, 4, 64, seed=i).requires_grad_() for i in range(3))
    out = fa().flash_attn_func(q, k, v, causal=True)
    want = torch.autograd.grad(out.float().sum(), (q, k, v), retain_graph=True)
    got = [None] * 4

    def run(i):
        got[i] = torch.autograd.grad(out.float().sum(), (q, k, v), retain_graph=True)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, want))


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("call", ["dense", "packed", "varlen", "int8"])
def test_traced_calls_are_operations_of_the_trace(call):
    slopes = torch.rand(2, 4, device=DEV)

    def run(x, y, cu):
        if call == "dense":
            return fa().flash_attn_func(x, y, y, causal=True, alibi_slopes=slopes)
        if call == "packed":
            return fa().flash_attn_qkvpacked_func(torch.stack((x, y, y), dim=2), causal=True) + 1
        if call == "varlen":
            flat = [t.reshape(512, 4, 64) for t in (x, y)]
            return fa().flash_attn_varlen_func(flat[0], flat[1], flat[1], cu, cu, 400, 400, causal=True)
        return fa().attention_int8(*(t.transpose(1, 2).contiguous() for t in (x, y, y)), causal=True) + 1

    cu = [torch.tensor([0, n, 512], dtype=torch.int32, device=DEV) for n in (200, 300)]
    args = [(mk(2, 256, 4, 64, seed=i).requires_grad_(), mk(2, 256, 4, 64, seed=9 + i).requires_grad_(), cu[i]) for i in (0, 1)]
    traced = torch.jit.trace(run, args[0], check_trace=False)
    got, want = traced(*args[1]), run(*args[1])
    assert torch.equal(got, want)
    for a, b in zip(torch.autograd.grad(got.float().sum(), args[1][:2]), torch.autograd.grad(want.float().sum(), args[1][:2])):
        assert torch.equal(a, b)
