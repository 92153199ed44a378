"""Launches that run at the same time and take their work from queues: many of them on two streams, and replayed graphs beside other
calls, give bit for bit what they give one behind the other."""
import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu

# each with more items than CTAs: two CTAs per SM; one persistent CTA per SM; INT8
CALLS = {"two CTAs": dict(B=12, S=256, H=16, D=64), "persistent": dict(B=1, S=4224, H=16, D=128, causal=False), "int8": dict(B=3, S=1024, H=16, D=64)}


def problem(name, seed):
    import flash_attn_triton_b200 as fa
    c = dict(CALLS[name])
    causal = c.pop("causal", True)
    g = torch.Generator(DEV).manual_seed(seed)
    if name == "int8":
        q, k, v = (torch.randn(c["B"], c["H"], c["S"], c["D"], device=DEV, dtype=torch.half, generator=g) for _ in range(3))
        return lambda: fa.attention_int8(q, k, v, causal=causal)
    q, k, v = (torch.randn(c["B"], c["S"], c["H"], c["D"], device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    return lambda: fa.flash_attn_func(q, k, v, causal=causal)


def training_step(seed):
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(seed)
    q, k, v, do = (torch.randn(6, 512, 16, 64, device=DEV, dtype=torch.half, generator=g) for _ in range(4))
    ts = [t.requires_grad_() for t in (q, k, v)]
    return lambda: torch.cat(torch.autograd.grad(fa.flash_attn_func(*ts, causal=True), ts, do))


def busy(streams):
    """Work in front of each stream, so that what is launched next is all under way together."""
    for s in streams:
        with torch.cuda.stream(s):
            torch.cuda._sleep(40_000_000)


@pytest.mark.parametrize("a,b", [("two CTAs", "two CTAs"), ("two CTAs", "persistent"), ("int8", "two CTAs"), ("train", "two CTAs"), ("train", "train")])
def test_many_launches_on_two_streams(a, b):
    from flash_attn_triton_b200 import _native as N
    calls = [training_step(n) if name == "train" else problem(name, n) for n, name in enumerate((a, b))]
    want = [c() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    busy(streams)
    got = ([], [])
    for i in range(90):                              # more than 64 on each
        for n, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[n].append(calls[n]())
    torch.cuda.synchronize()
    assert N.lib().fa_device_wait_status(0) == 0
    for n in range(2):
        for i, o in enumerate(got[n]):
            assert torch.equal(o, want[n]), (n, i)


@pytest.mark.parametrize("name", list(CALLS))
def test_a_replayed_graph_beside_other_calls(name):
    """A captured launch has its counters for good: neither eager calls, any number of them, nor another graph get them."""
    from flash_attn_triton_b200 import _native as N
    calls = [problem(name, n) for n in range(3)]
    want = [c() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    graphs, outs = [], []
    for c, s in zip(calls[:2], streams):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            outs.append(c())
        graphs.append(graph)
    torch.cuda.synchronize()
    busy(streams)
    eager, replayed = [], ([], [])
    for i in range(90):
        for n, (graph, s) in enumerate(zip(graphs, streams)):
            with torch.cuda.stream(s):
                graph.replay()
                if i % 9 == 0:
                    replayed[n].append(outs[n].clone())
                outs[n].fill_(float("nan"))
        with torch.cuda.stream(streams[2]):
            eager.append(calls[2]())
    torch.cuda.synchronize()
    assert N.lib().fa_device_wait_status(0) == 0
    for n in range(2):
        assert all(torch.equal(o, want[n]) for o in replayed[n])
    assert all(torch.equal(o, want[2]) for o in eager)


def test_branches_of_one_graph():
    """Launches of one graph that do not depend on one another may run together."""
    calls = [problem("two CTAs", n) for n in range(4)]
    want = [c() for c in calls]
    side = [torch.cuda.Stream() for _ in calls]
    graph, outs = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        for c, s in zip(calls, side):
            s.wait_stream(main)
            with torch.cuda.stream(s):
                outs.append(c())
        for s in side:
            main.wait_stream(s)
    for _ in range(5):
        for o in outs:
            o.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(outs, want))
