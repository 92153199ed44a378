"""Value checks of cache calls: who owns the result that the attention kernels read."""
import ctypes as C

import pytest
import torch

from util import DEV

pytestmark = pytest.mark.gpu


def problem(tokens, page, lens, seed=0):
    """(arguments of flash_attn_with_kvcache, with every page of the pool in the table once)"""
    g = torch.Generator(DEV).manual_seed(seed)
    mk = lambda *s: torch.randn(*s, device=DEV, dtype=torch.half, generator=g)
    B, H, Hkv, D = len(lens), 16, 4, 128
    n = -(-(max(lens) + tokens) // page)
    return dict(q=mk(B, tokens, H, D), k_cache=mk(B * n, page, Hkv, D), v_cache=mk(B * n, page, Hkv, D), k=mk(B, tokens, Hkv, D),
                v=mk(B, tokens, Hkv, D), cache_seqlens=torch.tensor(lens, dtype=torch.int32, device=DEV),
                block_table=torch.randperm(B * n, device=DEV, generator=g).to(torch.int32).view(B, n), causal=True)


# a chunk (checks inside its first kernel), a chunk and a decode step with more table entries than are checked there
KINDS = [(512, 64, [4000] * 8), (64, 16, [3000] * 8), (1, 16, [20000] * 16)]


@pytest.mark.parametrize("tokens,page,lens", KINDS)
@pytest.mark.parametrize("first_bad", [False, True])
def test_result_of_a_call_is_not_that_of_another_stream(tokens, page, lens, first_bad):
    import flash_attn_triton_b200 as fa
    good = problem(tokens, page, lens)
    bad = problem(tokens, page, lens, seed=1)
    bad["block_table"][-1, -1] = 1 << 20
    want = fa.flash_attn_with_kvcache(**good)
    kept = bad["k_cache"].clone()
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        for stream, call in zip(streams, (bad, good) if first_bad else (good, bad)):
            with torch.cuda.stream(stream):
                if call is bad:
                    with pytest.raises(ValueError, match="invalid physical page"):
                        fa.flash_attn_with_kvcache(**bad)
                else:
                    got = fa.flash_attn_with_kvcache(**good)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        assert torch.equal(bad["k_cache"], kept)


@pytest.mark.parametrize("tokens,page,lens", KINDS)
def test_without_room_for_the_result(tokens, page, lens):
    """A workspace of fa_decode_workspace_bytes: the call waits for its checks before it launches the attention."""
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    p = problem(tokens, page, lens)
    want = fa.flash_attn_with_kvcache(**p)
    q, kc, vc, out = p["q"], p["k_cache"], p["v_cache"], torch.zeros_like(p["q"])
    bshd = (0, 1, 2)
    a = N.DecodeArgs()
    a.dtype, a.device = N.dtype_code(q.dtype), 0
    a.batch, a.seqlen_q, a.heads_q, a.head_dim = q.shape
    a.heads_kv, a.page_size, a.num_pages = kc.shape[2], kc.shape[1], kc.shape[0]
    a.q, a.o, a.k_cache, a.v_cache, a.k_new, a.v_new = (t.data_ptr() for t in (q, out, kc, vc, p["k"], p["v"]))
    a.q_stride, a.o_stride, a.kc_stride, a.vc_stride, a.kn_stride, a.vn_stride = (
        N.strides3(t, bshd) for t in (q, out, kc, vc, p["k"], p["v"]))
    a.seqlen_new = tokens
    a.cache_seqlens, a.block_table, a.block_table_stride = (
        p["cache_seqlens"].data_ptr(), p["block_table"].data_ptr(), p["block_table"].shape[1])
    a.softmax_scale, a.causal, a.window_left, a.window_right = q.shape[-1] ** -0.5, 1, -1, -1
    need = N.lib().fa_decode_workspace_bytes(C.byref(a))
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = (ws.data_ptr() if need else None), need
    failed = C.c_uint32(99)
    call = lambda: N.check(N.lib().fa_decode_paged_checked(C.byref(a), C.byref(failed), N.stream_ptr(q.device)), "checked")
    call()
    assert failed.value == 0
    assert torch.equal(out, want)
    p["block_table"][0, 0] = -1
    out.zero_()
    call()
    assert failed.value == 1                    # FA_CHECK_PAGES
    torch.cuda.synchronize()
    assert not out.any()


def decode_call(stream_no, tokens=1):
    """A call whose sequences are cut into pieces (the merge counters are per stream), and what it gives alone."""
    import flash_attn_triton_b200 as fa
    p = problem(tokens, 64, [3000, 700, 4100], seed=stream_no)
    return p, fa.flash_attn_with_kvcache(**p)


def test_more_streams_than_counter_buffers():
    """Every stream has merge counters of its own; the 33rd takes the place of the first."""
    import flash_attn_triton_b200 as fa
    calls = [decode_call(i) for i in range(3)]
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(32)]      # 32 streams of each priority exist
    got = []
    torch.cuda.synchronize()
    for again in range(2):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got.append((i % 3, fa.flash_attn_with_kvcache(**calls[i % 3][0])))
    torch.cuda.synchronize()
    for i, out in got:
        assert torch.equal(out, calls[i][1])


@pytest.mark.parametrize("tokens", [1, 40])
def test_threads_with_a_stream_each(tokens):
    import threading

    import flash_attn_triton_b200 as fa
    calls = [decode_call(i, tokens) for i in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                if not torch.equal(fa.flash_attn_with_kvcache(**calls[i][0]), calls[i][1]):
                    wrong.append(i)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("tokens", [1, 40])
def test_captured_call_replays(tokens):
    """Value checks off: the call goes into a CUDA graph, with merge counters of its own that the graph sets to zero."""
    import flash_attn_triton_b200 as fa
    (p, want), (other, want_other) = decode_call(0, tokens), decode_call(1, tokens)
    fa.set_validation(False)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = fa.flash_attn_with_kvcache(**p)
        for _ in range(3):
            out.zero_()
            graph.replay()
            assert torch.equal(out, want)
        for name in ("q", "k", "v", "k_cache", "v_cache", "cache_seqlens", "block_table"):
            p[name].copy_(other[name])
        graph.replay()
        assert torch.equal(out, want_other)
    finally:
        fa.set_validation(True)


def test_checked_call_under_capture_is_refused():
    import flash_attn_triton_b200 as fa
    p, want = decode_call(0)
    with pytest.raises(RuntimeError, match="captured"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            fa.flash_attn_with_kvcache(**p)
    torch.cuda.synchronize()
    assert torch.equal(fa.flash_attn_with_kvcache(**p), want)
