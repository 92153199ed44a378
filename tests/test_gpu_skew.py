"""Backward kernels whose element-wise warps, and forwards with two CTAs per SM whose warps of all roles are made to drift apart (csrc/skew.cuh, a
build of its own): results stay bit for bit those of the shipped build, whichever warps are late."""
import hashlib
import json
import os
import random
import subprocess
import sys

import pytest
import torch

import cases
from util import DEV

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "flash_attn_triton_b200")
LIB = os.path.join(PKG, "libfa_b200_skew.so")

CALLS = {                                        # several items of each kind per CTA
    "causal": dict(B=12, Sq=400, Sk=400, causal=True),
    "odd": dict(B=10, Sq=385, Sk=640),
    "window": dict(B=8, Sq=700, Sk=700, window_size=(100, 30)),
    "dropout": dict(B=12, Sq=512, Sk=512, causal=True, dropout_p=0.2),
    "options": dict(B=12, Sq=384, Sk=384, causal=True, softcap=20.0, alibi=True, window_size=(200, 0)),
    "packed": dict(lens=[1, 300, 128, 513, 64, 257, 400, 129, 700, 31, 256, 512] * 3, causal=True),
}


def gradients():
    """Digests of dQ, dK, dV of every call."""
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    out = {}
    for name, call in CALLS.items():
        for D in (64, 128):
            kw, H = dict(call), 8
            slopes = torch.tensor([0.5 ** (i + 1) for i in range(H)], device=DEV) if kw.pop("alibi", False) else None
            if "lens" in kw:
                lens = kw.pop("lens")
                q, k, v, do, cu, _ = cases.varlen_case(11 + D, lens, lens, H, H, D)
                fn, extra = fa.flash_attn_varlen_func, (cu.to(DEV), cu.to(DEV), max(lens), max(lens))
            else:
                q, k, v, do = cases.dense_case(D, kw.pop("B"), kw.pop("Sq"), kw.pop("Sk"), H, H // 2, D)
                fn, extra = fa.flash_attn_func, ()
            ts = [t.to(DEV).requires_grad_() for t in (q, k, v)]
            random.seed(3)                       # the dropout mask
            grads = torch.autograd.grad(fn(*ts, *extra, alibi_slopes=slopes, **kw), ts, do.to(DEV))
            for g, what in zip(grads, ("dq", "dk", "dv")):
                assert torch.isfinite(g).all(), (name, D, what)
                out[f"{name}-{D}-{what}"] = hashlib.sha256(g.cpu().numpy().tobytes()).hexdigest()
    assert N.lib().fa_device_wait_status(0) == 0
    return out


FORWARDS = {                                     # more than 2.5 tiles per SM, several items for each CTA
    "one tile": dict(B=60, Sq=128, Sk=128),
    "causal": dict(B=14, Sq=400, Sk=400, causal=True),
    "odd": dict(B=14, Sq=385, Sk=640),
    "window": dict(B=10, Sq=700, Sk=700, window_size=(200, 30)),
    "dropout": dict(B=14, Sq=512, Sk=512, causal=True, dropout_p=0.2),
    "options": dict(B=14, Sq=384, Sk=384, causal=True, softcap=20.0, alibi=True),
    "packed": dict(lens=[0, 300, 128, 513, 64, 257, 0, 129, 700, 31, 256, 512] * 4, keys=[128, 0, 300, 128, 513, 64, 257, 0, 129, 700, 31, 256] * 4),
    "int8": dict(B=6, Sq=1088, Sk=1088, causal=True),
}


def forwards():
    """Digests of O of every call."""
    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    out = {}
    for name, call in FORWARDS.items():
        for D in (64, 128):
            kw, H = dict(call), 16
            if kw.pop("alibi", False):
                kw["alibi_slopes"] = torch.tensor([0.5 ** (i + 1) for i in range(H)], device=DEV)
            g = torch.Generator(DEV).manual_seed(D)
            mk = lambda *s: torch.randn(*s, D, device=DEV, dtype=torch.half, generator=g)
            random.seed(3)                       # the dropout mask
            if "lens" in kw:
                lens, keys = kw.pop("lens"), kw.pop("keys")
                cu, ck = (torch.tensor([0] + x, dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32) for x in (lens, keys))
                o = fa.flash_attn_varlen_func(mk(sum(lens), H), mk(sum(keys), 4), mk(sum(keys), 4), cu, ck, max(lens), max(keys), **kw)
            else:
                B, Sq, Sk = kw.pop("B"), kw.pop("Sq"), kw.pop("Sk")
                assert 2 * B * H * -(-Sq // 128) > 5 * torch.cuda.get_device_properties(0).multi_processor_count
                if name == "int8":
                    o = fa.attention_int8(mk(B, H, Sq), mk(B, H, Sk), mk(B, H, Sk), **kw)
                else:
                    o = fa.flash_attn_func(mk(B, Sq, H), mk(B, Sk, H), mk(B, Sk, H), **kw)
            assert torch.isfinite(o).all(), (name, D)
            out[f"{name}-{D}-o"] = hashlib.sha256(o.cpu().numpy().tobytes()).hexdigest()
    assert N.lib().fa_device_wait_status(0) == 0
    return out


def skewed(results):
    from flash_attn_triton_b200 import _native as N
    modes = {}
    for mode in range(5):
        assert N.lib().fa_debug_skew(mode) == 0
        modes[mode] = globals()[results]()
    print("digests " + json.dumps(modes))


def after_a_failed_wait():
    """fa_device_wait_clear() also puts the counters of the work queues back to zero: a launch that gave up leaves them."""
    from flash_attn_triton_b200 import _native as N
    L = N.lib()
    want = gradients()
    assert L.fa_debug_dirty_queues(3) == 0 and L.fa_device_wait_clear(0) == 0
    for _ in range(4):
        got = gradients()
        wrong = [n for n in want if got[n] != want[n]]
        assert not wrong, wrong
    print("queues ok")


def without_queues():
    """Where no pair of counters is left, a CTA per item does the work, with the same results."""
    from flash_attn_triton_b200 import _native as N
    L = N.lib()
    want = gradients()
    assert L.fa_debug_no_queues(1) == 0
    got = gradients()
    wrong = [n for n in want if got[n] != want[n]]
    assert not wrong, wrong
    print("no queues ok")


def captured_pairs():
    """The counters of captured launches come back when their graph is gone, not before."""
    import gc
    import time

    import flash_attn_triton_b200 as fa
    from flash_attn_triton_b200 import _native as N
    L = N.lib()
    q = torch.randn(12, 256, 16, 64, device=DEV, dtype=torch.half)
    want = fa.flash_attn_func(q, q, q, causal=True)
    assert L.fa_debug_captured_queues(0) == 0
    for _ in range(3):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [fa.flash_attn_func(q, q, q, causal=True) for _ in range(3)]
        assert L.fa_debug_captured_queues(0) == 3
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs) and L.fa_debug_captured_queues(0) == 3
        del graph, outs
        gc.collect()
        for _ in range(100):                     # the driver gives them back on a thread of its own
            if L.fa_debug_captured_queues(0) == 0:
                break
            torch.cuda.synchronize()
            time.sleep(0.05)
        assert L.fa_debug_captured_queues(0) == 0
    print("captured ok")


def library():
    """The build with delays, made where it is missing or older than a source."""
    files = [os.path.join(PKG, "csrc", f) for f in os.listdir(os.path.join(PKG, "csrc"))]
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(map(os.path.getmtime, files)):
        env = dict(os.environ, FA_BUILD_TAG="skew", FA_BUILD_DEFS="-DFA_SKEW")
        subprocess.run([sys.executable, "-m", "flash_attn_triton_b200.build"], cwd=ROOT, env=env, check=True, timeout=900)


def child(*what):
    library()
    r = subprocess.run([sys.executable, os.path.abspath(__file__), *what], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, FA_B200_LIB=LIB, PYTHONPATH=os.pathsep.join(sys.path)))
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("results", ["gradients", "forwards"])
def test_late_warps_do_not_change_results(results):
    modes = json.loads(child("skewed", results).split("digests ", 1)[1])
    want = globals()[results]()
    for mode, got in modes.items():
        wrong = [n for n in want if got[n] != want[n]]
        assert not wrong, (mode, wrong)


def test_queues_are_cleared_with_the_wait_status():
    assert "queues ok" in child("after_a_failed_wait")


def test_results_without_a_queue():
    assert "no queues ok" in child("without_queues")


def test_captured_launches_give_their_queues_back():
    assert "captured ok" in child("captured_pairs")


if __name__ == "__main__":
    globals()[sys.argv[1]](*sys.argv[2:])
