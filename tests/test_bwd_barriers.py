"""The barriers between the issuer and the element-wise warps of the backward kernels (8, with score options 16), as a model on the CPU: warps, issuer
and tensor pipe run in random orders with some of them slow, and every step checks that what it reads is complete and that
what it overwrites has been read."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attn_triton_b200", "csrc")
WARPS = (8, 16)


class Fault(AssertionError):
    pass


def need(ok, what):
    if not ok:
        raise Fault(what)


class Barrier:
    def __init__(self, count):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def done(self, parity):                     # mbarrier.try_wait.parity
        return (self.phase & 1) != parity


def run(agents, rng):
    """Each agent is a generator that yields the condition it waits for (None: just a step)."""
    waits = {a: None for a in agents}
    pace = {a: rng.choice([0.02, 0.3, 1.0]) for a in agents}
    idle = 0
    while waits:
        a = rng.choice(list(waits))
        if rng.random() > pace[a]:
            continue
        if waits[a] is not None and not waits[a]():
            idle += 1
            need(idle < 20000, "deadlock")
            continue
        idle = 0
        try:
            waits[a] = next(a)
        except StopIteration:
            del waits[a]


def dkdv(items, buffers, p_barriers, rng, warps=8):
    """Tiles of dK/dV: `items` are numbers of query tiles, `buffers` score buffers, `p_barriers` barriers for "P stored"."""
    s_full, dp_full = [Barrier(1) for _ in range(buffers)], Barrier(1)
    p_ready, ds_ready = [Barrier(warps) for _ in range(p_barriers)], Barrier(warps)
    pipe, closed = [], []
    s_done, dp_done = {}, -1                     # buffer -> tile computed in it
    loaded_s, stored_p, loaded_dp, stored_ds = ([-1] * warps for _ in range(4))
    total = sum(items)

    def tensor_pipe():
        nonlocal dp_done
        while True:
            yield lambda: bool(pipe) or bool(closed)
            if not pipe:
                return
            op, i = pipe.pop(0)
            if op == "S":
                need(min(loaded_s) >= i - buffers, f"S({i}) over scores that a warp has not read")
                s_done[i % buffers] = i
                s_full[i % buffers].arrive()
            elif op == "dP":
                need(min(loaded_dp) >= i - 1, f"dP({i}) over dP that a warp has not read")
                dp_done = i
                dp_full.arrive()
            elif op == "dV":
                need(min(stored_p) >= i and s_done[i % buffers] == i, f"dV({i}) without P of every warp")
            else:
                need(min(stored_ds) >= i and dp_done == i, f"dK({i}) without dS of every warp")

    def issuer():
        pos = 0
        for n in items:
            issue = lambda op, i: pipe.append((op, pos + i)) if i < n else None
            issue("S", 0)
            issue("dP", 0)
            if buffers == 2:
                issue("S", 1)
            for i in range(n):
                ps = pos + i
                yield lambda: p_ready[ps % p_barriers].done((ps // p_barriers) & 1)
                issue("dV", i)
                issue("S", i + buffers)
                yield lambda: ds_ready.done(ps & 1)
                issue("dK", i)
                issue("dP", i + 1)
            pos += n
        closed.append(1)

    def warp(w):
        for i in range(total):
            yield lambda: s_full[i % buffers].done((i // buffers) & 1)
            need(s_done[i % buffers] == i, f"warp {w} reads scores of another tile than {i}")
            loaded_s[w] = i
            yield None
            stored_p[w] = i
            p_ready[i % p_barriers].arrive()
            yield lambda: dp_full.done(i & 1)
            need(dp_done == i, f"warp {w} reads dP of another tile than {i}")
            loaded_dp[w] = i
            yield None
            stored_ds[w] = i
            ds_ready.arrive()

    run([tensor_pipe(), issuer()] + [warp(w) for w in range(warps)], rng)


def dq_results(items, last_waits, rng, warps=8):
    """Result tiles of the dQ kernel on their way to the store lane; `last_waits`: the warps wait for one another
    before the message that ends it."""
    ready, taken, products, last = Barrier(warps), Barrier(1), Barrier(warps), Barrier(warps)
    staged, message = [-1] * warps, None

    def store_lane():
        for n in range(items + 1):
            yield lambda: ready.done(n & 1)
            need(message == n, f"message {message} instead of {n}")
            need(n == items or min(staged) >= n, f"tile {n} stored before every warp has staged it")
            taken.arrive()

    def warp(w):
        nonlocal message
        for n in range(items + 1):
            if n < items:
                products.arrive()                # the item's products need dS of every warp
                yield lambda: products.done(n & 1)
                yield None
            elif last_waits:
                last.arrive()
                yield lambda: last.done(0)
            if w == 0:
                if n > 0:
                    yield lambda: taken.done((n - 1) & 1)
                message = n
            if n < items:
                staged[w] = n
            ready.arrive()

    run([store_lane()] + [warp(w) for w in range(warps)], rng)


ITEMS = [[5], [1, 1, 1, 1], [3, 2, 1], [2, 7]]


def kernel_source():
    return open(os.path.join(CSRC, "bwd_sm100.cu")).read()


def test_barriers_count_every_element_wise_thread():
    """Both numbers of groups: what the model takes for granted."""
    src = kernel_source()
    counts = re.findall(r"mbar_init\(smem_u32\(&sh->(?:p_ready|ds_ready|stg_ready)(?:\[\d\])?\), (.*?)\);", src)
    assert len(counts) == 7 and set(counts) == {"R::kEwThreads"}
    assert "kEwThreads = 128 * G, kEwWarps = 4 * G;" in src and "return f == Feat::kNone ? 2 : 4;" in src


@pytest.mark.parametrize("warps", WARPS)
@pytest.mark.parametrize("items", ITEMS, ids=str)
@pytest.mark.parametrize("head_dim", [64, 128])
def test_dkdv_tiles(items, head_dim, warps):
    src = kernel_source()
    buffers = int(re.search(r"kSBuf = D == 64 \? (\d) : (\d);", src).group(1 if head_dim == 64 else 2))
    declared = re.search(r"uint64_t p_ready(?:\[(\d)\])?;", src).group(1)
    per_buffer = "p_ready[sbuf(pos)]" in src and "p_ready[sbuf(ps)], sphase(ps)" in src
    assert not per_buffer or int(declared) >= buffers
    for seed in range(60):
        dkdv(items, buffers, buffers if per_buffer else 1, random.Random(seed), warps)


def test_the_model_sees_an_early_phase():
    """One barrier for two score buffers: a warp that is a tile ahead completes the phase for one that is late."""
    with pytest.raises(Fault):
        for seed in range(400):
            dkdv([7], 2, 1, random.Random(seed))


@pytest.mark.parametrize("warps", WARPS)
@pytest.mark.parametrize("items", [0, 1, 2, 5])
def test_dq_results(items, warps):
    end = kernel_source().split("No more items: the store lane may leave")[-1]
    last_waits = re.search(r'"bar\.sync 1, %0;\\n" ::"n"\(R::kEwThreads\)', end.split("post_store(sh, 0, wi, -1")[0]) is not None
    for seed in range(100):
        dq_results(items, last_waits, random.Random(seed), warps)


def test_the_model_sees_a_tile_stored_early():
    with pytest.raises(Fault):
        for seed in range(400):
            dq_results(1, False, random.Random(seed))
