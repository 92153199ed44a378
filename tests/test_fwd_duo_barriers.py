"""The barriers of the forward with two CTAs per SM (csrc/fwd_duo_sm100.cu), as a model on the CPU: producer, TMA unit, issuer, tensor pipe, softmax
warps, store agent and (INT8) the loader of the scales run in random orders with some of them slow, over items of different lengths and without
tiles; every step checks that what it reads is complete and that what it overwrites has been read."""
import os
import random
import re

import pytest

from test_bwd_barriers import CSRC, Barrier, Fault, need, run

WARPS, SCHED, SCALES = 4, 4, 4


class Cta:
    """own_p: P in columns of its own; split: P V in two key halves; slots of the K/V ring; `broken`: what is left out."""

    def __init__(self, items, own_p, split, slots, int8, rng, broken=None):
        self.items, self.own_p, self.split, self.S, self.int8, self.broken = items + [-1], own_p, split, slots, int8, broken
        one = lambda n: [Barrier(1) for _ in range(n)]
        self.q_full, self.q_empty, self.s_full, self.o_ready, self.stg_taken = one(5)
        self.kv_full, self.kv_empty, self.sched_full, self.sk_full = one(slots), one(slots), one(SCHED), one(SCALES)
        self.s_free, self.p_half, self.p_ready, self.stg_ready = (Barrier(WARPS) for _ in range(4))
        self.sk_empty = [Barrier(WARPS) for _ in range(SCALES)]
        self.sched_empty = [Barrier(WARPS + 2 + int8) for _ in range(SCHED)]
        self.entry, self.slot, self.q, self.scales = [None] * SCHED, [None] * slots, None, [None] * SCALES
        self.loads, self.pipe, self.ends = [], [], 0
        self.S_tile = self.O_tile = -1
        self.first_of = []                               # item of each tile, whether it is the item's first one
        for n, nt in enumerate(items):
            self.first_of += [(n, j == 0) for j in range(nt)]
        self.loaded, self.half, self.stored, self.drained = ([-1] * WARPS for _ in range(4))
        self.staged = [[-1] * WARPS for _ in range(slots)]       # over the item's last V tile
        run([self.producer(), self.tma(), self.issuer(), self.tensor(), self.store_agent()] + ([self.scale_loader()] if int8 else [])
            + [self.softmax(w) for w in range(WARPS)], rng)
        need(self.written == [n for n, nt in enumerate(items) if nt > 0], f"outputs {self.written}")

    written = property(lambda self: self._written)
    _written = None

    def producer(self):
        fidx = pos = qi = nt = i = item = 0
        self._written = []
        while True:
            if i + 1 >= 2 * nt:
                yield lambda: self.sched_empty[fidx % SCHED].done(((fidx // SCHED) & 1) ^ 1)
                self.entry[fidx % SCHED] = fidx
                self.sched_full[fidx % SCHED].arrive()
                fidx += 1
            if i < 2 * nt:
                s = pos % self.S
                yield lambda: self.kv_empty[s].done(((pos // self.S) & 1) ^ 1)
                self.loads.append(("kv", s, (item, "KV"[i & 1], i >> 1)))
                pos += 1
                i += 1
            if i >= 2 * nt:
                item = self.entry[(fidx - 1) % SCHED]
                need(item == fidx - 1, "entry of the ring overwritten")
                nt, i = self.items[item], 0
                if nt < 0:
                    self.ends += 1
                    return
                if nt > 0:
                    yield lambda: self.q_empty.done((qi & 1) ^ 1)
                    self.loads.append(("q", 0, item))
                    qi += 1

    def tma(self):
        while True:
            yield lambda: bool(self.loads) or self.ends > 0
            if not self.loads:
                return
            kind, s, what = self.loads.pop(0)
            if kind == "q":
                need(self.q is None, "Q overwritten")
                self.q = what
                self.q_full.arrive()
            else:
                need(self.slot[s] is None, f"{self.slot[s]} overwritten by {what}")
                self.slot[s] = what
                self.kv_full[s].arrive()

    def entries(self):
        """Items as a consuming warp sees them."""
        for sidx in range(len(self.items)):
            yield sidx, lambda: self.sched_full[sidx % SCHED].done((sidx // SCHED) & 1)

    def get(self, sidx):
        need(self.entry[sidx % SCHED] == sidx, "entry of the ring overwritten")
        return self.items[sidx]

    def issuer(self):
        pos = qi = tc = 0
        for sidx, there in self.entries():
            yield there
            nt = self.get(sidx)
            self.sched_empty[sidx % SCHED].arrive()
            if nt < 0:
                break
            if nt == 0:
                continue
            yield lambda: self.q_full.done(qi & 1)
            qi += 1
            for j in range(nt + 1):
                if self.own_p and j > 0 and self.broken != "s_free":
                    yield lambda: self.s_free.done((tc + j - 1) & 1)
                for what in (("pv", "qk") if not self.own_p else ("qk", "pv")):
                    if what == "qk" and j < nt:
                        ps = pos + 2 * j
                        yield lambda: self.kv_full[ps % self.S].done((ps // self.S) & 1)
                        self.pipe.append(("qk", sidx, j, tc + j, ps % self.S, j + 1 == nt))
                    if what == "pv" and j > 0:
                        ps, t = pos + 2 * j - 1, tc + j - 1
                        yield lambda: self.kv_full[ps % self.S].done((ps // self.S) & 1)
                        if self.split:
                            yield lambda: self.p_half.done(t & 1)
                            self.pipe.append(("half", sidx, j - 1, t, ps % self.S, False))
                        yield lambda: self.p_ready.done(t & 1)
                        self.pipe.append(("pv", sidx, j - 1, t, ps % self.S, j == nt))
            pos += 2 * nt
            tc += nt
        self.ends += 1

    def tensor(self):
        while True:
            yield lambda: bool(self.pipe) or self.ends >= 2
            if not self.pipe:
                return
            op, item, j, t, s, last = self.pipe.pop(0)
            if op == "qk":
                need(self.q == item and self.slot[s] == (item, "K", j), f"Q K({t}) of {self.q}, {self.slot[s]}")
                need(min(self.loaded) >= t - 1, f"Q K({t}) over scores that a warp has not read")
                need(self.own_p or t == 0 or self.O_tile == t - 1, f"Q K({t}) over P({t - 1})")
                self.S_tile = t
                self.s_full.arrive()
                self.slot[s] = None
                self.kv_empty[s].arrive()
                if last:
                    self.q = None
                    self.q_empty.arrive()
                continue
            need(self.slot[s] == (item, "V", j), f"P V({t}) of {self.slot[s]}")
            need(min(self.half if op == "half" else self.stored) >= t, f"P V({t}) without P of every warp")
            n, first = self.first_of[t]
            if first:                                    # overwrites the accumulator
                need(min(self.drained) >= max([m for m in range(n) if self.items[m] > 0], default=-1), f"P V({t}) over a result not read")
            if op == "pv":
                self.O_tile = t
                self.o_ready.arrive()
                if not last:
                    self.slot[s] = None
                    self.kv_empty[s].arrive()

    def store_agent(self):
        pos = wi = 0
        for sidx, there in self.entries():
            yield there
            nt = self.get(sidx)
            self.sched_empty[sidx % SCHED].arrive()
            if nt < 0:
                return
            if nt == 0:
                continue
            pos += 2 * nt
            s = (pos - 1) % self.S
            yield lambda: self.stg_ready.done(wi & 1)
            wi += 1
            need(self.staged[s] == [sidx] * WARPS, f"output of item {sidx}: {self.staged[s]}")
            self.stg_taken.arrive()
            yield None                                   # the unit reads the tile
            need(self.staged[s] == [sidx] * WARPS and self.slot[s] == (sidx, "V", nt - 1), f"output of item {sidx} overwritten")
            self._written.append(sidx)
            self.slot[s] = None
            self.kv_empty[s].arrive()

    def scale_loader(self):
        tc = 0
        for sidx, there in self.entries():
            yield there
            nt = self.get(sidx)
            self.sched_empty[sidx % SCHED].arrive()
            for j in range(nt):
                s = tc % SCALES
                yield lambda: self.sk_empty[s].done(((tc // SCALES) & 1) ^ 1)
                self.scales[s] = tc
                self.sk_full[s].arrive()
                tc += 1

    def softmax(self, w):
        wi = tc = 0
        for sidx, there in self.entries():
            yield there
            nt = self.get(sidx)
            if nt < 0:
                return
            for j in range(nt):
                t = tc + j
                yield lambda: self.s_full.done(t & 1)
                need(self.S_tile == t, f"warp {w} reads scores of tile {self.S_tile} as {t}")
                yield None
                need(self.S_tile == t, f"scores {t} overwritten under warp {w}")
                self.loaded[w] = t
                if self.own_p:
                    self.s_free.arrive()
                if self.int8:
                    s = t % SCALES
                    yield lambda: self.sk_full[s].done((t // SCALES) & 1)
                    need(self.scales[s] == t, f"warp {w} reads scales of tile {self.scales[s]} as {t}")
                    yield None
                    need(self.scales[s] == t, f"scales {t} overwritten under warp {w}")
                    self.sk_empty[s].arrive()
                if j > 0 and (self.own_p or (t + w) % 3 == 0):     # P V before: its P is read; or the accumulator is rescaled
                    yield lambda: self.o_ready.done((t - 1) & 1)
                    need(self.O_tile == t - 1, f"warp {w} rescales the accumulator of tile {self.O_tile} as {t - 1}")
                need(not self.own_p or t == 0 or self.O_tile >= t - 1, f"P({t}) over P({t - 1}) that is being read")
                self.half[w] = t
                if self.split:
                    self.p_half.arrive()
                yield None
                self.stored[w] = t
                self.p_ready.arrive()
            tc += nt
            if nt > 0:
                yield lambda: self.o_ready.done((tc - 1) & 1)
                need(self.O_tile == tc - 1, f"warp {w} reads the accumulator of tile {self.O_tile} as {tc - 1}")
                yield None
                need(self.O_tile == tc - 1, f"accumulator {tc - 1} overwritten under warp {w}")
                self.drained[w] = sidx
                s = (2 * tc - 1) % self.S
                need(self.slot[s] == (sidx, "V", nt - 1), f"output of item {sidx} over {self.slot[s]}")
                self.staged[s][w] = sidx
                if wi > 0 and self.broken != "stg_taken":
                    yield lambda: self.stg_taken.done((wi - 1) & 1)
                self.stg_ready.arrive()
                wi += 1
            need(self.entry[sidx % SCHED] == sidx, f"entry {sidx} overwritten under warp {w}")
            self.sched_empty[sidx % SCHED].arrive()


ITEMS = [[3], [1, 1, 1, 1, 1, 1], [0, 2, 0, 0, 1, 3], [5, 1, 0, 2], [2] * 7, [0] * 9 + [1]]


def source():
    return open(os.path.join(CSRC, "fwd_duo_sm100.cu")).read()


def test_counts_of_the_barriers():
    """What the model takes for granted of the kernel."""
    src = source()
    counts = dict(re.findall(r"mbar_init\(smem_u32\(&sh->(\w+)(?:\[i\])?\), (.*?)\);", src))
    many = {"s_free", "p_half", "p_ready", "stg_ready", "sk_empty"}
    assert {n for n, c in counts.items() if c == "128"} == many
    assert counts.pop("sched_empty") == "kConsumers + (kInt8 ? 1 : 0)" and "kConsumers = 6;" in src
    assert {c for n, c in counts.items() if n not in many} == {"1"} and len(counts) == 14
    assert f"kSched = {SCHED};" in src and f"kSkSlots = {SCALES};" in src and "kStages = (D == 128) ? 2 : 4;" in src


@pytest.mark.parametrize("items", ITEMS, ids=str)
@pytest.mark.parametrize("own_p,split,slots,int8", [(False, True, 2, False), (False, False, 2, False), (False, True, 4, False), (True, True, 4, False),
                                                    (True, False, 4, False), (True, True, 4, True)])
def test_items_one_behind_the_other(items, own_p, split, slots, int8):
    for seed in range(40):
        Cta(items, own_p, split, slots, int8, random.Random(seed))


@pytest.mark.parametrize("broken,own_p", [("s_free", True), ("stg_taken", False)])
def test_the_model_sees_a_wait_left_out(broken, own_p):
    with pytest.raises(Fault):
        for seed in range(400):
            Cta([1, 1, 2, 1, 1, 3], own_p, True, 4, False, random.Random(seed), broken)
