"""Items of the kernel that takes them by number (csrc/items.cuh, csrc/queue.cuh and the draw in csrc/fwd_duo_sm100.cu), compiled for the CPU with the
lanes of a warp in turn: every tile of rows is worked on once, whatever the lengths, the order and the way in which the CTAs get their candidates."""
import ctypes as C
import os
import random
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "flash_attn_triton_b200", "csrc")
SOURCE = r"""
#include <ucontext.h>
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include "fa_b200.h"
#define __device__
#define __forceinline__ inline

struct dim3 { unsigned x, y, z; dim3(unsigned x, unsigned y = 1, unsigned z = 1) : x(x), y(y), z(z) {} };
static dim3 gridDim(1), blockIdx(0);
using std::max;
using std::min;

// Lanes of a warp: each runs until it votes; the votes are counted when all have, and every lane goes on.
static ucontext_t lanes[32], scheduler;
static char stacks[32][65536];
static int current, done;
static unsigned votes[32], ballot, value0;
static int largest;
static void vote(unsigned v) { votes[current] = v; swapcontext(&lanes[current], &scheduler); }
static unsigned __ballot_sync(unsigned, bool p) { vote(p); return ballot; }
static int __reduce_max_sync(unsigned, int v) { vote((unsigned)v); return largest; }
static unsigned __shfl_sync(unsigned, unsigned v, int) { vote(v); return value0; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static unsigned atomicAdd(unsigned* p, unsigned n) { unsigned v = *p; *p += n; return v; }
static void __threadfence() {}

namespace fa {
struct ScoreCfg { int causal, wl, wr, unit_group; bool packed_list; };
static int sm_count(int) { return 148; }
}
#include "items.cuh"
#include "queue.cuh"

using namespace fa;
static const fa_attn_args* g_a;
static ScoreCfg g_cfg;
static int g_by_weight, g_ncand, g_h[32], g_b[32], g_mt[32];
static unsigned* g_counter;
static int g_last[32];
static bool g_found[32];
static int g_fidx;
struct Item { int nt; };
static void lane_main() {
  const int lane = current, fidx = g_fidx, ncand = g_ncand, by_weight = g_by_weight;
  unsigned* const queue = g_counter;
  const fa_attn_args& p = *g_a;
  const ScoreCfg& cfg = g_cfg;
  auto item_of = [](const fa_attn_args& p, const ScoreCfg& cfg, int by_weight, int c, int lane, Item& w) {
    SeqInfo si;
    w.nt = 1;
    return item_tile<128>(p, cfg, by_weight, c, lane, g_h[lane], g_b[lane], si, g_mt[lane]);
  };
  int c = g_last[lane];
  Item w;
  // from fwd_duo_sm100.cu
  DRAW
  g_last[lane] = c;
  g_found[lane] = w.nt >= 0;
  ++done;
}
static void run_warp() {
  done = 0;
  for (int i = 0; i < 32; ++i) {
    getcontext(&lanes[i]);
    lanes[i].uc_stack.ss_sp = stacks[i];
    lanes[i].uc_stack.ss_size = sizeof(stacks[i]);
    lanes[i].uc_link = &scheduler;
    makecontext(&lanes[i], lane_main, 0);
  }
  while (done == 0) {
    for (current = 0; current < 32; ++current) swapcontext(&scheduler, &lanes[current]);
    if (done != 0 && done != 32) abort();          // lanes that do not vote together
    ballot = 0;
    largest = (int)votes[0];
    value0 = votes[0];
    for (int i = 0; i < 32; ++i) {
      ballot |= (votes[i] != 0u ? 1u : 0u) << i;
      largest = max(largest, (int)votes[i]);
    }
  }
}
extern "C" {
int candidates(const fa_attn_args* a, int causal, int wl, int wr) {
  g_a = a;
  g_cfg = {causal, wl, wr, 1, false};
  g_ncand = (int)item_candidates<128>(*a, g_cfg, g_by_weight);
  return g_ncand;
}
// The next item of CTA `cta` of `grid`, whose last candidate was *last (-1: none yet): 0 behind the last one.  counter: null without a queue.
int next_item(int grid, int cta, unsigned* counter, int* last, int* h, int* b, int* mt) {
  gridDim.x = grid;
  blockIdx.x = cta;
  g_counter = counter;
  g_fidx = *last < 0 ? 0 : 1;
  for (int i = 0; i < 32; ++i) g_last[i] = g_fidx == 0 ? cta : *last;
  run_warp();
  for (int i = 1; i < 32; ++i)
    if (g_found[i] != g_found[0] || g_last[i] != g_last[0] || (g_found[0] && (g_h[i] != g_h[0] || g_b[i] != g_b[0] || g_mt[i] != g_mt[0]))) abort();
  *last = g_last[0];
  *h = g_h[0]; *b = g_b[0]; *mt = g_mt[0];
  return g_found[0];
}
void finish(int grid, int cta, unsigned* counter) { gridDim.x = grid; blockIdx.x = cta; queue_finish(counter, g_ncand); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    kernel = open(os.path.join(CSRC, "fwd_duo_sm100.cu")).read()
    draw = re.search(r"int c = blockIdx.x;.*?Item w;\n(.*?)\n        if \(fidx == 0\)", kernel, re.S).group(1)
    (d / "items.cpp").write_text(SOURCE.replace("DRAW", draw))
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    str(d / "items.cpp"), "-o", str(d / "items.so")], check=True)
    return C.CDLL(str(d / "items.so"))


def tiles_worked_on(lib, args, mask, grid_of, use_queue, rng):
    """(h, b, mt) of every item of a launch whose CTAs go at random paces."""
    ncand = lib.candidates(C.byref(args), *mask)
    grid = grid_of(ncand)
    counter = (C.c_uint * 2)(0, 0)
    last = [C.c_int(-1) for _ in range(grid)]
    h, b, mt = C.c_int(), C.c_int(), C.c_int()
    got, running = [], list(range(grid))
    while running:
        i = rng.randrange(len(running))
        cta = running[i]
        if lib.next_item(grid, cta, counter if use_queue else None, C.byref(last[cta]), C.byref(h), C.byref(b), C.byref(mt)):
            got.append((h.value, b.value, mt.value))
        else:
            running[i] = running[-1]
            running.pop()
            if use_queue:
                lib.finish(grid, cta, counter)
    assert list(counter) == [0, 0]                   # as the next launch has to find them
    return got


def call(q_lens, heads, heads_kv, packed, max_q=None, used=None, first=0):
    from flash_attn_triton_b200 import _native as N
    a = N.AttnArgs()
    a.batch, a.heads_q, a.heads_kv, a.head_dim = len(q_lens), heads, heads_kv, 128
    a.seqlen_q = a.seqlen_k = max(q_lens) if max_q is None else max_q
    keep = []
    if packed:
        cu = np.concatenate([[first], first + np.cumsum(q_lens)]).astype(np.int32)
        a.total_q = a.total_k = int(cu[-1])
        a.cu_seqlens_q = a.cu_seqlens_k = cu.ctypes.data
        keep.append(cu)
    if used is not None:
        u = np.array(used, dtype=np.int32)
        a.seqused_q = u.ctypes.data
        keep.append(u)
    return a, keep


MASKS = {"none": (0, -1, -1), "causal": (1, -1, -1), "narrow": (0, 100, 60), "left": (0, 200, -1), "right": (0, -1, 60)}


def check(lib, q_lens, heads, heads_kv, packed, mask, grid_of, use_queue, rng, max_q=None, used=None, first=0):
    a, keep = call(q_lens, heads, heads_kv, packed, max_q, used, first)
    got = tiles_worked_on(lib, a, MASKS[mask], grid_of, use_queue, rng)
    rows = [min(n, a.seqlen_q) for n in q_lens] if used is None else [min(n, u, a.seqlen_q) for n, u in zip(q_lens, used)]
    want = sorted((h, b, t) for b, n in enumerate(rows) for t in range(-(-n // 128)) for h in range(heads))
    assert sorted(got) == want, (q_lens, heads, mask, use_queue)


HALF = lambda n: max(1, (n + 1) // 2)                # two items for each CTA
FEW = lambda n: min(n, 7)
LENGTHS = {"list": [256, 512, 384, 640, 128, 768, 256, 512], "grid": [128] * 12 + [256] * 6, "short first": [30] + [252] * 5,
           "empty first": [0] + [256] * 12, "empty last": [256] * 6 + [0, 0], "in between": [300, 0, 1, 640, 0, 0, 129]}


@pytest.mark.parametrize("use_queue", [False, True])
@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("lens", LENGTHS)
def test_every_tile_once(lib, lens, mask, use_queue):
    rng = random.Random(7)
    for grid_of in (HALF, FEW, lambda n: n):
        check(lib, LENGTHS[lens], 4, 2, True, mask, grid_of, use_queue, rng)


@pytest.mark.parametrize("use_queue", [False, True])
@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("first", [1, 127, 128, 300, 6000])
def test_rows_before_the_first_sequence(lib, first, mask, use_queue):
    """A first sequence that does not start at row 0 (refused by the value checks, which a caller may have switched off)."""
    rng = random.Random(first)
    for lens in ([300, 0, 129, 64], [200] * 40):
        check(lib, lens, 4, 2, True, mask, HALF, use_queue, rng, first=first)


@pytest.mark.parametrize("seed", range(12))
def test_random_calls(lib, seed):
    rng = random.Random(seed)
    for _ in range(6):
        n = rng.choice((1, 3, 9, 31, 33, 40))
        lens = [rng.choice((0, 1, rng.randint(1, 128), rng.randint(1, 1100))) for _ in range(n)]
        lens[rng.randrange(n)] += 1
        max_q = max(lens) + rng.choice((0, 0, 200)) - (rng.choice((0, 100)) if max(lens) > 200 else 0)
        used = None if rng.random() < .7 else [rng.randint(0, m) for m in lens]
        check(lib, lens, 4, rng.choice((1, 4)), True, rng.choice(list(MASKS)), rng.choice((HALF, FEW)), rng.random() < .5, rng, max_q, used)
        B, S = rng.randint(1, 6), rng.randint(1, 700)
        used = None if rng.random() < .5 else [rng.randint(0, S) for _ in range(B)]
        check(lib, [S] * B, rng.choice((1, 3, 8)), 1, False, rng.choice(list(MASKS)), rng.choice((HALF, FEW)), rng.random() < .5, rng, S, used)


def test_two_launches_with_one_pair_lose_tiles(lib):
    """Why launches that run at the same time need counters of their own: the CTAs of two calls in turn, on one pair and on two."""
    rng = random.Random(1)
    a, keep = call([700] * 3, 4, 2, True)
    h, b, mt = C.c_int(), C.c_int(), C.c_int()
    ncand = lib.candidates(C.byref(a), *MASKS["causal"])
    lost = {}
    for pairs in (1, 2):
        counters = [(C.c_uint * 2)(0, 0) for _ in range(pairs)]
        last = {(n, cta): C.c_int(-1) for n in range(2) for cta in range(5)}
        got, running = {0: set(), 1: set()}, list(last)
        while running:
            n, cta = rng.choice(running)
            if lib.next_item(5, cta, counters[n % pairs], C.byref(last[n, cta]), C.byref(h), C.byref(b), C.byref(mt)):
                got[n].add((h.value, b.value, mt.value))
            else:
                running.remove((n, cta))
                lib.finish(5, cta, counters[n % pairs])
        lost[pairs] = 2 * 3 * 6 * 4 - len(got[0]) - len(got[1])
    assert ncand > 5 and lost[1] > 0 and lost[2] == 0
