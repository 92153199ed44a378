"""Which launch has which counter pair of the work queues (csrc/queue_slots.h), compiled for the CPU."""
import ctypes as C
import os
import subprocess
import threading

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attn_triton_b200", "csrc")
SOURCE = """
#include "queue_slots.h"
using Slots = fa::QueueSlots<8, 5>;
extern "C" {
void* make() { return new Slots(); }
void drop(void* s) { delete static_cast<Slots*>(s); }
int of_stream(void* s, unsigned long long id) { return static_cast<Slots*>(s)->of_stream(id); }
int take(void* s) { return static_cast<Slots*>(s)->take(); }
void give(void* s, int i) { static_cast<Slots*>(s)->give(i); }
int taken(void* s) { return static_cast<Slots*>(s)->taken(); }
}
"""
NONE, STREAMS, CAPTURED = -1, 8, 5


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("queues")
    (d / "queues.cpp").write_text(SOURCE)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + CSRC, str(d / "queues.cpp"), "-o",
                    str(d / "queues.so")], check=True)
    m = C.CDLL(str(d / "queues.so"))
    m.make.restype = C.c_void_p
    for f in (m.drop, m.take, m.taken):
        f.argtypes = [C.c_void_p]
    m.of_stream.argtypes = [C.c_void_p, C.c_ulonglong]
    m.give.argtypes = [C.c_void_p, C.c_int]
    return m


@pytest.fixture
def s(lib):
    p = lib.make()
    yield p
    lib.drop(p)


def test_a_stream_keeps_its_pair(lib, s):
    ids = [0, 1, 2, 1 << 40, (1 << 64) - 1, 77, 1 << 63, 12345]      # ids of any kind
    pairs = [lib.of_stream(s, i) for i in ids]
    assert sorted(pairs) == list(range(STREAMS))
    assert [lib.of_stream(s, i) for i in reversed(ids)] == pairs[::-1]
    assert lib.of_stream(s, 99) == NONE                               # none that it would share with another stream
    assert [lib.of_stream(s, i) for i in ids] == pairs


def test_captured_launches_share_with_nobody_until_their_graph_is_gone(lib, s):
    stream = lib.of_stream(s, 5)
    out = [lib.take(s) for _ in range(CAPTURED)]
    assert len({stream, *out}) == CAPTURED + 1 and all(STREAMS <= i < STREAMS + CAPTURED for i in out)
    assert lib.take(s) == NONE and lib.taken(s) == CAPTURED
    lib.give(s, out[3])
    assert lib.taken(s) == CAPTURED - 1
    assert lib.take(s) == out[3] and lib.take(s) == NONE
    for i in out:
        lib.give(s, i)
    assert lib.taken(s) == 0
    assert sorted(lib.take(s) for _ in range(CAPTURED)) == sorted(out)


def test_threads(lib, s):
    """Each thread has a stream of its own and captures; what one holds no other one gets."""
    held, mu, wrong = set(), threading.Lock(), []

    def work(t):
        mine = lib.of_stream(s, t)
        for _ in range(3000):
            if lib.of_stream(s, t) != mine:
                wrong.append(t)
            i = lib.take(s)
            if i == NONE:
                continue
            with mu:
                if i in held:
                    wrong.append(i)
                held.add(i)
            with mu:
                held.discard(i)
            lib.give(s, i)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(STREAMS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and lib.taken(s) == 0
    assert sorted(lib.of_stream(s, t) for t in range(STREAMS)) == list(range(STREAMS))
