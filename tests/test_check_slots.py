"""Who has which word of the value checks (csrc/check_slots.h), compiled for the CPU."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attn_triton_b200", "csrc")
SOURCE = """
#include "check_slots.h"
static volatile uint32_t words[8 * 16];
using Slots = fa::CheckSlots<8, 4>;
extern "C" {
void* make() { for (int i = 0; i < 8; ++i) words[i * 16] = 0u; return new Slots(words); }
void drop(void* s) { delete static_cast<Slots*>(s); }
int take_on(void* s, int ticket, int device) { return static_cast<Slots*>(s)->take(ticket != 0, device); }
int take(void* s, int ticket) { return take_on(s, ticket, 0); }
int device_of(void* s, int i) { int d = -1; return static_cast<Slots*>(s)->hand_in(i, &d) ? d : -1; }
int hand_in(void* s, int i) { return device_of(s, i) >= 0; }
void give(void* s, int i, int queued) { static_cast<Slots*>(s)->give(i, queued != 0); }
void answer(int i) { *Slots::word_of(words, i) = 1u; }
int word(int i) { return (int)*Slots::word_of(words, i); }
}
"""
NONE, NEVER = -1, -2


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "slots.cpp").write_text(SOURCE)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + CSRC, str(d / "slots.cpp"), "-o",
                    str(d / "slots.so")], check=True)
    m = C.CDLL(str(d / "slots.so"))
    m.make.restype = C.c_void_p
    for f in (m.drop, m.take, m.hand_in, m.give, m.device_of, m.take_on):
        f.argtypes = [C.c_void_p] + [C.c_int] * {"drop": 0, "take": 1, "hand_in": 1, "give": 2, "device_of": 1, "take_on": 2}[f.__name__]
    return m


@pytest.fixture
def s(lib):
    p = lib.make()
    yield p
    lib.drop(p)


def test_tickets_leave_words_for_calls(lib, s):
    out = [lib.take(s, 1) for _ in range(4)]
    assert len(set(out)) == 4 and min(out) >= 0
    assert lib.take(s, 1) == NONE                        # no more tickets, from any thread
    calls = [lib.take(s, 0) for _ in range(4)]
    assert sorted(out + calls) == list(range(8))
    assert lib.take(s, 0) == NONE                        # until one of the calls is through
    lib.give(s, calls[0], 0)
    assert lib.take(s, 0) == calls[0]
    lib.answer(out[2])
    assert lib.hand_in(s, out[2])
    lib.give(s, out[2], 1)
    assert lib.take(s, 1) == out[2] and lib.word(out[2]) == 0


def test_a_ticket_is_handed_in_once(lib, s):
    i = lib.take(s, 1)
    lib.answer(i)
    assert lib.hand_in(s, i) and not lib.hand_in(s, i)
    lib.give(s, i, 1)
    assert not lib.hand_in(s, i)                         # nor later
    assert not any(lib.hand_in(s, j) for j in (-1, 8, 1 << 20, *range(8)))
    call = lib.take(s, 0)
    assert not lib.hand_in(s, call)                      # the word of a call is no ticket
    lib.give(s, call, 0)
    assert sorted(lib.take(s, 0) for _ in range(8)) == list(range(8))


def test_a_word_without_an_answer_stays_out_of_use(lib, s):
    for _ in range(8):                                   # every owner gave up while its kernel was queued
        lib.give(s, lib.take(s, 0), 1)
    assert lib.take(s, 0) == NEVER                       # a wait for a free word would not end
    lib.answer(5)
    assert lib.take(s, 0) == 5 and lib.word(5) == 0
    lib.give(s, 5, 0)                                    # nothing was launched: free at once
    assert lib.take(s, 0) == 5


def test_no_wait_for_words_that_only_tickets_hold(lib, s):
    for _ in range(4):
        assert lib.take(s, 1) >= 0
    for _ in range(4):
        lib.give(s, lib.take(s, 0), 1)
    assert lib.take(s, 0) == NEVER


def test_a_ticket_knows_its_device(lib, s):
    """The thread that hands it in may have another device current."""
    out = {lib.take_on(s, 1, d): d for d in (3, 0, 7)}
    lib.give(s, lib.take_on(s, 0, 5), 0)
    for i, d in out.items():
        lib.answer(i)
        assert lib.device_of(s, i) == d and lib.device_of(s, i) == -1
        lib.give(s, i, 1)
    assert lib.device_of(s, lib.take_on(s, 1, 2)) == 2
