"""The count of bound-and-split's unfinished work (mp_handover.h, compiled for
the host): whatever order relaxed updates of different words arrive in, the
work ends once, after its last unit, with every bundle in a slot of its own.

A thread's steps are partially ordered: updates of one word in program order,
and a step after those whose results it needs.  Every order that this allows
is run.  The same search finds the early end when slot and unit are counted in
two words, so it can see the fault.
"""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "micropolis_gb300", "csrc")
SOURCE = """
#include "mp_handover.h"
using namespace mp;
extern "C" {
unsigned long long start(unsigned long long r) { return handover_start(r); }
unsigned long long give() { return handover_give(); }
unsigned long long slot(unsigned long long b) { return handover_slot(b); }
unsigned long long finish(unsigned u) { return handover_finish(u); }
int ended(unsigned long long b, unsigned u) { return handover_ended(b, u); }
}
"""


@pytest.fixture(scope="module")
def word(tmp_path_factory):
    d = tmp_path_factory.mktemp("handover")
    (d / "w.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "w.so"), str(d / "w.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "w.so"))
    u64 = ctypes.c_uint64
    for name, args in (("start", [u64]), ("give", []), ("slot", [u64]), ("finish", [ctypes.c_uint32])):
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = u64, args
    lib.ended.argtypes = [u64, ctypes.c_uint32]
    return lib


def _orders(steps):
    """Every order of steps (name -> names that come before it)."""
    def rec(done, left):
        if not left:
            yield done
        for s in left:
            if all(b in done for b in steps[s]):
                yield from rec(done + [s], [x for x in left if x != s])
    yield from rec([], list(steps))


# one root's warp gives bundles a and b; a's receiver gives c; each finishes one unit
GIVES = {"a": "root", "b": "root", "c": "a"}


def _steps(two_words):
    steps, last = {}, {}
    for bundle, by in GIVES.items():
        before = [last[by]] if by in last else []                    # same word, program order
        needs = ["read " + by] if by != "root" else []
        steps["give " + bundle] = before + needs
        last[by] = "give " + bundle
        if two_words:   # the unit, on another word: after nothing but its own word's updates
            steps["unit " + bundle] = needs + (["unit " + p for p, q in GIVES.items() if q == by and p < bundle])
        steps["read " + bundle] = ["give " + bundle]                 # written to the slot, found there
    for who in ["root", *GIVES]:
        own = [g for g, by in GIVES.items() if by == who]
        steps["end " + who] = (["read " + who] if who != "root" else []) + \
            (["unit " + g for g in own] if two_words else ["give " + g for g in own])
    return steps


def _run(word, order, capacity, two_words):
    """Ends seen, each as the number of units not yet finished; the slots; what is left."""
    m = 2 ** 64
    count, tail, slots, ends, open_units = word.start(1), 0, [], [], 1
    for s in order:
        what, who = s.split()
        if what == "give":
            if two_words:
                slot, tail = tail, tail + 1
            else:
                slot, count = word.slot(count), (count + word.give()) % m
                if slot >= capacity:
                    count = (count + word.finish(1)) % m
            slots.append(slot)
            open_units += 1
        elif what == "unit":
            count = (count + 1) % m
        elif what == "end":
            ended, count = word.ended(count, 1), (count + word.finish(1)) % m
            open_units -= 1
            if ended:
                ends.append(open_units)
    return ends, slots, count % 2 ** 32


def test_ends_once_after_the_last_unit(word):
    n = 0
    for order in _orders(_steps(False)):
        ends, slots, left = _run(word, order, 8, False)
        assert ends == [0] and left == 0 and sorted(slots) == [0, 1, 2], order
        n += 1
    assert n > 100


def test_two_words_end_early(word):
    assert any(_run(word, order, 8, True)[0] != [0] for order in _orders(_steps(True)))


def test_no_slot_keeps_the_unit_with_its_giver(word):
    count = word.start(2)
    before = count
    count += word.give()
    assert word.slot(before) == 0 and word.slot(count) == 1
    count = (count + word.finish(1)) % 2 ** 64     # capacity 0: taken back
    assert not word.ended(count, 1) and word.ended(count, 2)
    assert word.slot((count + word.finish(2)) % 2 ** 64) == 1     # no borrow from the slots


def test_root_batches_in_one_update(word):
    big = 2 ** 31 - 1
    count = word.start(big)
    assert not word.ended(count, big - 1) and word.ended(count, big)
