"""The words that the CTAs of the device seed loop exchange
(psod_b200/csrc/psod_loop.cuh), compiled for the host and walked through every
interleaving of small cases."""

import ctypes as C
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "psod_b200", "csrc")

SHIM = r"""
#include "psod_loop.cuh"
typedef void (*hook_fn)();
struct HookMem {  // what other CTAs do between two accesses
  hook_fn hook;
  void between() { if (hook) { hook_fn h = hook; hook = nullptr; h(); } }
  unsigned load(const unsigned *p) { const unsigned v = *p; between(); return v; }
  unsigned exchange(unsigned *p, unsigned v) { const unsigned old = *p; *p = v; return old; }
  unsigned cas(unsigned *p, unsigned was, unsigned v) { const unsigned old = *p; if (old == was) *p = v; return old; }
};
extern "C" {
int ring_take(unsigned *place, unsigned *block, hook_fn hook) { HookMem m{hook}; return psod::ring_take(m, place, *block); }
int ring_put(unsigned *place, unsigned block) { HookMem m{nullptr}; return psod::ring_put(m, place, block); }
unsigned long long open_word(unsigned n) { return psod::refine_open(n); }
long wrong_splits(int sx, int sy, int sz) {
  long bad = 0;
  const int total = sx * sy * sz;
  for (int z = 0, e = 0; z < sz; z++)
    for (int y = 0; y < sy; y++)
      for (int x = 0; x < sx; x++, e++) {
        int a, b, c;
        psod::box_split(e, sx, sy, total, a, b, c);
        bad += a != x || b != y || c != z;
      }
  return bad;
}
int take(unsigned long long drawn, unsigned *item) { return psod::refine_take(drawn, *item); }
}
"""


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    d = tmp_path_factory.mktemp("loop")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.open_word.restype = C.c_ulonglong
    lib.take.argtypes = [C.c_ulonglong, C.POINTER(C.c_uint)]
    return lib


def refine_runs(open_word, take, two_step, items=(1, 2), helpers=2, draws=3):
    """Every interleaving of an owner that publishes seeds of `items` items in
    one slot (publish, take items itself, wait for all, close) with helper warps
    of `draws` draws each.  A step is one access to shared memory.  Yields the
    multiset of (seed whose data were read, item) of each complete run, or None
    for one in which the owner went on with items unfinished."""
    # shared: word, count (read apart in the two-step form), done, seed published
    # owner: (seed, phase, drawn); helper: (draws left, drawn or None)
    start = ((0, 0, 0, -1), ("publish", 0, None), ((draws, None),) * helpers, ())
    stack, seen = [start], set()
    while stack:
        state = stack.pop()
        if state in seen:
            continue
        seen.add(state)
        (word, count, done, seed), owner, help_, ran = state
        phase, k, drawn = owner
        if phase == "end" and all(h == (0, None) for h in help_):
            yield ran
            continue
        # the owner's next step
        if phase == "publish":
            stack.append(((open_word(items[k]), items[k], 0, k), ("draw", k, None), help_, ran))
        elif phase == "draw":
            stack.append(((word + 1, count, done, seed), ("check", k, word), help_, ran))
        elif phase == "check":
            item = take(drawn, count)
            if item is None:
                stack.append(((word, count, done, seed), ("wait", k, None), help_, ran))
            else:
                stack.append(((word, count, done + 1, seed), ("draw", k, None), help_,
                              tuple(sorted(ran + ((seed, item),)))))
        elif phase == "wait" and done >= items[k]:
            if sum(1 for s, _ in ran if s == k) != items[k] or len(set(ran)) != len(ran):
                yield None
                continue
            nxt = ("publish", k + 1, None) if k + 1 < len(items) else ("end", k, None)
            stack.append(((open_word(0), 0 if not two_step else count, done, seed), nxt, help_, ran))
        # a helper's next step
        for i, (left, d) in enumerate(help_):
            if d is None and left:
                h = help_[:i] + ((left, word),) + help_[i + 1 :]
                stack.append(((word + 1, count, done, seed), owner, h, ran))
            elif d is not None:
                item = take(d, count)
                if item is None:  # it leaves
                    h = help_[:i] + ((0, None),) + help_[i + 1 :]
                    stack.append(((word, count, done, seed), owner, h, ran))
                else:
                    h = help_[:i] + ((left - 1, None),) + help_[i + 1 :]
                    stack.append(((word, count, done + 1, seed), owner, h, tuple(sorted(ran + ((seed, item),)))))


def test_every_item_runs_once_for_its_own_seed(loop):
    def take(drawn, _count):
        item = C.c_uint()
        return item.value if loop.take(drawn, C.byref(item)) else None

    runs = list(refine_runs(loop.open_word, take, False))
    assert runs and set(runs) == {((0, 0), (1, 0), (1, 1))}


def test_the_walk_sees_a_late_ticket():
    """The item and its bound read in two steps: a warp that drew past the end
    of one seed accepts the number as an item of the next."""
    closed = 1 << 30
    runs = list(refine_runs(lambda n: 0 if n else closed, lambda d, count: d if d < count else None, True))
    assert None in runs or any(r != ((0, 0), (1, 0), (1, 1)) for r in runs)


HOOK = C.CFUNCTYPE(None)
EMPTY = 0xFFFFFFFF


def test_a_ring_value_is_taken_once(loop):
    """Consumers of three laps at one place, each with what the others can do
    between its look at the place and its exchange."""
    place = C.c_uint(EMPTY)
    taken = []

    def put(v):
        return loop.ring_put(C.byref(place), C.c_uint(v))

    def take(hook=None):
        got = C.c_uint(EMPTY)
        ok = loop.ring_take(C.byref(place), C.byref(got), HOOK(hook) if hook else C.cast(None, HOOK))
        if ok:
            taken.append(got.value)
        return ok

    assert not take()  # nothing was put yet
    assert put(7) and not put(8)  # the place is full until 7 is taken
    # the consumer a lap later takes 7 after this one saw it: this one waits
    assert not take(lambda: take())
    assert taken == [7]
    # ... and gets the value put for the other
    assert put(8) and take()
    # between look and exchange the other takes the value and the next is put:
    # the exchange has the new value, each value went out once
    assert put(9) and take(lambda: (take(), put(10)))
    assert taken == [7, 8, 9, 10] and place.value == EMPTY


def test_heads_are_acquired_before_a_block_is_marked():
    """A block found ready from heads that other CTAs moved is kept by its
    finder: between the reads of the heads and the mark stands a fence of the
    threads that read them (no test on one GPU can show a stale line, so this
    reads the source)."""
    src = open(os.path.join(CSRC, "psod_sod.cu")).read()
    for fn, read, mark in (("bool mark_if_ready_warp(", "ld_state(&F.head[", "mark_ready("),
                           ("void finish_block(", "raw[e] = ld_state(&F.head[", "mark_ready(")):
        body = src[src.index(fn) :]
        body = body[: re.search(r"^}", body, re.M).end()]
        i = body.index(read)
        j = body.index(mark, i)
        assert "__threadfence()" in body[i:j], fn


@pytest.mark.parametrize("sides", [(1, 1, 1), (9, 9, 9), (33, 17, 25), (161, 161, 161), (161, 161, 162), (163, 163, 163),
                                   (4, 1024, 1024), (1023, 1, 4100), (1, 2047, 2049), (329, 329, 329), (401, 165, 401)])
def test_places_of_a_box(loop, sides):
    """Both sides of the 2^22 places up to which the FP32 quotient is exact."""
    assert loop.wrong_splits(*sides) == 0
