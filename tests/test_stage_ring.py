"""CPU check of the stage ring of the pipelined binary-coded GEMV (`csrc/stage_ring.h`): producer, consumer warps and barrier
phases are replayed with copies that land late and out of order.  The schedule and the parities come from the header itself, compiled
here; the order of the waits is the kernel's."""
import ctypes
import functools
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "decdec_b200" / "csrc"
WRAPPERS = """
#include "stage_ring.h"
extern "C" {
uint32_t fulls(uint32_t s, uint32_t g) { return dd::ring_full_barriers(s, g); }
uint32_t place(uint32_t i, uint32_t n) { return dd::ring_place(i, n, dd::ring_inverse(n)); }
uint32_t parity(uint32_t i, uint32_t n) { return dd::ring_parity(i, dd::ring_inverse(n)); }
}
"""


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(WRAPPERS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "ring.cpp"), "-o", str(d / "ring.so")], check=True)
    lib = ctypes.CDLL(str(d / "ring.so"))

    class Ring:
        fulls = lib.fulls
        place, parity = staticmethod(functools.cache(lib.place)), staticmethod(functools.cache(lib.parity))
    return Ring


class OneBarrierPerSlot:
    """The rule that the header excludes."""
    fulls = staticmethod(lambda s, g: s)
    place = staticmethod(lambda i, n: i % n)
    parity = staticmethod(lambda i, n: i // n & 1)


class Barrier:
    """mbarrier: a wait with parity p returns once the current phase's parity differs from p."""
    def __init__(self, count):
        self.count, self.phase, self.left, self.tx = count, 0, count, 0

    def passes(self, parity):
        return self.phase & 1 != parity

    def settle(self):
        if self.left == 0 and self.tx == 0:
            self.phase, self.left = self.phase + 1, self.count

    def arrive(self):
        assert self.left > 0, "an arrival too many in one phase"
        self.left -= 1
        self.settle()


def replay(ring, slots, stages, rng, warps=2, groups=3):
    """One run under a random schedule; some copies and some warps are held back for long."""
    copies = 2
    fulls = ring.fulls(slots, groups)
    full = [Barrier(1) for _ in range(fulls)]
    free = [Barrier(warps) for _ in range(slots)]
    landed = [set() for _ in range(slots)]                 # (stage, part) now in a slot
    readers = [set() for _ in range(slots)]
    flying, taken = [], {}

    def producer():
        for i in range(stages):
            s, b = ring.place(i, slots), ring.place(i, fulls)
            if i >= slots:
                while not free[s].passes(ring.parity(i - slots, slots)):
                    yield
            full[b].tx += copies
            full[b].arrive()
            flying.extend((i, part) for part in range(copies))
            yield

    def copy_lands():
        while True:
            if flying and rng.random() < lands:
                i, part = flying.pop(rng.randrange(len(flying)) if rng.random() < 0.8 else -1)
                s, b = ring.place(i, slots), ring.place(i, fulls)
                assert not readers[s], f"stage {i} lands in a slot that is being read"
                if any(stage != i for stage, _ in landed[s]):
                    landed[s].clear()
                landed[s].add((i, part))
                full[b].tx -= 1
                full[b].settle()
            yield

    def warp(group, w):
        for i in range(group, stages, groups):
            s, b = ring.place(i, slots), ring.place(i, fulls)
            while not full[b].passes(ring.parity(i, fulls)):
                yield
            assert landed[s] == {(i, part) for part in range(copies)}, f"group {group} passed to stage {i} before it landed"
            readers[s].add((group, w))
            for _ in range(rng.randrange(4)):
                yield
            assert landed[s] == {(i, part) for part in range(copies)}, f"stage {i} was overwritten while it was read"
            readers[s].remove((group, w))
            taken[i, w] = taken.get((i, w), 0) + 1
            free[s].arrive()
            yield

    lands = rng.choice((1.0, 0.3, 0.05))
    agents = [producer(), copy_lands()] + [warp(g, w) for g in range(groups) for w in range(warps)]
    pace = [1.0 if a == 1 else rng.choice((1.0, 1.0, 0.1)) for a in range(len(agents))]
    left = set(range(len(agents))) - {1}
    for _ in range(20000 * (stages + 1)):
        if not left:
            break
        a = rng.randrange(len(agents))
        if rng.random() > pace[a] or (a != 1 and a not in left):
            continue
        try:
            next(agents[a])
        except StopIteration:
            left.discard(a)
    assert not left, "a wait never ended"
    assert taken == {(i, w): 1 for i in range(stages) for w in range(warps)}


@pytest.mark.parametrize("slots", range(1, 9))
def test_no_group_passes_before_its_stage(ring, slots):
    rng = random.Random(slots)
    for stages in range(1, 17):
        for _ in range(25):
            replay(ring, slots, stages, rng)


@pytest.mark.parametrize("n", range(1, 17))
def test_places_of_long_tiles(ring, n):
    for i in range(1 << 12):
        assert (ring.place(i, n), ring.parity(i, n)) == (i % n, i // n & 1)


def test_barriers_fit_the_header(ring):
    assert [ring.fulls(s, 3) for s in range(1, 9)] == [4, 6, 3, 8, 10, 6, 14, 16]


@pytest.mark.parametrize("slots,stages", [(2, 6), (4, 12), (5, 15)])
def test_replay_sees_one_barrier_per_slot(slots, stages):
    """Two slots fail by themselves; four and five rely on the order in which copies land."""
    rng = random.Random(0)
    with pytest.raises(AssertionError):
        for _ in range(3000):
            replay(OneBarrierPerSlot, slots, stages, rng)
