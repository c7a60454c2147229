"""The ring of raw blocks of the matmuls on pairs of CTAs (qmm_cp_kernel), as a model: a loader, copies that land in any order, two groups of warps
that take the chunks in turn, MMAs in order.  A wait on a barrier sees only whether the phase that ended last has the parity it asks for."""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dmlx_b200", "csrc", "qmm.cu")


class _Barrier:
    def __init__(self):
        self.phases, self.armed, self.bytes = 0, False, 0

    def passed(self, parity):
        return (self.phases - 1) & 1 == parity

    def arrive(self, copying=False):
        assert not self.armed, "arrived on twice in one phase"
        self.armed, self.bytes = True, int(copying)
        self._end()

    def landed(self):
        self.bytes = 0
        self._end()

    def _end(self):
        if self.armed and not self.bytes:
            self.phases, self.armed = self.phases + 1, False


def _run(slots, bars, stages, chunks, rng):
    full, free, done = ([_Barrier() for _ in range(n)] for n in (bars, bars, stages))
    content, flying, loaded, at, has_read, stored, multiplied = [None] * slots, [], 0, [0, 1], [False, False], set(), 0
    while multiplied < chunks:
        ready = []
        n = loaded  # the slot's last chunk was n - slots; a barrier that was never used lets parity 1 pass
        if n < chunks and free[(n - slots) % bars].passed((n - slots) // bars & 1):
            ready.append("load")
        ready += [("land", c) for c in flying]
        for g in (0, 1):
            i = at[g]
            if i < chunks and not has_read[g] and full[i % bars].passed(i // bars & 1):
                ready.append(("read", g))
            if i < chunks and has_read[g] and done[i % stages].passed((i // stages - 1) & 1):
                ready.append(("store", g))
        if multiplied in stored:
            ready.append("multiply")
        assert ready, "nothing can go on"
        # copies are late more often than not
        what = rng.choice([r for r in ready if r[0] != "land"] or ready) if rng.random() < 0.8 else rng.choice(ready)
        if what == "load":
            full[n % bars].arrive(copying=True)
            flying.append(n)
            loaded += 1
        elif what == "multiply":
            done[multiplied % stages].arrive()
            multiplied += 1
        elif what[0] == "land":
            flying.remove(what[1])
            content[what[1] % slots] = what[1]
            full[what[1] % bars].landed()
        elif what[0] == "read":
            i = at[what[1]]
            assert content[i % slots] == i, f"chunk {i} is read where {content[i % slots]} lies"
            free[i % bars].arrive()
            has_read[what[1]] = True
        else:
            i = at[what[1]]
            assert multiplied > i - stages, f"chunk {i} is stored where {i - stages} is still multiplied"
            stored.add(i)
            at[what[1]], has_read[what[1]] = i + 2, False


def _rings():
    text = open(SOURCE).read()
    slots = int(re.search(r"kRawSlots = kDense \? 0 : (\d+)", text).group(1))
    bars = re.search(r"kRawBars = (\d+) \* kRawSlots", text)
    return slots, slots * int(bars.group(1)) if bars else slots


@pytest.mark.parametrize("stages", [2, 4, 5, 6, 8])
def test_every_chunk_is_read_when_it_is_there(stages):
    for seed in range(300):
        _run(*_rings(), stages, 64, random.Random(seed))


def test_the_model_sees_a_wait_for_every_other_phase():
    with pytest.raises(AssertionError):
        for seed in range(300):
            _run(5, 5, 6, 64, random.Random(seed))
