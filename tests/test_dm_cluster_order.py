"""Order of the shared-memory accesses between the blocks of a cluster in the
density-matrix sweep of windows 9 and 10 (csrc/dm_fact.cuh, dm_fwd_fact_cl), by
the memory model: a store into another block's shared memory has to come after
every earlier read of that place.  The kernel's accesses and barriers are replayed
with vector clocks, the arrival's form (release or relaxed: a relaxed arrival
orders nothing before it) read from the source (no GPU)."""
import itertools
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "mentpy_gb300", "csrc", "dm_fact.cuh")
BLOCKS, WARPS = 2, 2  # warp 0 sends and arrives apart from the others


class Cluster:
    """Vector clocks of BLOCKS x WARPS warps; a phase runs warp by warp."""

    def __init__(self):
        self.n = BLOCKS * WARPS
        self.clock = [[0] * self.n for _ in range(self.n)]
        self.reads, self.races = {}, []

    def warps(self):
        return [(b * WARPS + w, b, w) for b in range(BLOCKS) for w in range(WARPS)]

    def _tick(self, t):
        self.clock[t][t] += 1

    def read(self, t, place):
        self._tick(t)
        self.reads.setdefault(place, []).append((t, self.clock[t][t]))

    def write(self, t, place):
        self._tick(t)
        for r, at in self.reads.pop(place, []):
            if self.clock[t][r] < at:
                self.races.append((place, r, t))

    def _join(self, group, published):
        top = [max([self.clock[p][i] for p in published] or [0]) for i in range(self.n)]
        for t in group:
            self.clock[t] = [max(a, b) for a, b in zip(self.clock[t], top)]

    def block_barrier(self):
        for b in range(BLOCKS):
            g = range(b * WARPS, (b + 1) * WARPS)
            self._join(g, g)

    def cluster_barrier(self, release):  # release(warp): its arrival's form
        self._join(range(self.n), [t for t, _, w in self.warps() if release(w)])


def _source(begin, end):
    s = open(SRC).read()
    s = s[s.index("dm_fwd_fact_cl(DmArgs A)"):]
    i = s.index(begin)
    return s[i:s.index(end, i)]


def test_layout_change_stores_after_every_load():
    arrive = re.findall(r"cluster_arrive\w*\(\)", _source("unit(l1, y);", "row_ptr"))
    assert len(arrive) == 1
    c = Cluster()
    for _ in range(2):  # from one layout to the other and back
        for t, b, w in c.warps():
            c.read(t, ("rows", b, w))
        c.cluster_barrier(lambda w: arrive[0] == "cluster_arrive()")
        for t, b, w in c.warps():
            c.write(t, ("rows", 1 - b, w))
        c.cluster_barrier(lambda w: True)
    assert not c.races


@pytest.mark.parametrize("kinds", list(itertools.product([(0,), (0, 1), (0, 2), (0, 1, 2)], repeat=3)))
def test_partials_are_sent_after_every_read_of_their_buffer(kinds):
    """kinds: the exchanges of each step (a Z step needs the trace, outcome 1 prob1)."""
    text = _source("auto exchange", "return collect();")
    assert len(re.findall(r"cluster_arrive", text)) == 3 and "if (tid < 32)" in text
    relaxed = re.search(r"else if \(what == (\d)\) \{\s*cluster_arrive_relaxed\(\);", text)
    c, par = Cluster(), 0
    for what in kinds + kinds[:1]:
        for x in what:
            for t, b, w in c.warps():
                if w == 0:
                    for other in range(BLOCKS):
                        c.write(t, (other, par, b))
            c.cluster_barrier(lambda w: w == 0 or x != int(relaxed.group(1)))
            for t, b, w in c.warps():
                for r in range(BLOCKS):
                    c.read(t, (b, par, r))
            par ^= 1
        c.block_barrier()  # the pass
    assert not c.races
