"""The waits of the fused quantized GEMM (csrc/tl_qgemm.cu), walked on the host for every instantiated tile: producer, converter groups
and MMA issuer step by step in random order, loads that land late.  A wait names the parity of a phase; it must never pass in another
phase than the one it means, and nobody may be left waiting."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRINT = """
#include <cstdio>
#include "tl_qgemm_ring.h"
int main() {
  for (const TcConfig& c : kTcConfigs) {
    const TcRing r = tl_tc_ring(c);
    std::printf("%d %d %d %d %d %d %d\\n", c.bn, c.kstep, c.stages, c.ncw, r.slots, r.groups, int(r.slot_first));
  }
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src, exe = d / "ring.cpp", d / "ring"
    src.write_text(PRINT)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "torchlette_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    return [tuple(map(int, line.split())) for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]


class Barrier:
    def __init__(self, arrivals=1):
        self.need, self.got, self.phase = arrivals, 0, 0

    def arrive(self):
        self.got += 1
        if self.got == self.need:
            self.got, self.phase = 0, self.phase + 1


def walk(stages, slots, groups, slot_first, steps, seed):
    """The first wait that passed in a phase that it did not mean, or None; a walk that stops short is an error."""
    rng = random.Random(seed)
    full, empty = [Barrier() for _ in range(stages)], [Barrier() for _ in range(stages)]
    ready, free = [Barrier() for _ in range(slots)], [Barrier() for _ in range(slots)]
    loads, mmas, wrong = [], [], []

    def wait(what, it, barrier, use):  # until completion number `use` (from 0) of the barrier, by parity as the hardware does
        while barrier.phase & 1 == use & 1:
            yield
        if barrier.phase != use + 1:
            wrong.append((what, it))

    def producer():
        for it in range(steps):
            if it >= stages:
                yield from wait("empty", it, empty[it % stages], it // stages - 1)
            loads.append((it, rng.random() < 0.05))
            yield

    def converter(group):
        def slot(it):
            if it >= slots:
                yield from wait("slot", it, free[it % slots], it // slots - 1)
        for it in range(group, steps, groups):
            if slot_first:
                yield from slot(it)
            yield from wait("full", it, full[it % stages], it // stages)
            yield
            if not slot_first:
                yield from slot(it)
            ready[it % slots].arrive()
            yield

    def issuer():
        for it in range(steps):
            yield from wait("full (mma)", it, full[it % stages], it // stages)
            yield from wait("ready", it, ready[it % slots], it // slots)
            mmas.append(it)
            yield

    def memory():  # lands loads in any order, late ones rarely; runs MMAs in order
        while True:
            if loads and rng.random() < 0.5:
                i = rng.randrange(len(loads))
                if not loads[i][1] or rng.random() < 0.01:
                    full[loads.pop(i)[0] % stages].arrive()
            if mmas and rng.random() < 0.7:
                it = mmas.pop(0)
                empty[it % stages].arrive()
                free[it % slots].arrive()
            yield

    agents = [producer(), issuer()] + [converter(g) for g in range(groups)]
    mem = memory()
    for _ in range(4000 * steps):
        a = rng.randrange(len(agents) + 1)
        if a == len(agents):
            next(mem)
        else:
            try:
                next(agents[a])
            except StopIteration:
                del agents[a]
        if wrong:
            return wrong[0]
        if not agents:
            return None
    raise AssertionError("a wait never ended")


def test_no_wait_passes_in_another_phase(tiles):
    assert len(tiles) >= 10 and any(t[5] == 2 for t in tiles)
    for bn, kstep, stages, ncw, slots, groups, slot_first in tiles:
        assert 2 <= slots <= stages
        for seed in range(20):
            assert walk(stages, slots, groups, slot_first, 60, seed) is None, (bn, kstep, stages, ncw)


def test_the_walk_sees_a_wait_that_is_too_early():
    """Two groups on an odd ring that look at the stage before they wait for their slot."""
    assert any(walk(3, 2, 2, False, 60, seed) for seed in range(20))
