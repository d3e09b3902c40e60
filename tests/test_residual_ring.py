"""The X ring of the tensor-core CP residual (residual_tc.cu k_residual_tc) as a
model on the CPU: a producer that loads tiles in order, loads that land in any
order, parity barriers, epilogue warps that each take one tile of a chunk.
Under random schedules no warp may read a tile that has not landed, and none
may lose its slot while it reads, at every ring depth the kernel can take."""
import os
import random
import re

import pytest

from conftest import PKG

SRC = open(os.path.join(PKG, "csrc", "residual_tc.cu")).read()


def _const(name):
    return int(re.search(r"constexpr int %s = (\d+);" % name, SRC).group(1))


PER_CHUNK = _const("RT_NJ") // _const("RT_XJ")  # X tiles per chunk
DEEPEST = _const("RT_XSMAX")
QUARTERS = 4                                    # warps that share a tile


def _kernel_guard():
    """Ring depth below which the kernel's warps wait for the issue first."""
    m = re.search(r"RT_XSFREE = (\d+) \* \(RT_NJ / RT_XJ\);", SRC)
    return int(m.group(1)) * PER_CHUNK if m and "if (mine && short_ring) rt_wait_issued" in SRC else 0


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passes(self, parity):
        return (self.phase & 1) != parity


def _run(xs, ntiles, nk, guard, rng):
    """One schedule; the first fault as text, or None."""
    nq = -(-ntiles // PER_CHUNK)
    chunks = [min(PER_CHUNK, ntiles - PER_CHUNK * q) for _ in range(nk) for q in range(nq)]
    total = ntiles * nk
    full, empty = [Barrier(1) for _ in range(xs)], [Barrier(QUARTERS) for _ in range(xs)]
    d_full, d_free = [Barrier(1) for _ in range(2)], [Barrier(PER_CHUNK * QUARTERS) for _ in range(2)]
    content, landed, flying, issued = [None] * xs, set(), [], 0
    reading = {}
    fault = []

    def producer():
        nonlocal issued
        for t in range(total):
            slot, use = t % xs, t // xs
            while use > 0 and not empty[slot].passes((use - 1) & 1):
                yield
            if any(s == slot for s in reading.values()):
                fault.append(f"tile {t} overwrites slot {slot} under a reader")
            content[slot] = t
            flying.append(t)
            issued += 1
            yield

    def mma():
        for ci in range(len(chunks)):
            while ci >= 2 and not d_free[ci & 1].passes(((ci >> 1) - 1) & 1):
                yield
            d_full[ci & 1].arrive()
            yield

    def epilogue(g, w):
        t = g
        for ci, tiles in enumerate(chunks):
            mine = g < tiles
            while not d_full[ci & 1].passes((ci >> 1) & 1):
                yield
            if mine:
                while xs < guard and issued <= t:
                    yield
                while not full[t % xs].passes((t // xs) & 1):
                    yield
                if content[t % xs] != t or t not in landed:
                    fault.append(f"chunk {ci}: tile {t} read before it landed")
                reading[g, w] = t % xs
                yield
                del reading[g, w]
                empty[t % xs].arrive()
            d_free[ci & 1].arrive()
            t += tiles
            yield

    actors = [producer(), mma()] + [epilogue(g, w) for g in range(PER_CHUNK) for w in range(QUARTERS)]
    weights = [rng.choice((1, 4, 20)) for _ in actors] + [rng.choice((1, 4))]
    idle = 0
    while actors:
        k = rng.choices(range(len(actors) + 1), weights)[0]
        if k == len(actors):  # one load lands, in no order
            if flying:
                t = flying.pop(rng.randrange(len(flying)))
                landed.add(t)
                full[t % xs].arrive()
        else:
            try:
                next(actors[k])
            except StopIteration:
                del actors[k], weights[k]
        if fault:
            return fault[0]
        idle += 1
        if idle > 200000:
            return "the schedule hangs"
    return None


@pytest.mark.parametrize("ntiles", [3, 13, 14, 16])
@pytest.mark.parametrize("xs", range(4, DEEPEST + 1))
def test_no_tile_is_read_before_it_lands(xs, ntiles):
    for seed in range(16):
        assert _run(xs, ntiles, 3, _kernel_guard(), random.Random(seed)) is None


def test_the_model_sees_the_missing_wait():
    assert any(_run(6, 16, 3, 0, random.Random(seed)) for seed in range(40))
