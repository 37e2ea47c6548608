"""Barrier protocol of the weight-gradient kernel (cnn.cuh, k_wgrad), simulated
on the CPU: the copying lane, the MMA-issuing warps (one per dz), the warps that sum
g, copies that land late and in any order, MMAs that finish late (each warp's in order, with
their commits), run in random interleavings.  No run may deadlock, overwrite a slot that an
unfinished MMA reads, or let an MMA read a plane other than its own.  The slots and the
arrivals that a phase takes are read from the kernel's source.
"""
import os
import random
import re

import pytest

with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       "distributednavierstokes_b200", "csrc", "cnn.cuh")) as f:
    SOURCE = f.read()
KERNEL = SOURCE[SOURCE.index("k_wgrad(const __grid_constant__"):]


def constant(name):
    return int(re.search(rf"constexpr int {name} = (\d+);", SOURCE).group(1))


def arrivals(bar):
    """The arrivals that complete a phase of a barrier: mb_init(&bar[i], a [+ b])."""
    return [int(v) for v in re.search(rf"mb_init\(&{bar}\[i\], (\d+(?: \+ \d+)?)\)", KERNEL).group(1).split(" + ")]


PLANES, GRADS = constant("WG_PLANES"), constant("WG_GRADS")
ISSUERS, SUMMERS = arrivals("gempty")
WARPS = constant("NTHREADS") // 32


def test_the_counts_are_those_of_the_roles():
    """One copying warp, ISSUERS issuing and SUMMERS summing; every issuing warp
    releases a plane of h, every one of both kinds a plane of g."""
    assert WARPS == 1 + ISSUERS + SUMMERS and ISSUERS == 3
    assert arrivals("hempty") == [ISSUERS] and arrivals("hfull") == arrivals("gfull") == [1]
    assert f"warp <= {ISSUERS})" in KERNEL       # the issuing warps; those above sum


class Bar:
    """mbarrier: phase parity only, as a waiter sees it."""

    def __init__(self, count):
        self.done, self.count, self.pend = 0, count, 0

    def complete(self):
        self.pend += 1
        if self.pend == self.count:
            self.done, self.pend = self.done + 1, 0

    def passed(self, parity):
        # the phase of this parity has completed: the current phase has the other one
        return (self.done & 1) != parity


def simulate(B, kpp, Do, nsplit, split, rng):
    n = B * kpp * Do
    s0, s1 = n * split // nsplit, n * (split + 1) // nsplit
    hfull, hempty = [Bar(1) for _ in range(PLANES)], [Bar(ISSUERS) for _ in range(PLANES)]
    gfull, gempty = [Bar(1) for _ in range(GRADS)], [Bar(ISSUERS + SUMMERS) for _ in range(GRADS)]
    hslot, gslot = [None] * PLANES, [None] * GRADS
    copies = []                                  # in flight
    mmas = [[], [], []]                          # per lane: (slots read, barriers to arrive on)
    read = [[], [], []]

    def under_mma(slot):
        return any(slot in m[0] for lane in mmas for m in lane)

    def land(kind, slot, what, bar):
        (hslot if kind == "h" else gslot)[slot] = what
        bar.complete()

    def producer():
        pl = gi = 0
        for s in range(s0, s1):
            col, z = divmod(s, Do)
            for pz in range(z if s == s0 or z == 0 else z + 2, z + 3):
                sl = pl % PLANES
                while not hempty[sl].passed(((pl // PLANES) & 1) ^ 1):
                    yield "wait"
                assert not under_mma(("h", sl)), "plane overwritten under an MMA"
                copies.append(("h", sl, (col, pz), hfull[sl]))
                pl += 1
                yield "go"
            st = gi % GRADS
            while not gempty[st].passed(((gi // GRADS) & 1) ^ 1):
                yield "wait"
            assert not under_mma(("g", st)), "g overwritten under an MMA"
            copies.append(("g", st, (col, z), gfull[st]))
            gi += 1
            yield "go"

    def issuer(dz):
        pl = g0 = 0
        s = s0
        while s < s1:
            n = min(s1 - s, Do - s % Do)
            for j in range(n + 2):
                sl = pl % PLANES
                while not hfull[sl].passed((pl // PLANES) & 1):
                    yield "wait"
                pl += 1
                if j < dz or j - dz >= n:
                    hempty[sl].complete()
                    yield "go"
                    continue
                gi = g0 + j - dz
                st = gi % GRADS
                while not gfull[st].passed((gi // GRADS) & 1):
                    yield "wait"
                col, z = divmod(s + j - dz, Do)
                assert gslot[st] == (col, z)
                assert hslot[sl] == (col, z + dz)
                mmas[dz].append(([("g", st), ("h", sl)], [gempty[st], hempty[sl]]))
                read[dz].append(s + j - dz)
                yield "go"
            s += n
            g0 += n

    def summer(out):
        for gi in range(s1 - s0):
            st = gi % GRADS
            while not gfull[st].passed((gi // GRADS) & 1):
                yield "wait"
            assert gslot[st] == divmod(s0 + gi, Do)
            yield "go"                           # reading: nothing may land in the slot meanwhile
            assert gslot[st] == divmod(s0 + gi, Do)
            out.append(s0 + gi)
            gempty[st].complete()
            yield "go"

    summed = [[] for _ in range(SUMMERS)]
    agents = {"p": producer(), **{dz: issuer(dz) for dz in range(ISSUERS)},
              **{f"s{i}": summer(out) for i, out in enumerate(summed)}}
    idle = 0
    while agents or copies or any(mmas):
        acts = list(agents) + (["copy"] if copies else []) + [("mma", d) for d in range(3) if mmas[d]]
        a = rng.choice(acts)
        if a == "copy":
            land(*copies.pop(rng.randrange(len(copies))))
            idle = 0
        elif isinstance(a, tuple):
            for f in mmas[a[1]].pop(0)[1]:
                f.complete()
            idle = 0
        else:
            try:
                idle = idle + 1 if next(agents[a]) == "wait" else 0
            except StopIteration:
                del agents[a]
        assert idle < 2000, "deadlock"
    assert read == [list(range(s0, s1))] * ISSUERS and summed == [list(range(s0, s1))] * SUMMERS


@pytest.mark.parametrize("B,kpp,Do,nsplit", [(1, 1, 1, 1), (1, 2, 1, 1), (2, 3, 2, 1), (2, 2, 5, 3),
                                             (3, 2, 4, 5), (2, 4, 7, 9), (1, 5, 3, 15), (2, 3, 9, 4)])
def test_no_deadlock_no_overwrite(B, kpp, Do, nsplit):
    rng = random.Random(1)
    for split in range(nsplit):
        for _ in range(20):
            simulate(B, kpp, Do, nsplit, split, rng)
