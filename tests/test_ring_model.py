"""CPU models of the rings that a producer warp fills by TMA and consumer warps
release: mbarrier counts, parities and slots as the kernels have them, run
under random interleavings.  Every read must find the plane it expects, no box
may land on a plane that some warp still reads, and every wait must end.

Models: the tiled entry of stencil functions (jit.cpp: two groups in flight),
the point sweeps (points_body.cuh: full, raw and empty barriers, planes in one
sequence over a CTA's items), the 7-point batch (batch.cu, s7_body.cuh: stages
released one at a time) and Himeno's two rings (himeno_body.cuh)."""
import random

import pytest


class Bar:
    """An mbarrier: completed phases, arrivals still pending, a box in flight."""

    def __init__(self, count):
        self.count, self.pending, self.phases, self.tx = count, count, 0, 0

    def _settle(self):
        if self.pending == 0 and self.tx == 0:
            self.phases += 1
            self.pending = self.count

    def arrive(self):
        assert self.pending > 0
        self.pending -= 1
        self._settle()

    def expect(self):  # arrive.expect_tx
        self.tx += 1
        self.arrive()

    def landed(self):
        self.tx -= 1
        self._settle()

    def done(self, parity):  # test_wait.parity
        return (self.phases & 1) != (parity & 1)


class Copies:
    """Boxes in flight: each lands at some later time."""

    def __init__(self, ring, rng):
        self.ring, self.rng, self.flying = ring, rng, []

    def issue(self, bar, slot, value):
        assert self.ring.readers[slot] == 0, "a box lands on a slot that is read"
        self.ring.data[slot] = None
        self.flying.append((bar, slot, value))

    def land(self):
        bar, slot, value = self.flying.pop(self.rng.randrange(len(self.flying)))
        assert self.ring.readers[slot] == 0
        self.ring.data[slot] = value
        bar.landed()


class Ring:
    def __init__(self, n):
        self.data, self.readers = [None] * n, [0] * n


def run(actors, copies, rng):
    """Runs the actors (generators that yield a condition to wait for, or None)
    in a random order until all have ended."""
    waits = {a: None for a in actors}
    idle = 0
    while waits or copies.flying:
        ready = [a for a, w in waits.items() if w is None or w()]
        if copies.flying and (not ready or rng.random() < 0.4):
            copies.land()
            idle = 0
            continue
        assert ready, "every actor waits and no box is in flight"
        a = ready[rng.randrange(len(ready))]
        try:
            waits[a] = next(a)
        except StopIteration:
            del waits[a]
        idle += 1
        assert idle < 100000


def held(ring, slots):
    for s in slots:
        ring.readers[s] += 1


def dropped(ring, slots):
    for s in slots:
        ring.readers[s] -= 1


# ---- tiled entry of stencil functions -----------------------------------------

def function_producer(n, rz, edge, full, raw, empty, copies, ring):
    S = 2 * rz + 2
    for i in range(n):
        if i >= 2:
            yield lambda i=i: empty[i & 1].done(((i - 2) >> 1) & 1)
        bar = raw[i & 1] if edge else full[i & 1]
        planes = range(2 * rz + 1) if i == 0 else [i + 2 * rz]
        bar.tx += len(planes)
        bar.arrive()
        for p in planes:
            copies.issue(bar, p if i == 0 else p % S, p)
        if edge:
            yield lambda bar=bar, i=i: bar.done((i >> 1) & 1)
            for p in planes:  # the halo rewritten in the plane that has landed
                assert ring.data[p % S] == p
            full[i & 1].arrive()
        yield None


def function_consumer(n, rz, full, empty, ring):
    S = 2 * rz + 2
    for i in range(n):
        yield lambda i=i: full[i & 1].done((i >> 1) & 1)
        slots = [(i + d) % S for d in range(2 * rz + 1)]
        held(ring, slots)
        yield None
        assert [ring.data[s] for s in slots] == [i + d for d in range(2 * rz + 1)]
        dropped(ring, slots)
        empty[i & 1].arrive()


@pytest.mark.parametrize("rz", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 16])
@pytest.mark.parametrize("warps,edge", [(4, False), (4, True), (16, False), (16, True)])
def test_function_ring(rz, n, warps, edge):
    for seed in range(6):
        rng = random.Random(seed)
        ring = Ring(2 * rz + 2)
        full, raw = [Bar(1) for _ in range(2)], [Bar(1) for _ in range(2)]
        empty = [Bar(warps) for _ in range(2)]
        copies = Copies(ring, rng)
        run([function_producer(n, rz, edge, full, raw, empty, copies, ring)]
            + [function_consumer(n, rz, full, empty, ring) for _ in range(warps)], copies, rng)


# ---- point sweeps --------------------------------------------------------------

def points_producer(items, ahead, full, raw, empty, copies, ring, rng):
    """items: (planes stepped, edge tile) of each; plane labels are (item, q)."""
    nst = len(ring.data)
    slot = fslot = phase = raws = 0
    used = False
    for it, (n, fix) in enumerate(items):
        filled = done = 0
        while done < n:
            while filled < n and filled - done < nst:
                if used:
                    par = ((phase >> slot) & 1) ^ 1
                    if fix and filled > done:
                        if not empty[slot].done(par):
                            break
                    else:
                        yield lambda s=slot, p=par: empty[s].done(p)
                bar = raw[slot] if fix else full[slot]
                bar.expect()
                copies.issue(bar, slot, (it, filled))
                phase ^= 1 << slot
                slot += 1
                if slot == nst:
                    slot, used = 0, True
                filled += 1
                if not fix:
                    done += 1
                    fslot = (fslot + 1) % nst
                if rng.random() < 0.3:
                    yield None
            if not fix:
                continue
            yield lambda s=fslot, p=(raws >> fslot) & 1: raw[s].done(p)
            raws ^= 1 << fslot
            assert ring.data[fslot] == (it, done)
            full[fslot].arrive()
            fslot = (fslot + 1) % nst
            done += 1
    for s in range(nst):  # the last copies land before the CTA may end
        if used or s < slot:
            yield lambda s=s, p=((phase >> s) & 1) ^ 1: full[s].done(p)


def points_consumer(items, zext, full, empty, ring):
    nst = len(ring.data)
    cs = wslot = phase = 0
    for it, (n, _) in enumerate(items):
        steps, waited = n - zext, 0
        for k in range(steps):
            while waited <= k + zext:
                yield lambda s=wslot, p=(phase >> wslot) & 1: full[s].done(p)
                phase ^= 1 << wslot
                waited += 1
                wslot = (wslot + 1) % nst
            slots = [(cs + l) % nst for l in range(zext + 1)]
            held(ring, slots)
            yield None
            assert [ring.data[s] for s in slots] == [(it, k + l) for l in range(zext + 1)]
            dropped(ring, slots)
            for _ in range(1 if k + 1 < steps else 1 + zext):
                empty[cs].arrive()
                cs = (cs + 1) % nst


@pytest.mark.parametrize("zext", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("ahead", [1, 2])
@pytest.mark.parametrize("warps", [1, 4])
def test_points_ring(zext, ahead, warps):
    for seed in range(12):
        rng = random.Random(seed)
        items = [(rng.choice([1, 2, 3, 9]) + zext, rng.random() < 0.5)
                 for _ in range(rng.choice([1, 2, 5]))]
        nst = zext + 1 + ahead
        ring = Ring(nst)
        full, raw = [Bar(1) for _ in range(nst)], [Bar(1) for _ in range(nst)]
        empty = [Bar(warps) for _ in range(nst)]
        copies = Copies(ring, rng)
        run([points_producer(items, ahead, full, raw, empty, copies, ring, rng)]
            + [points_consumer(items, zext, full, empty, ring) for _ in range(warps)], copies, rng)


# ---- batches and Himeno ---------------------------------------------------------

class Pos:
    """RingPos / HRing: a stage and the phase of its next completion."""

    def __init__(self):
        self.stage, self.phase = 0, 0

    def advance(self, n):
        self.stage += 1
        if self.stage == n:
            self.stage, self.phase = 0, self.phase ^ 1


def march_producer(items, rings):
    """rings: (full, empty, copies, ring, planes ahead of the first step)."""
    pos = [Pos() for _ in rings]
    for it, n in enumerate(items):
        for q in range(-2, n):
            for r, (full, empty, copies, ring, lead) in enumerate(rings):
                if q < -lead:
                    continue
                p = pos[r]
                yield lambda e=empty, s=p.stage, f=p.phase ^ 1: e[s].done(f)
                full[p.stage].expect()
                copies.issue(full[p.stage], p.stage, (r, it, q))
                p.advance(len(ring.data))


def batch7_consumer(items, full, empty, ring):
    ns = len(ring.data)
    cons, rel = Pos(), Pos()

    def release():
        empty[rel.stage].arrive()
        rel.advance(ns)

    for it, n in enumerate(items):
        window = []
        for q in range(-2, n):
            yield lambda s=cons.stage, f=cons.phase: full[s].done(f)
            window.append((cons.stage, (0, it, q)))
            cons.advance(ns)
            if q == -2:
                continue
            # plane q's cells go to registers; the row halo of plane q - 1 is read
            slots = [s for s, _ in window[-2:]]
            held(ring, slots)
            yield None
            assert [ring.data[s] for s, _ in window[-2:]] == [v for _, v in window[-2:]]
            dropped(ring, slots)
            release()
        release()


def himeno_consumer(items, p, c):
    (pfull, pempty, _, pring, _), (cfull, cempty, _, cring, _) = p, c
    pc, prel, cc = Pos(), Pos(), Pos()
    nsp, nsc = len(pring.data), len(cring.data)
    for it, n in enumerate(items):
        window = []
        for q in range(-2, n):
            yield lambda s=pc.stage, f=pc.phase: pfull[s].done(f)
            window.append((pc.stage, (0, it, q)))
            pc.advance(nsp)
            if q < 0:
                continue
            yield lambda s=cc.stage, f=cc.phase: cfull[s].done(f)
            slots = [s for s, _ in window[-3:]]
            held(pring, slots)
            held(cring, [cc.stage])
            yield None
            assert [pring.data[s] for s in slots] == [v for _, v in window[-3:]]
            assert cring.data[cc.stage] == (1, it, q)
            dropped(pring, slots)
            dropped(cring, [cc.stage])
            pempty[prel.stage].arrive()
            prel.advance(nsp)
            cempty[cc.stage].arrive()
            cc.advance(nsc)
        for _ in range(2):
            pempty[prel.stage].arrive()
            prel.advance(nsp)


def _ring(n, warps, rng, lead):
    ring = Ring(n)
    return [Bar(1) for _ in range(n)], [Bar(warps) for _ in range(n)], Copies(ring, rng), ring, lead


class Both:
    """The copies of two rings."""

    def __init__(self, a, b, rng):
        self.parts, self.rng = (a, b), rng

    @property
    def flying(self):
        return self.parts[0].flying + self.parts[1].flying

    def land(self):
        self.rng.choice([p for p in self.parts if p.flying]).land()


@pytest.mark.parametrize("ns", [2, 3, 4, 8])
@pytest.mark.parametrize("warps", [1, 4])
def test_batch7_ring(ns, warps):
    for seed in range(12):
        rng = random.Random(seed)
        items = [rng.choice([1, 2, 5]) for _ in range(rng.choice([1, 4]))]
        r = _ring(ns, warps, rng, 2)
        run([march_producer(items, [r])]
            + [batch7_consumer(items, r[0], r[1], r[3]) for _ in range(warps)], r[2], rng)


@pytest.mark.parametrize("nsp,nsc", [(3, 1), (4, 2), (5, 2), (16, 8)])
@pytest.mark.parametrize("warps", [1, 4])
def test_himeno_rings(nsp, nsc, warps):
    for seed in range(12):
        rng = random.Random(seed)
        items = [rng.choice([1, 2, 5]) for _ in range(rng.choice([1, 4]))]
        p, c = _ring(nsp, warps, rng, 2), _ring(nsc, warps, rng, 0)
        run([march_producer(items, [p, c])] + [himeno_consumer(items, p, c) for _ in range(warps)],
            Both(p[2], c[2], rng), rng)
