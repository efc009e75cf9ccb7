"""The barriers of the integer-tile Q4_K GEMM (csrc/gemm_q4k_int.cu) as a model on the CPU: roles of a pair of CTAs run in random
order over mbarriers with phases.  An arrive orders what its thread did before for waiters of the SAME CTA only: an arrive on the
other CTA's barrier carries no release at cluster scope, and a commit none at all.  Followed here: a row scale is written before
it is read by an order of that kind, no slot of the scales is overwritten before it is read, and no wait hangs."""
import random

import pytest

RING, SCALES = 4, 8


class Barrier:
    def __init__(self, cta, count):
        self.cta, self.count, self.left, self.phase, self.clock = cta, count, count, 0, {}

    def arrive(self, clock):
        for t, c in (clock or {}).items():
            self.clock[t] = max(self.clock.get(t, 0), c)
        self.left -= 1
        assert self.left >= 0
        if self.left == 0:
            self.phase, self.left = self.phase + 1, self.count

    def passed(self, parity):
        return self.phase % 2 != parity


class Pair:
    def __init__(self, sb, units, own_barriers):
        self.sb, self.units, self.own = sb, units, own_barriers
        self.full = [[Barrier(0, 3) for _ in range(RING)], [Barrier(1, 2) for _ in range(RING)]]  # builders (+ the other CTA's relay)
        self.done = [[Barrier(c, 1) for _ in range(RING)] for c in (0, 1)]
        self.scaled = [[Barrier(c, 1) for _ in range(RING)] for c in (0, 1)]
        self.empty = [Barrier(0, 2) for _ in range(2)]
        self.clocks, self.written, self.read = {}, {}, {}

    def tick(self, me):
        c = self.clocks.setdefault(me, {})
        c[me] = c.get(me, 0) + 1
        return c

    def arrive(self, me, bar):
        """a thread's arrive: orders nothing where the barrier is the other CTA's"""
        bar.arrive(dict(self.tick(me)) if me[0] == bar.cta else None)

    def seen(self, me, bar):
        assert me[0] == bar.cta
        c = self.tick(me)
        for t, v in bar.clock.items():
            c[t] = max(c.get(t, 0), v)

    def wait(self, me, bar, use):
        while not bar.passed(use % 2):
            yield
        self.seen(me, bar)

    def builder(self, cta, step):
        me = (cta, "builder", step)
        for g in range(2 * self.units):
            n = g // 2
            if g % 2 == 0 and step == 0:
                assert n < SCALES or (cta, n - SCALES) in self.read, "slot overwritten before it is read"
                self.written[cta, n % SCALES] = (n, me, self.tick(me)[me])
                yield
            if g >= self.sb:
                yield from self.wait(me, self.done[cta][(g - self.sb) % RING], (g - self.sb) // RING)
            if g % 2 == 0 and step == 0 and self.own:
                self.arrive(me, self.scaled[cta][n % RING])
            self.arrive(me, self.full[cta][g % RING])
            yield

    def relay(self):
        me = (1, "relay")
        for g in range(2 * self.units):
            yield from self.wait(me, self.full[1][g % RING], g // RING)
            self.arrive(me, self.full[0][g % RING])

    def mma(self, mine):
        me = (0, "mma", mine)
        for n in range(mine, self.units, 2):
            if n >= 2:
                yield from self.wait(me, self.empty[mine], n // 2 - 1)
            for g in (2 * n, 2 * n + 1):
                yield from self.wait(me, self.full[0][g % RING], g // RING)
                self.commits.append(g)
                yield

    def tensor_core(self):
        """completes what the two lanes issued, a unit's groups in order, for both CTAs"""
        for _ in range(2 * self.units):
            while not self.commits:
                yield
            g = self.commits.pop(0)
            for c in (0, 1):
                self.done[c][g % RING].arrive(None)
            yield

    def drain(self, cta):
        me = (cta, "drain")
        for n in range(self.units):
            g = 2 * n + 1
            if self.own:
                yield from self.wait(me, self.scaled[cta][n % RING], n // RING)
            yield from self.wait(me, self.done[cta][g % RING], g // RING)
            unit, writer, at = self.written[cta, n % SCALES]
            assert unit == n
            assert self.tick(me).get(writer, 0) >= at, "row scale read without an order after its write"
            yield
            self.read[cta, n] = True
            self.arrive(me, self.empty[n % 2])

    def run(self, rng):
        self.commits = []
        roles = [self.builder(c, s) for c in (0, 1) for s in (0, 1)] + [self.relay(), self.mma(0), self.mma(1), self.tensor_core(), self.drain(0), self.drain(1)]
        weight = [10.0 ** rng.uniform(-2, 0) for _ in roles]  # some roles are much slower than others
        for _ in range(400000):
            if not roles:
                return
            i = rng.choices(range(len(roles)), weight)[0]
            try:
                next(roles[i])
            except StopIteration:
                del roles[i], weight[i]
        raise AssertionError("a wait hangs")


@pytest.mark.parametrize("sb", [2, 3, 4])
def test_row_scales_are_ordered(sb):
    for seed in range(25):
        Pair(sb, 24, True).run(random.Random(seed))


def test_the_model_sees_a_missing_order():
    with pytest.raises(AssertionError, match="without an order"):
        Pair(4, 24, False).run(random.Random(0))


# ---- two sets of builders, several accumulators ----
BARS, SCALES2 = 16, 8


class PairOfSets(Pair):
    """Four groups a unit; builders of even and of odd units, each unit's groups by two of its set's warps; `accs` accumulators
    handed back by the drains; packed blocks in a ring of `sp` stages that completes out of order."""

    def __init__(self, sb, accs, sp, units):
        self.sb, self.accs, self.sp, self.units, self.own = sb, accs, sp, units, True
        self.full = [Barrier(0, 2) for _ in range(BARS)]  # one warp of either CTA
        self.done = [[Barrier(c, 1) for _ in range(BARS)] for c in (0, 1)]
        self.scaled = [[Barrier(c, 1) for _ in range(SCALES2)] for c in (0, 1)]
        self.packed = [[Barrier(c, 1) for _ in range(sp)] for c in (0, 1)]
        self.free = [[Barrier(c, 2) for _ in range(sp)] for c in (0, 1)]
        self.empty = [Barrier(0, 2) for _ in range(accs)]
        self.clocks, self.written, self.read = {}, {}, {}
        self.landing = {0: [], 1: []}
        self.stage = {0: {}, 1: {}}

    def packer(self, cta):
        me = (cta, "packer")
        for n in range(self.units):
            if n >= self.sp:
                yield from self.wait(me, self.free[cta][n % self.sp], n // self.sp - 1)
            self.landing[cta].append(n)
            yield

    def memory(self, cta, rng):
        """copies land in any order"""
        for _ in range(self.units):
            while not self.landing[cta]:
                yield
            n = self.landing[cta].pop(rng.randrange(len(self.landing[cta])))
            self.stage[cta][n % self.sp] = n
            self.packed[cta][n % self.sp].arrive(None)
            yield

    def builder(self, cta, odd, half):
        me = (cta, "builder", odd, half)
        for n in range(odd, self.units, 2):
            yield from self.wait(me, self.packed[cta][n % self.sp], n // self.sp)
            assert self.stage[cta].get(n % self.sp) == n, "another unit's packed block"
            if half == 0:
                assert n < SCALES2 or (cta, n - SCALES2) in self.read, "slot overwritten before it is read"
                self.written[cta, n % SCALES2] = (n, me, self.tick(me)[me])
            yield
            for h in (0, 1):
                g = 4 * n + 2 * half + h
                if g >= self.sb:
                    yield from self.wait(me, self.done[cta][(g - self.sb) % BARS], (g - self.sb) // BARS)
                    assert g - self.sb in self.finished, "a group of weights overwritten before it is multiplied"
                if h == 1:
                    self.arrive(me, self.free[cta][n % self.sp])
                    if half == 0:
                        self.arrive(me, self.scaled[cta][n % SCALES2])
                self.built.setdefault(g, set()).add(cta)
                self.arrive(me, self.full[g % BARS])
                yield

    def mma(self, mine):
        me = (0, "mma", mine)
        for n in range(mine, self.units, 2):
            if n >= self.accs:
                yield from self.wait(me, self.empty[n % self.accs], n // self.accs - 1)
                assert all((c, n - self.accs) in self.read for c in (0, 1)), "an accumulator overwritten before it is read"
            for g in range(4 * n, 4 * n + 4):
                yield from self.wait(me, self.full[g % BARS], g // BARS)
                assert self.built[g] == {0, 1}, "multiplied before it is built"
                self.commits.append(g)
                yield

    def tensor_core(self):
        for _ in range(4 * self.units):
            while not self.commits:
                yield
            g = self.commits.pop(0)
            self.finished.add(g)
            for c in (0, 1):
                self.done[c][g % BARS].arrive(None)
            yield

    def drain(self, cta):
        me = (cta, "drain")
        for n in range(self.units):
            yield from self.wait(me, self.scaled[cta][n % SCALES2], n // SCALES2)
            yield from self.wait(me, self.done[cta][(4 * n + 3) % BARS], (4 * n + 3) // BARS)
            assert 4 * n + 3 in self.finished
            unit, writer, at = self.written[cta, n % SCALES2]
            assert unit == n
            assert self.tick(me).get(writer, 0) >= at, "row scale read without an order after its write"
            yield
            self.read[cta, n] = True
            self.arrive(me, self.empty[n % self.accs])

    def run(self, rng):
        self.commits, self.finished, self.built = [], set(), {}
        roles = [self.builder(c, o, h) for c in (0, 1) for o in (0, 1) for h in (0, 1)]
        roles += [self.packer(0), self.packer(1), self.memory(0, rng), self.memory(1, rng), self.mma(0), self.mma(1), self.tensor_core(), self.drain(0), self.drain(1)]
        weight = [10.0 ** rng.uniform(-2, 0) for _ in roles]
        for _ in range(600000):
            if not roles:
                return
            i = rng.choices(range(len(roles)), weight)[0]
            try:
                next(roles[i])
            except StopIteration:
                del roles[i], weight[i]
        raise AssertionError("a wait hangs")


@pytest.mark.parametrize("sb,accs", [(8, 4), (7, 3), (8, 2), (6, 2), (4, 2)])
@pytest.mark.parametrize("sp", [2, 4])
def test_sets_of_builders(sb, accs, sp):
    for seed in range(25):
        PairOfSets(sb, accs, sp, 41).run(random.Random(seed))


def test_an_odd_ring_of_packed_blocks_is_caught():
    """With three stages a set of builders takes a stage's barrier for that of its own unit while the other set's copy is under way."""
    with pytest.raises(AssertionError):
        for seed in range(200):
            PairOfSets(8, 4, 3, 41).run(random.Random(seed))
