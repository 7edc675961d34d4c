"""Who waits for whom in the e4m3 gate/up GEMM of 64-row tiles, whose two promotion groups take narrow units in turn: a CTA's
UMMA warp, scale-table warp and eight promotion warps, step by step over many random schedules (CPU)."""

import random

import pytest

TABLES, ACCUMULATORS, WARPS = 2, 4, 8  # scale tables, accumulator stages, promotion warps (two groups of four)


class Barrier:
    """An mbarrier: a phase ends with the `expected`-th arrival; waits look at the parity of the phase only."""

    def __init__(self, expected):
        self.expected, self.pending, self.phase = expected, 0, 0

    def arrive(self, n=1):
        self.pending += n
        assert self.pending <= self.expected, "an arrival counts into the next phase"
        if self.pending == self.expected:
            self.pending, self.phase = 0, self.phase + 1

    def passed(self, parity):
        return (self.phase - 1) & 1 == parity & 1


class Cta:
    """One CTA's work.  `rule`: how a group passes a unit that is not its own.  "waits": it waits for the unit's table and
    arrives for itself on the barrier that frees it; "silent": the other group arrives for both; "at once": it arrives
    without the wait."""

    def __init__(self, units, report, rule="waits"):
        self.units, self.report, self.rule = units, report, rule  # units: (wide, K blocks)
        self.tbl_full, self.tbl_free = [Barrier(1) for _ in range(TABLES)], [Barrier(WARPS) for _ in range(TABLES)]
        self.acc_full, self.acc_empty = [Barrier(1) for _ in range(ACCUMULATORS)], [Barrier(WARPS) for _ in range(ACCUMULATORS)]
        self.stored = [Barrier(WARPS) for _ in range(2)]
        self.met = [Barrier(4) for _ in range(2)]
        self.table, self.acc = [None] * TABLES, [None] * ACCUMULATORS
        self.read = {}   # (unit, K block): promotion warps that are done with it
        self.left = {}   # unit: promotion warps that have stored it

    def owners(self, n):
        return 8 if self.units[n][0] else 4

    def umma(self):
        at = 0
        for n, (_, blocks) in enumerate(self.units):
            for j in range(blocks):
                s, phase = at % ACCUMULATORS, at // ACCUMULATORS
                yield self.acc_empty[s], phase + 1
                assert self.acc[s] is None or self.read.get(self.acc[s], 0) == self.owners(self.acc[s][0])
                self.acc[s] = (n, j)
                yield None
                self.acc_full[s].arrive()
                at += 1

    def tables(self):
        def stored(k):
            yield self.stored[k % 2], k >> 1
            assert self.left.get(k, 0) == self.owners(k), "reported before it is stored"

        for n in range(len(self.units)):
            if n >= TABLES:
                yield self.tbl_free[n % TABLES], n // TABLES - 1
                assert self.read.get((n - TABLES, self.units[n - TABLES][1] - 1), 0) == self.owners(n - TABLES)
            self.table[n % TABLES] = n
            if self.report and n >= 2:
                yield from stored(n - 2)
            self.tbl_full[n % TABLES].arrive()
            yield None
        for k in range(max(0, len(self.units) - 2), len(self.units)):
            if self.report:
                yield from stored(k)

    def promotion(self, group):
        at, skipped, met = 0, False, 0
        for n, (wide, blocks) in enumerate(self.units):
            buf, phase = n % TABLES, n // TABLES
            share = 1 if wide else 2
            if not wide and group != n & 1:
                if self.rule == "waits":
                    yield self.tbl_full[buf], phase
                if self.rule != "silent":
                    self.tbl_free[buf].arrive()
                at, skipped = at + blocks, True
                yield None
                continue
            if skipped:
                skipped = False
                yield self.tbl_free[(n - 1) % TABLES], (n - 1) // TABLES
                assert self.read.get((n - 1, self.units[n - 1][1] - 1), 0) == 4, "the other group is not done"
            yield self.tbl_full[buf], phase
            for j in range(blocks):
                s = at % ACCUMULATORS
                yield self.acc_full[s], at // ACCUMULATORS
                assert self.acc[s] == (n, j) and self.table[buf] == n, "another unit's sums or scales"
                yield None
                self.read[n, j] = self.read.get((n, j), 0) + 1
                self.acc_empty[s].arrive(share)
                at += 1
            self.tbl_free[buf].arrive(share if self.rule == "silent" else 1)
            for _ in range(2):  # the epilogue's meetings
                yield None
                self.met[group].arrive()
                yield self.met[group], met
                met += 1
            self.left[n] = self.left.get(n, 0) + 1
            if self.report:
                self.stored[n % 2].arrive(share)
            yield None

    def run(self, rng):
        """True when everybody is done, False when nobody can go on."""
        actors = [self.umma(), self.tables()] + [self.promotion(w // 4) for w in range(WARPS)]
        waits = {a: None for a in actors}
        speed = {a: 1.0 for a in actors}
        while actors:
            ready = [a for a in actors if waits[a] is None or waits[a][0].passed(waits[a][1])]
            if not ready:
                return False
            if rng.random() < 0.05:  # some fall behind for a while
                speed = {a: rng.choice((0.01, 0.1, 1.0)) for a in actors}
            a = rng.choices(ready, [speed[x] for x in ready])[0]
            try:
                waits[a] = next(a)
            except StopIteration:
                actors.remove(a)
        return True


def work(rng, blocks, n):
    pattern = rng.choice(("any", "narrow", "one wide"))
    wide = {"any": lambda i: rng.random() < 0.5, "narrow": lambda i: False, "one wide": lambda i: i % 3 == 1}[pattern]
    return [(wide(i), rng.choice(blocks)) for i in range(n)]


@pytest.mark.parametrize("report", [False, True])
@pytest.mark.parametrize("blocks", [(1,), (2,), (1, 2), (3,), (4, 8), (1, 2, 3, 4, 5, 9, 32)])
def test_every_schedule_ends_with_each_unit_read_from_its_own_sums(blocks, report):
    for seed in range(150 if max(blocks) < 9 else 40):
        rng = random.Random(seed)
        assert Cta(work(rng, blocks, 12), report).run(rng)


@pytest.mark.parametrize("rule", ["silent", "at once"])
def test_these_schedules_find_rules_that_do_not_hold(rule):
    found = 0
    for seed in range(200):
        rng = random.Random(seed)
        try:
            found += not Cta(work(rng, (1, 2), 12), False, rule).run(rng)
        except AssertionError:
            found += 1
    assert found > 10
