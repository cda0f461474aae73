"""The barriers of a CTA pair in the tensor-core prefill kernel, as a model whose roles run in random order.

A wait looks at one bit, the parity of the phase.  It is right as long as the barrier can neither be a phase
behind the one waited for nor a phase beyond it: a wait that passes early reads or overwrites what is in use, one
that comes two phases late never ends.  The model knows the phase that each wait means and checks both.
"""
import random

import pytest

BUFS = 3


class Wrong(Exception):
    pass


class Bar:
    def __init__(self, count):
        self.count = self.left = count
        self.tx = self.done = 0

    def add(self, arrivals=0, tx=0):
        self.left -= arrivals
        self.tx += tx
        if self.left == 0 and self.tx == 0:
            self.done += 1
            self.left = self.count
        if self.left < 0:
            raise Wrong("an arrival too many")


class Pair:
    """units: (key tiles, blocks of the last tile, whether CTA 0 has rows)."""

    def __init__(self, units, rng, wait_without_keys=False):
        self.units, self.rng, self.wait_without_keys = units, rng, wait_without_keys
        both = lambda n, counts: [[Bar(counts) for _ in range(n)] for _ in range(2)]  # noqa: E731
        self.q_ready = [Bar(1) for _ in range(2)]
        self.rows_set = both(2, 4)
        self.scores_go = [Bar(2) for _ in range(BUFS)]
        self.s_full, self.pv_done = both(BUFS, 1), both(BUFS, 1)
        self.pv_go = [[Bar(10) for _ in range(BUFS)], [Bar(8) for _ in range(BUFS)]]
        self.o_free = Bar(8)
        self.l_set = both(2, 4)
        self.m = [[-1, -1], [-1, -1]]  # of a CTA and group: the tile its maximum stands after
        self.pipe, self.copies = [], []  # products in order; copies in any
        for b in self.scores_go:
            b.add(1)

    def wait(self, bar, phase):
        while (bar.done & 1) == (phase & 1):  # the parity that the hardware compares
            if bar.done > phase:
                raise Wrong(f"waits for phase {phase}, {bar.done} are over")
            yield
        if bar.done != phase + 1:
            raise Wrong(f"phase {phase} was waited for, {bar.done} are over")

    def tiles(self):
        n = 0
        for u, (count, last, two) in enumerate(self.units):
            for j in range(count):
                yield u, j, n, (last if j == count - 1 else 8), count, two
                n += 1

    def rows_out(self, cta, u):
        yield from self.wait(self.rows_set[cta][u & 1], u >> 1)

    def keys(self, cta):
        for u, j, n, blocks, _, two in self.tiles():
            if j == 0:
                if u >= 2:
                    yield from self.rows_out(cta, u - 2)
                bar = self.q_ready[u & 1]
                if cta == 0:
                    bar.add(1, 2 if two else 1)
                if cta == 1 or two:
                    self.copies.append((bar, 1))
            yield  # (block ids are on their way)
            here = min(4, blocks) if cta == 0 else blocks - 4
            if n >= BUFS and (here > 0 or self.wait_without_keys):
                yield from self.wait(self.s_full[cta][n % BUFS], n // BUFS - 1)
            go = self.scores_go[n % BUFS]
            if cta == 0:
                go.add(1, blocks)
            self.copies += [(go, 1)] * max(here, 0)
            yield
        for u in range(max(0, len(self.units) - 2), len(self.units)):
            yield from self.rows_out(cta, u)

    def values(self, cta):
        for _, _, n, blocks, _, _ in self.tiles():
            if n >= BUFS:
                yield from self.wait(self.pv_done[cta][n % BUFS], n // BUFS - 1)
            go = self.pv_go[0][n % BUFS]
            if blocks == 8:
                go.add(1, 16 if cta == 0 else 0)
                self.copies += [(go, 1)] * 8
            else:
                yield  # (landed, zeroed beyond the newest token)
                go.add(1)
            yield

    def scores(self):
        for u, j, n, *_ in self.tiles():
            if j == 0:
                yield from self.wait(self.q_ready[u & 1], u >> 1)
            yield from self.wait(self.scores_go[n % BUFS], n // BUFS)
            self.pipe.append([self.s_full[0][n % BUFS], self.s_full[1][n % BUFS]])
            yield

    def weights_times_values(self):
        for u, j, n, *_ in self.tiles():
            if j == 0 and u > 0:
                yield from self.wait(self.o_free, u - 1)
            for half in range(2):
                yield from self.wait(self.pv_go[half][n % BUFS], n // BUFS)
            self.pipe.append([self.scores_go[n % BUFS], self.pv_done[0][n % BUFS], self.pv_done[1][n % BUFS]])
            yield

    def softmax(self, cta, g):
        shared = 0  # units so far in which both groups had tiles
        for u, j, n, _, count, _ in self.tiles():
            last = n + count - 1 - j
            if n % 2 == g:
                yield from self.wait(self.s_full[cta][n % BUFS], n // BUFS)
                while n > 0 and self.m[cta][1 - g] != n - 1:
                    if self.m[cta][1 - g] > n - 1:
                        raise Wrong("a maximum was overwritten")
                    yield
                self.m[cta][g] = n
                if j > 0 and self.rng.random() < 0.3:  # rescales O
                    yield from self.wait(self.pv_done[cta][(n - 1) % BUFS], (n - 1) // BUFS)
                for half in range(2):
                    self.pv_go[half][n % BUFS].add(4)
                    yield
            if j < count - 1:
                continue
            if last % 2 != g:
                if count > 1:
                    self.l_set[cta][shared & 1].add(4)
            else:
                if count > 1:
                    yield from self.wait(self.l_set[cta][shared & 1], shared >> 1)
                yield from self.wait(self.pv_done[cta][last % BUFS], last // BUFS)
                self.o_free.add(4)
                yield
                self.rows_set[cta][u & 1].add(4)
            shared += count > 1

    def products(self):
        while True:
            if self.pipe:
                for bar in self.pipe.pop(0):
                    bar.add(1)
            yield

    def landing(self):
        while True:
            if self.copies:
                bar, n = self.copies.pop(self.rng.randrange(len(self.copies)))
                bar.add(0, -n)
            yield

    def run(self):
        roles = [self.scores(), self.weights_times_values()]
        for cta in range(2):
            roles += [self.keys(cta), self.values(cta), self.softmax(cta, 0), self.softmax(cta, 1)]
        engines = [self.products(), self.landing()]
        pace = {id(r): self.rng.choice([1, 1, 0.2, 0.03]) for r in roles + engines}
        idle = 0
        while roles:
            role = self.rng.choice(roles + engines)
            if self.rng.random() > pace[id(role)]:
                continue
            before = self.progress()
            try:
                next(role)
            except StopIteration:
                roles.remove(role)
                idle = 0
            idle = 0 if self.progress() != before else idle + 1
            if idle > 20000:
                raise Wrong("nothing moves")

    def progress(self):
        return len(self.pipe), len(self.copies), sum(b.done * 64 - b.left for b in self.scores_go + self.pv_go[0] + self.pv_go[1]), self.o_free.left


def draw(rng):
    one_tile = rng.random() < 0.4
    return [(1 if one_tile else rng.choice([1, 1, 2, 3, 4, 7]), rng.choice([1, 3, 4, 5, 8]), rng.random() < 0.4)
            for _ in range(rng.randint(1, 9))]


@pytest.mark.parametrize("part", range(4))
def test_every_wait_ends_in_its_phase(part):
    for seed in range(part * 50, part * 50 + 50):
        rng = random.Random(seed)
        Pair(draw(rng), rng).run()


def test_a_wait_that_its_barrier_can_outrun_is_found():
    """CTA 1's wait for scores that need no keys of its own."""
    found = 0
    for seed in range(60):
        rng = random.Random(seed)
        try:
            Pair([(1, 1, False)] * 8, rng, wait_without_keys=True).run()
        except Wrong:
            found += 1
    assert found
