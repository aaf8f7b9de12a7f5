"""The hand-overs inside a pair of CTAs of attention_kernel (csrc/omni_attn.cu), run as a model on the CPU.

The loading warps, the MMA warp, the softmax warps, the tensor pipe and the copies in flight of a pair are generators that take their
steps in random order, with the kernel's barriers, counts and parities, the number of score buffers and stages read from its source.
Whatever the order: every step finds the data of its own item and block, no wait is for a parity that a later phase could
answer, no barrier gets a second arrival before it was met, and all warps come to their end -- also when any one wait
runs out.  Two of the four quadrants of 32 rows are run: a quadrant meets the others only in the counts of two barriers."""
import random
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "cleffa_b200" / "csrc" / "omni_attn.cu").read_text()
STAGES, BUFS = (int(v) for v in re.search(r"AT_KV_STAGES = (\d+), AT_BUFS = (\d+);", SOURCE).groups())
CTAS, QUADS = 2, 2


class Mbarrier:
    """Arrivals and bytes of the running phase; `done` phases are complete."""

    def __init__(self, count):
        self.count = self.pending = count
        self.bytes = self.done = 0

    def update(self, arrivals=0, nbytes=0):
        self.pending -= arrivals
        self.bytes += nbytes
        assert self.pending >= 0
        if self.pending == 0 and self.bytes == 0:
            self.done, self.pending = self.done + 1, self.count


class Pair:
    def __init__(self, items, rng, late=None):
        self.items, self.rng = items, rng                              # key blocks of each item that the pair takes
        self.late, self.waits, self.quit = late, 0, False              # the wait that runs out
        both = lambda n, count=1: [[Mbarrier(count) for _ in range(n)] for _ in range(CTAS)]
        self.q_full, self.k_full, self.v_full = ([Mbarrier(1) for _ in range(n)] for n in (2, STAGES, STAGES))
        self.q_empty, self.k_empty, self.v_empty = both(2), both(STAGES), both(STAGES)
        self.s_full, self.pv_done = both(BUFS), both(BUFS)
        self.p_full = [Mbarrier(QUADS * CTAS) for _ in range(BUFS)]
        self.o_empty = Mbarrier(QUADS * CTAS)
        self.fin_full = [[both(2, BUFS - 1)[0] for _ in range(QUADS)] for _ in range(CTAS)]
        self.fin_empty = [[both(2)[0] for _ in range(QUADS)] for _ in range(CTAS)]
        self.named = {}                                                # (cta, group, quadrant) -> has the group's warp arrived
        none = lambda *n: None if not n else [none(*n[1:]) for _ in range(n[0])]
        self.q, self.k, self.v = none(CTAS, 2), none(CTAS, STAGES), none(CTAS, STAGES)
        self.s, self.p, self.m = none(CTAS, BUFS), none(CTAS, BUFS, QUADS), none(CTAS, BUFS, QUADS)
        self.fin = none(CTAS, 2, BUFS, QUADS)
        self.o, self.o_busy, self.o_read = [None] * CTAS, False, [[-1] * QUADS for _ in range(CTAS)]
        self.pipe, self.copies, self.idle, self.written = [], [], False, set()

    def check(self, ok):
        assert ok or self.quit                                         # what is computed after a wait ran out is given up

    # a wait for the end of phase `k` of a barrier by its parity, as mbarrier.try_wait sees it; False: it ran out
    def wait(self, bar, parity, k):
        assert parity == k & 1
        self.waits += 1
        if self.waits == self.late:
            self.quit = True
            return False

        def over():
            self.check(bar.done in (k, k + 1))
            return (bar.done & 1) != parity
        yield lambda: over() or self.quit
        return (bar.done & 1) != parity

    def named_arrive(self, key):
        assert not self.named.get(key)
        self.named[key] = True

    def named_sync(self, key):
        yield lambda: self.named.get(key)
        self.named[key] = False

    def copy(self, place, i, what, bar, nbytes, use):
        def land():
            self.check(bar.done == use)
            place[i] = what
            bar.update(nbytes=-nbytes)
        self.copies.append(land)

    def load(self, cta):
        items, n = self.items, dict(k=0, v=0)
        at = dict(k=[0, 0], v=[0, 0])                                  # item, block

        def one(kind, place, full, empty):
            use, (item, block) = n[kind], at[kind]
            st, phase = use % STAGES, use // STAGES & 1
            if not (yield from self.wait(empty[cta][st], phase ^ 1, use // STAGES - 1)):
                return False
            if cta == 0:
                full[st].update(1, CTAS)
            self.check(place[cta][st] is None)
            self.copy(place[cta], st, (item, block), full[st], 1, use // STAGES)
            n[kind] += 1
            at[kind] = [item, block + 1] if block + 1 < items[item] else [item + 1, 0]
            return True

        def load_k():
            item, block = at["k"]
            if block == 0:
                b, ph = item & 1, item >> 1 & 1
                if not (yield from self.wait(self.q_empty[cta][b], ph ^ 1, (item >> 1) - 1)):
                    return False
                if cta == 0:
                    self.q_full[b].update(1, CTAS)
                self.copy(self.q[cta], b, item, self.q_full[b], 1, item >> 1)
            return (yield from one("k", self.k, self.k_full, self.k_empty))

        left = lambda kind: at[kind][0] < len(items)
        for _ in range(BUFS):
            if left("k") and not (yield from load_k()):
                return
        while left("v"):
            if not (yield from one("v", self.v, self.v_full, self.v_empty)):
                return
            if left("k") and not (yield from load_k()):
                return

    def mma(self):
        items = self.items
        seq = [(i, j) for i, n in enumerate(items) for j in range(n)]
        every = lambda bars, i: [bars[c][i] for c in range(CTAS)]      # a commit arrives in both CTAs

        def scores(n):
            item, j = seq[n]
            b, st, buf = item & 1, n % STAGES, n % BUFS
            if j == 0 and not (yield from self.wait(self.q_full[b], item >> 1 & 1, item >> 1)):
                return False
            if not (yield from self.wait(self.k_full[st], n // STAGES & 1, n // STAGES)):
                return False

            def run():
                for c in range(CTAS):
                    self.check(self.q[c][b] == item and self.k[c][st] == (item, j))
                    self.check(self.s[c][buf] is None)                 # the block before has been read, and its P multiplied
                    self.s[c][buf], self.k[c][st] = (item, j), None
            self.pipe.append((run, every(self.s_full, buf) + every(self.k_empty, st) + (every(self.q_empty, b) if j == items[item] - 1 else []), False))
            return True

        for n in range(min(BUFS, len(seq))):
            if not (yield from scores(n)):
                return
        for n, (item, j) in enumerate(seq):
            st, buf = n % STAGES, n % BUFS
            ok = yield from self.wait(self.v_full[st], n // STAGES & 1, n // STAGES)
            if ok and j == 0 and item > 0:
                ok = yield from self.wait(self.o_empty, item - 1 & 1, item - 1)
            if ok:
                ok = yield from self.wait(self.p_full[buf], n // BUFS & 1, n // BUFS)
            if not ok:
                return

            def run(item=item, j=j, st=st, buf=buf):
                for c in range(CTAS):
                    self.check(self.p[c][buf] == [(item, j)] * QUADS and self.v[c][st] == (item, j))
                    self.check(self.o_read[c] == [item - 1] * QUADS if j == 0 else self.o[c] == (item, j - 1))
                    self.o[c], self.v[c][st], self.s[c][buf] = (item, j), None, None
            self.pipe.append((run, every(self.v_empty, st) + every(self.pv_done, buf), True))
            if n + BUFS < len(seq) and not (yield from scores(n + BUFS)):
                return

    def tensor_pipe(self):
        while True:
            yield lambda: self.pipe or self.idle
            if not self.pipe:
                return
            run, commits, value = self.pipe[0]
            self.o_busy = value
            yield lambda: True
            run()
            self.o_busy = False
            self.pipe.pop(0)
            for bar in commits:
                bar.update(1)
                yield lambda: True

    def softmax(self, cta, grp, quad):
        items, rng = self.items, self.rng
        before = (grp + BUFS - 1) % BUFS
        alive, at, phase, uses, first_ever = True, 0, 0, 0, True
        for item, n_blocks in enumerate(items):
            last, slot, slot_phase = (at + n_blocks - 1) % BUFS, item & 1, item >> 1 & 1
            for j in range((grp + BUFS - at) % BUFS, n_blocks, BUFS):
                diagonal = j == n_blocks - 1
                alive = alive and (yield from self.wait(self.s_full[cta][grp], phase, uses))
                if alive:
                    self.check(self.s[cta][grp] == (item, j))
                if at + j > 0 or not first_ever:
                    yield from self.named_sync((cta, before, quad))
                    if j > 0:
                        self.check(self.m[cta][before][quad] == (item, j - 1))
                yield lambda: True
                self.m[cta][grp][quad] = (item, j)
                if not diagonal or item + 1 < len(items):
                    self.named_arrive((cta, grp, quad))
                if j > 0 and rng.random() < 0.5:                       # O is rescaled
                    alive = alive and (yield from self.wait(self.pv_done[cta][before], phase ^ 1 if grp == 0 else phase, uses - (grp == 0)))
                    if alive:
                        self.check(self.o[cta] == (item, j - 1) and not self.o_busy)
                        yield lambda: True
                        self.check(self.o[cta] == (item, j - 1) and not self.o_busy)
                if alive:
                    yield lambda: True
                    self.check(self.s[cta][grp] == (item, j))
                    self.p[cta][grp][quad] = (item, j)
                    yield lambda: True
                    self.p_full[grp].update(1)
                phase, uses = phase ^ 1, uses + 1
            first_ever = False
            if grp != last:
                alive = alive and (yield from self.wait(self.fin_empty[cta][quad][slot], slot_phase ^ 1, (item >> 1) - 1))
                self.fin[cta][slot][grp][quad] = item
                yield lambda: True
                self.fin_full[cta][quad][slot].update(1)
            else:
                alive = alive and (yield from self.wait(self.fin_full[cta][quad][slot], slot_phase, item >> 1))
                self.check(all(self.fin[cta][slot][g][quad] == item for g in range(BUFS) if g != grp))
                yield lambda: True
                self.fin_empty[cta][quad][slot].update(1)
                alive = alive and (yield from self.wait(self.pv_done[cta][grp], phase ^ 1, uses - 1))
                if alive:
                    for _ in range(2):
                        self.check(self.o[cta] == (item, n_blocks - 1) and not self.o_busy)
                        yield lambda: True
                    self.o_read[cta][quad] = item
                    self.o_empty.update(1)
                    self.written.add((item, cta, quad))
            at = (at + n_blocks) % BUFS

    def run(self):
        warps = [self.load(c) for c in range(CTAS)] + [self.mma()] + [self.softmax(c, g, q) for c in range(CTAS) for g in range(BUFS) for q in range(QUADS)]
        actors = {a: next(a, None) for a in warps + [self.tensor_pipe()]}
        actors = {a: ready for a, ready in actors.items() if ready}
        pace = {a: self.rng.choice((1, 1, 4, 30)) for a in actors}    # some are much slower than others
        while actors:
            self.idle = not any(a in actors for a in warps)
            ready = [a for a, can in actors.items() if can()]
            if self.copies and (not ready or self.rng.random() < 0.2):
                self.copies.pop(self.rng.randrange(len(self.copies)))()
                continue
            assert ready, "nobody can go on"
            a = self.rng.choices(ready, [1 / pace[a] for a in ready])[0]
            try:
                actors[a] = next(a)
            except StopIteration:
                del actors[a]
        assert not any(self.named.values())                            # no barrier is left half met
        return self


def item_list(rng):
    return [rng.choice((1, 1, 2, 3, 4, 5, 7)) for _ in range(rng.randint(1, 6))]


@pytest.mark.parametrize("seed", range(6))
def test_every_hand_over_finds_its_own_block(seed):
    rng = random.Random(seed)
    for _ in range(40):
        items = item_list(rng)
        pair = Pair(items, rng).run()
        assert pair.written == {(i, c, q) for i in range(len(items)) for c in range(CTAS) for q in range(QUADS)}


@pytest.mark.parametrize("seed", range(6))
def test_no_warp_is_left_behind_when_a_wait_runs_out(seed):
    rng = random.Random(100 + seed)
    for _ in range(40):
        items = item_list(rng)
        total = Pair(items, rng).run().waits
        pair = Pair(items, rng, late=rng.randint(1, total)).run()      # that all of them end is what is seen here
        assert pair.quit or pair.waits < pair.late                     # rescaling is drawn: a run may have fewer waits


@pytest.mark.parametrize("pairs", [1, 3, 74])
def test_items_are_dealt_once(pairs):
    """AttnItems: rounds over the pairs in alternating direction; a pair stops at the first index behind the list."""
    for n in (1, 2, pairs - 1, pairs, pairs + 1, 3 * pairs + 2):
        dealt = []
        for p in range(pairs):
            r = 0
            while (i := r * pairs + (pairs - 1 - p if r & 1 else p)) < n:
                dealt.append(i)
                r += 1
        assert sorted(dealt) == list(range(n))
