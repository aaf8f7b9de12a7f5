"""The hand-overs inside a pair of CTAs, or one CTA, of expert_pair_kernel (csrc/omni_expert.cu), run as a model on the CPU.

The scheduler, the producers of weights and of tokens (by TMA, or by gathering threads that hand a stage over some stages after they filled it), the
MMA warp, the epilogue warps, the tensor pipe and the copies in flight are generators that take their steps in random order, with
the kernel's barriers and counts; ring depths and lags are read from its source.  A stage's weights and tokens, of both CTAs, share one full and one empty
barrier.  Whatever the order: every MMA finds the slabs of its own item in both CTAs, nothing is staged over what is still to be read, no wait is for
a parity that a later phase could answer, and all warps come to their end -- also when any one wait runs out."""
import random
import re
from pathlib import Path

import pytest

from test_attention_schedule_cpu import Mbarrier, Pair

SOURCE = (Path(__file__).resolve().parents[1] / "cleffa_b200" / "csrc" / "omni_expert.cu").read_text()
RING_DEPTHS = tuple(int(v) for v in re.search(r"int STAGES = MODE == X_OPROJ \? (\d) : (\d);", SOURCE).groups())
LAGS = tuple(int(v) for v in re.search(r"int LAG = CTAS == 2 \? (\d) : (\d);", SOURCE).groups())        # pairs, single CTAs
ITEM_RING = int(re.search(r"X_RING = (\d+);", SOURCE).group(1))
GATHER, EPILOGUE = 2, 2                       # gathering warps and epilogue warps of a CTA that the model runs
assert "mbar_init(full_bar(s), 1 + tok_arrivals); mbar_init(empty_bar(s), 1);" in SOURCE


class Expert(Pair):
    """The waits, checks and copies are those of the attention's model."""

    def __init__(self, n_items, slabs, rng, ctas=2, stages=6, gathering=True, late=None):
        self.n_items, self.slabs, self.rng, self.ctas, self.stages, self.gathering = n_items, slabs, rng, ctas, stages, gathering
        self.late, self.waits, self.quit = late, 0, False
        both = lambda n, count=1: [[Mbarrier(count) for _ in range(n)] for _ in range(ctas)]
        self.full = [Mbarrier(1 + (GATHER * ctas if gathering else 1)) for _ in range(stages)]
        self.empty, self.acc_full = both(stages), both(2)
        self.acc_empty = [Mbarrier(EPILOGUE * ctas) for _ in range(2)]
        self.item_full = both(ITEM_RING)
        self.item_empty = [Mbarrier(1 + ctas * (1 + (GATHER if gathering else 1) + EPILOGUE)) for _ in range(ITEM_RING)]
        self.ring = [[None] * ITEM_RING for _ in range(ctas)]
        self.weights = [[None] * stages for _ in range(ctas)]
        self.tokens = [[[None] * stages for _ in range(GATHER if gathering else 1)] for _ in range(ctas)]
        self.acc, self.read = [[None, None] for _ in range(ctas)], [[[-1, -1] for _ in range(EPILOGUE)] for _ in range(ctas)]
        self.pipe, self.copies, self.idle, self.written = [], [], False, set()

    def scheduler(self):
        for it in range(self.n_items + 1):
            slot, use = it % ITEM_RING, it // ITEM_RING
            if not (yield from self.wait(self.item_empty[slot], use & 1 ^ 1, use - 1)):
                return
            for c in range(self.ctas):
                yield lambda: True
                self.ring[c][slot] = it if it < self.n_items else "stop"
                self.item_full[c][slot].update(1)

    def take(self, cta, it):
        """A warp of this CTA takes item `it` out of the ring; whether there is one."""
        slot, use = it % ITEM_RING, it // ITEM_RING
        if not (yield from self.wait(self.item_full[cta][slot], use & 1, use)):
            return False
        got = self.ring[cta][slot]
        self.check(got == (it if it < self.n_items else "stop"))
        yield lambda: True
        self.item_empty[slot].update(1)
        return got != "stop"

    def stage_of(self, it, ks):
        n = it * self.slabs + ks
        return n % self.stages, n // self.stages

    def fill(self, cta, place, it, ks, announce):
        st, use = self.stage_of(it, ks)
        if not (yield from self.wait(self.empty[cta][st], use & 1 ^ 1, use - 1)):
            return False
        if announce and cta == 0:
            self.full[st].update(1, self.ctas)                         # arrives and expects the bytes of both CTAs
        self.check(place[st] is None)
        if announce:
            self.copy(place, st, (it, ks), self.full[st], 1, use)
        else:
            place[st] = (it, ks)                                       # landed at the latest when it is handed over
        return True

    def producer(self, cta, place):
        it = 0
        while (yield from self.take(cta, it)):
            for ks in range(self.slabs):
                if not (yield from self.fill(cta, place, it, ks, True)):
                    return
            it += 1

    def gather(self, cta, warp):
        lag, pending, it = LAGS[0 if self.ctas == 2 else 1], [], 0

        def hand_over():
            self.full[pending.pop(0)].update(1)

        more = yield from self.take(cta, it)
        while more:
            for ks in range(self.slabs):
                if ks >= lag:
                    hand_over()
                if not (yield from self.fill(cta, self.tokens[cta][warp], it, ks, False)):
                    return
                pending.append(self.stage_of(it, ks)[0])
            it += 1
            more = yield from self.take(cta, it)
            while pending:
                hand_over()
                yield lambda: True

    def mma_warp(self):
        every = lambda bars, i: [bars[c][i] for c in range(self.ctas)]      # a commit arrives in both CTAs
        it = 0
        while (yield from self.take(0, it)):
            buf, use = it & 1, it >> 1
            if not (yield from self.wait(self.acc_empty[buf], use & 1 ^ 1, use - 1)):
                return
            for ks in range(self.slabs):
                st, n = self.stage_of(it, ks)
                if not (yield from self.wait(self.full[st], n & 1, n)):
                    return

                def run(it=it, ks=ks, st=st, buf=buf):
                    for c in range(self.ctas):
                        self.check(self.weights[c][st] == (it, ks) and all(t[st] == (it, ks) for t in self.tokens[c]))
                        if ks == 0:
                            self.check(all(r[buf] == max(it - 2, -1) for r in self.read[c]))
                        else:
                            self.check(self.acc[c][buf] == (it, ks - 1))
                        self.weights[c][st], self.acc[c][buf] = None, (it, ks)
                        for t in self.tokens[c]:
                            t[st] = None
                self.pipe.append((run, every(self.empty, st) + (every(self.acc_full, buf) if ks == self.slabs - 1 else []), False))
            it += 1

    def epilogue(self, cta, warp):
        it = 0
        while (yield from self.take(cta, it)):
            buf, use = it & 1, it >> 1
            if not (yield from self.wait(self.acc_full[cta][buf], use & 1, use)):
                return
            for _ in range(2):
                self.check(self.acc[cta][buf] == (it, self.slabs - 1))
                yield lambda: True
            self.read[cta][warp][buf] = it
            self.acc_empty[buf].update(1)
            self.written.add((it, cta, warp))
            it += 1

    def run(self):
        warps = [self.scheduler(), self.mma_warp()]
        for c in range(self.ctas):
            warps.append(self.producer(c, self.weights[c]))
            warps += [self.gather(c, w) for w in range(GATHER)] if self.gathering else [self.producer(c, self.tokens[c][0])]
            warps += [self.epilogue(c, w) for w in range(EPILOGUE)]
        actors = {a: next(a, None) for a in warps + [self.tensor_pipe()]}
        actors = {a: ready for a, ready in actors.items() if ready}
        pace = {a: self.rng.choice((1, 1, 4, 30)) for a in actors}          # some are much slower than others
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
        return self


def shapes(rng):
    return dict(n_items=rng.randint(0, 7), slabs=rng.choice((1, 3, 4, 9)), ctas=rng.choice((1, 2)), stages=rng.choice(RING_DEPTHS), gathering=rng.random() < 0.5)


@pytest.mark.parametrize("seed", range(6))
def test_every_product_finds_its_own_slabs(seed):
    rng = random.Random(seed)
    for _ in range(40):
        s = shapes(rng)
        e = Expert(rng=rng, **s).run()
        assert e.written == {(i, c, w) for i in range(s["n_items"]) for c in range(s["ctas"]) for w in range(EPILOGUE)}


@pytest.mark.parametrize("seed", range(6))
def test_no_warp_is_left_behind_when_a_wait_runs_out(seed):
    rng = random.Random(100 + seed)
    for _ in range(40):
        s = shapes(rng)
        total = Expert(rng=rng, **s).run().waits
        assert Expert(rng=rng, late=rng.randint(1, total), **s).run().quit     # that all of them end is what is seen here
