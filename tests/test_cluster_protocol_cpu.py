"""The cluster engine's exchange (csrc/cluster.cu) as a model under random
schedules: CTAs whose warps publish words to one another, counted on two barriers
by step parity, with waits that may give up at any poll.  Checked: no arrival
beyond a phase's count, no word that lands after its CTA has left, and no wait
that never ends -- in both time loops (several items a warp behind a CTA-wide
wait; an item a warp, each warp waiting and arriving by itself)."""
import random

import pytest


class Barrier:
    def __init__(self, count):
        self.count = self.pending = count
        self.tx = self.phase = 0

    def check(self):
        if self.pending == 0 and self.tx == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def arrive(self, n=1):
        assert self.pending >= n, "arrival beyond the count"
        self.pending -= n
        self.check()

    def arm(self, words):
        self.tx += words
        self.arrive()

    def complete(self, words=1):
        self.tx -= words
        self.check()


def run(seed, one, p_give_up, drain):
    r = random.Random(seed)
    ctas, warps, steps = r.randint(1, 4), r.randint(1, 3), r.randint(1, 9)
    per = 1 if one else r.randint(1, 2)  # items of a warp
    items = warps * per
    expect = (ctas - 1) * items
    bars = [[Barrier(1 + items if one else 1) for _ in range(2)] for _ in range(ctas)]
    dead, left, armed = [False] * ctas, [False] * ctas, [min(2, steps)] * ctas
    sent, arrived = [[0, 0] for _ in range(ctas)], [[0, 0] for _ in range(ctas)]
    under_way, met, cta_met = [], [0, 0], [[0] * (steps + 1) for _ in range(ctas)]
    for b in bars:
        for p in range(min(2, steps)):
            b[p].arm(expect)

    def give_up(c):
        dead[c] = True
        yield
        for q in r.sample(range(ctas), ctas):
            dead[q] = True
            yield

    def cluster_sync(i):
        met[i] += 1
        while met[i] < ctas * warps:
            yield

    def warp(c, w):
        own, mine = [[0, 0] for _ in range(ctas)], [0, 0]
        if w == 0 and r.random() < p_give_up:
            yield from give_up(c)  # the wait for the in-edges
        for k in range(steps + 1):
            if k > 0:
                bar, phase = bars[c][(k - 1) & 1], (k - 1) >> 1
                if one or w == 0:
                    while bar.phase <= phase and not dead[c]:
                        if r.random() < p_give_up:
                            yield from give_up(c)
                            break
                        yield
                    if w == 0 and not dead[c] and k + 1 < steps:
                        bar.arm(expect)
                        armed[c] = k + 2
                yield
                if not one:
                    cta_met[c][k] += 1
                    while cta_met[c][k] < warps:
                        yield
            if k == steps:
                break
            for _ in range(per):
                for q in r.sample(range(ctas), ctas):
                    gone = dead[c]
                    if r.random() < 0.3:
                        yield
                    if gone:
                        continue
                    if q != c:
                        under_way.append((q, k & 1))
                        own[q][k & 1] += 1
                    elif one:
                        bars[c][k & 1].arrive()
                        mine[k & 1] += 1
                    if r.random() < 0.3:
                        yield
        yield from cluster_sync(0)
        if drain and dead[c]:
            for p in (0, 1):
                arrived[c][p] += mine[p]
                for q in range(ctas):
                    sent[q][p] += own[q][p]
            yield from cluster_sync(1)
            if w == 0:
                for p in (0, 1):
                    phases = (armed[c] + 1 - p) // 2
                    if not phases:
                        continue
                    never = phases * expect - sent[c][p]
                    late = phases * items - arrived[c][p] if one else 0
                    assert never >= 0 and late >= 0
                    if never:
                        bars[c][p].complete(never)
                        yield
                    if late:
                        bars[c][p].arrive(late)
                        yield
                    while bars[c][p].phase < phases:
                        yield
                    assert bars[c][p].phase == phases
        if w == 0:
            left[c] = True
            assert all(q != c for q, _ in under_way), "a word under way to a CTA that has left"

    tasks = [warp(c, w) for c in range(ctas) for w in range(warps)]
    for _ in range(200000):
        if not (tasks or under_way):
            return dead[0]
        if under_way and r.random() < r.choice((0.02, 0.5)):
            q, p = under_way.pop(r.randrange(len(under_way)))
            assert not left[q], "a word landed after its CTA had left"
            bars[q][p].complete()
        elif tasks:
            t = r.choice(tasks)
            try:
                next(t)
            except StopIteration:
                tasks.remove(t)
    raise AssertionError("a wait that never ends")


@pytest.mark.parametrize("one", [False, True])
def test_every_schedule_ends_with_no_word_under_way(one):
    gave_up = sum(run(seed, one, (0.0, 0.002, 0.02, 0.2)[seed % 4], True) for seed in range(1200))
    assert gave_up > 200


@pytest.mark.parametrize("one", [False, True])
def test_the_model_sees_words_under_way_without_the_drain(one):
    seen = 0
    for seed in range(4000):
        try:
            run(seed, one, (0.0, 0.002, 0.02, 0.2)[seed % 4], False)
        except AssertionError as e:
            assert "has left" in str(e) or "had left" in str(e)
            seen += 1
    assert seen > 0
