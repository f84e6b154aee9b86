"""Models of the small-batch kernel's protocols (csrc/linear_sb.cu), run under random interleavings on the CPU.

Inside a CTA a warpgroup works on its own: an issuer (ring of weight stages, MMAs and their commits) and four compute warps (words
of unit i + 1 into tensor memory and of unit i + 2 out of shared memory beside the MMAs of unit i; its sums read before the
MMAs of unit i + 1 are released through a named barrier).  mbarriers are waited on by PARITY, as on the device, so a waiter that
fell two phases behind would be caught as aliasing.  Between CTAs (`group`) the K chunks' sums meet when a group's CTAs are through, by a
word in which each counts itself and, where the sums are few, in slots whose value is its own mark; a CTA that runs out of patience
leaves its share to the last one, so that none depends on another's running at the same time.  The tests check: no deadlock, no
aliasing, no stage, operand or sum that is overwritten before all of its readers are done, every sum added exactly once and after all
chunks' stores, slots and word empty after a launch, whatever the number of CTAs that run at a time; and that the same
checks do flag protocols with a step out of place.
"""
import random

import pytest

CW = 4                                             # compute warps of a warpgroup


class MBar:
    def __init__(self):
        self.ph = 0

    def done(self, k):                             # the hardware's test for "phase k complete" through its parity
        return (self.ph & 1) != (k & 1), self.ph - k >= 2


def warpgroup(n, ST, abuf, seed, mistake=None):
    """One warpgroup over n units with ST stages and `abuf` A buffers; returns what went wrong."""
    rnd = random.Random(seed)
    a_full, mma_bar = [MBar() for _ in range(ST)], MBar()
    bar = [0] * (n + 1)                            # arrivals of the compute warps for the MMAs of unit i
    stage = [None] * ST                            # unit whose words a stage holds (None: in flight)
    stage_unit, stage_read = [None] * ST, [set() for _ in range(ST)]
    A = [[None] * CW for _ in range(abuf)]         # unit each warp's quarter of an A buffer holds
    D, d_read = None, set()
    copies, mmas, errors = [], [], []

    def issuer():
        issued = 0

        def load():
            nonlocal issued
            s = issued % ST
            if stage_unit[s] is not None and len(stage_read[s]) < CW:
                errors.append(("stage refilled early", issued))
            stage[s], stage_unit[s], stage_read[s] = None, issued, set()
            copies.append((s, issued))
            issued += 1
        for _ in range(min(n, ST)):
            load()
            yield
        for i in range(n):
            if mistake == "early refill" and issued < n:
                load()
            while bar[i] < CW:
                yield
            mmas.append(i)                         # executed in order, completed later
            yield
            if issued < n:
                load()
                yield

    def compute(c):
        def fetch(i):
            s = i % ST
            while True:
                ok, alias = a_full[s].done(i // ST)
                if alias:
                    errors.append(("alias a_full", c, i))
                if ok:
                    break
                yield
            if stage[s] != i:
                errors.append(("wrong words", c, i, stage[s]))
            stage_read[s].add(c)

        def step(i):                               # unit i + 1 into A, unit i + 2 out of shared memory
            if i + 1 < n:
                A[(i + 1) % abuf][c] = i + 1
                yield
                if i + 2 < n:
                    yield from fetch(i + 2)
        yield from fetch(0)
        A[0][c] = 0
        if n > 1:
            yield from fetch(1)
        bar[0] += 1
        for i in range(n):
            yield
            if abuf == 2 or mistake == "early expansion":
                yield from step(i)
            if mistake == "early arrival" and i + 1 < n:
                bar[i + 1] += 1
            while True:
                ok, alias = mma_bar.done(i)
                if alias:
                    errors.append(("alias mma_bar", c, i))
                if ok:
                    break
                yield
            if abuf == 1 and mistake != "early expansion":
                yield from step(i)
            if D != i:
                errors.append(("wrong sums", c, i, D))
            d_read.add(c)
            yield
            if mistake != "early arrival" and i + 1 < n:
                bar[i + 1] += 1

    agents = [issuer()] + [compute(c) for c in range(CW)]
    alive, idle = list(range(len(agents))), 0
    while alive:
        if copies and rnd.random() < 0.4:
            s, i = copies.pop(rnd.randrange(len(copies)))
            stage[s] = i
            a_full[s].ph += 1
            idle = 0
        if mmas and rnd.random() < 0.4:
            i = mmas.pop(0)
            if A[i % abuf] != [i] * CW:
                errors.append(("operand overwritten", i, list(A[i % abuf])))
            if D is not None and len(d_read) < CW:
                errors.append(("sums overwritten", i))
            D, d_read = i, set()
            mma_bar.ph += 1
            idle = 0
        a = rnd.choice(alive)
        before = (sum(bar), len(copies), len(mmas))
        try:
            next(agents[a])
        except StopIteration:
            alive.remove(a)
            idle = 0
        idle = 0 if before != (sum(bar), len(copies), len(mmas)) else idle + 1
        if idle > 5000 and not copies and not mmas:
            errors.append(("deadlock", alive))
        if errors:
            break
    return errors


@pytest.mark.parametrize("abuf", [1, 2])
def test_warpgroup_has_no_deadlock_aliasing_or_early_reuse(abuf):
    for trial in range(150):
        rnd = random.Random(trial)
        n, ST = rnd.randint(1, 14), rnd.randint(2, 4)
        assert warpgroup(n, ST, abuf, trial) == [], (n, ST, trial)


@pytest.mark.parametrize("abuf,mistake", [(2, "early refill"), (2, "early arrival"), (1, "early arrival"), (1, "early expansion")])
def test_model_flags_a_step_out_of_place(abuf, mistake):
    assert any(warpgroup(12, 2, abuf, trial, mistake) for trial in range(40))


def group(KC, launches, tagged, seed, resident=None, late=0.0, mistake=None):
    """KC CTAs of a group, launch after launch: a CTA stores its sums, counts itself in the group's word, and adds its share of every chunk's
    sums -- or, out of patience (with probability `late` per look), leaves what is not there yet to the last CTA.  At most `resident`
    of them run at a time; the next one starts when one has ended."""
    rnd = random.Random(seed)
    E = 2                                          # elements of a share
    slots = [[[None] * KC for _ in range(E)] for _ in range(KC)]          # [share][element][chunk]: launch whose sum it holds
    added = []                                     # (launch, share, element)
    errors = []
    word = {"count": 0, "mask": 0}

    def element(share, e, launch):                 # all sums have been seen: cleared one after the other
        if slots[share][e] != [launch] * KC:
            errors.append(("added before all chunks are stored", share, e))
        added.append((launch, share, e))
        if tagged:
            for c in range(KC):
                slots[share][e][c] = None
                yield

    def share_of(share, launch, all_here):
        done = True
        for e in range(E):
            while tagged and None in slots[share][e]:
                if all_here or not done or rnd.random() < late:
                    break
                yield
            if tagged and None in slots[share][e]:
                done = False
                if all_here and mistake == "adds again":
                    added.append((launch, share, e))
                continue
            yield from element(share, e, launch)
        return done

    def cta(chunk, launch):
        for share in rnd.sample(range(KC), KC):
            for e in range(E):
                yield
                if tagged and slots[share][e][chunk] is not None:
                    errors.append("slot still full")
                if mistake != "count first":
                    slots[share][e][chunk] = launch
        before = dict(word)                        # (one atomic addition; the count is zero again with the last of them)
        word["count"] = (word["count"] + 1) % KC
        yield
        if mistake == "count first":
            for share in range(KC):
                for e in range(E):
                    yield
                    slots[share][e][chunk] = launch
        done = False
        if tagged:
            done = yield from share_of(chunk, launch, False)
        mine, shares = set() if done else {chunk}, set()
        if before["count"] == KC - 1:
            shares = mine | {c for c in range(KC) if before["mask"] >> c & 1}
            if mistake != "no reset":
                word["mask"] = 0
        elif not done:
            while not tagged and word["count"] and rnd.random() >= late:
                yield
            yield
            if word["count"] == 0 and mistake != "always leaves":          # (a compare-and-swap that finds zero: all are there)
                shares = mine
            else:
                word["mask"] |= 1 << chunk
        for share in sorted(shares):
            yield from share_of(share, launch, True)

    for launch in range(launches):                 # (a launch begins when the one before has ended)
        waiting = [cta(c, launch) for c in rnd.sample(range(KC), KC)]
        agents, steps = [], 0
        while (agents or waiting) and not errors:
            while waiting and len(agents) < (resident or KC):
                agents.append(waiting.pop())
            steps += 1
            if steps > 100000:
                return errors + ["deadlock"]
            a = rnd.choice(agents)
            try:
                next(a)
            except StopIteration:
                agents.remove(a)
        if not errors and sorted(x[1:] for x in added if x[0] == launch) != [(s, e) for s in range(KC) for e in range(E)]:
            errors.append("an element is not added exactly once")
        if not errors and (word["count"] or word["mask"]):
            errors.append("the word is not zero after a launch")
        if not errors and tagged and any(v is not None for sh in slots for el in sh for v in el):
            errors.append("a slot is full after a launch")
    return errors


@pytest.mark.parametrize("tagged", [False, True])
@pytest.mark.parametrize("late", [0.0, 0.02, 0.3, 1.0])
def test_chunks_of_a_group_meet(tagged, late):
    for trial in range(150):
        rnd = random.Random(trial)
        KC = rnd.randint(2, 8)
        assert group(KC, rnd.randint(1, 3), tagged, trial, resident=rnd.randint(1, KC) if late else KC, late=late) == []


@pytest.mark.parametrize("tagged", [False, True])
def test_without_patience_a_group_that_does_not_fit_hangs(tagged):
    assert group(4, 1, tagged, 1, resident=3, late=0.0) == ["deadlock"]


@pytest.mark.parametrize("tagged,mistake", [(False, "count first"), (True, "count first"), (True, "adds again"), (False, "no reset"), (True, "no reset"),
                                            (False, "always leaves"), (True, "always leaves")])
def test_group_model_flags_a_step_out_of_place(tagged, mistake):
    assert any(group(4, 2, tagged, trial, late=late, mistake=mistake) for trial in range(300) for late in (0.3, 1.0))
