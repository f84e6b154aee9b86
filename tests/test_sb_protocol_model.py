"""Models of the small-batch kernel's protocols (csrc/linear_sb.cu), run under random interleavings on the CPU.

Inside a CTA a warpgroup works on its own: an issuer (ring of weight stages, MMAs and their commits) and four compute warps (words
of unit i + 1 into tensor memory and of unit i + 2 out of shared memory beside the MMAs of unit i; its sums read before the
MMAs of unit i + 1 are released through a named barrier).  mbarriers are waited on by PARITY, as on the device, so a waiter that
fell two phases behind would be caught as aliasing.  Between CTAs the K chunks' sums meet when a group's CTAs are through: at a counter
that wraps to zero, or in slots whose value is its own mark (`group`; `chunks` is the protocol before that: stored, counted a
unit later and looked at another unit later).  The tests check: no deadlock, no aliasing, no stage, operand or sum that is overwritten
before all of its readers are done, exactly one warp that adds a quarter and all chunks' stores before it; and that the same
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


def chunks(KC, tiles, seed, mistake=None):
    """KC CTAs, a warp each, over `tiles` whole tiles of one quarter: stored, counted a step later, looked at another step later."""
    rnd = random.Random(seed)
    stored = [set() for _ in range(tiles)]
    counter, added, errors = [0] * tiles, [0] * tiles, []

    def warp(chunk):
        pend, tile, old = 0, None, 0

        def settle():
            nonlocal pend, old
            if pend == 1:
                old = counter[tile]
                counter[tile] += 1
                pend = 2
            elif pend == 2:
                pend = 0
                if old == KC - 1:
                    if len(stored[tile]) < KC:
                        errors.append(("added before all chunks are stored", tile))
                    counter[tile] = 0
                    added[tile] += 1
        for t in range(tiles):
            for _ in range(rnd.choice([1, 1, 2, 4])):              # units of the tile
                yield
                if pend:
                    settle()
            while pend:
                settle()
                yield
            if mistake == "count first":
                pend, tile = 1, t
                settle()
                yield
                stored[t].add(chunk)
            else:
                stored[t].add(chunk)
                pend, tile = 1, t
        while pend:
            yield
            settle()

    agents = [warp(c) for c in range(KC)]
    while agents:
        a = rnd.choice(agents)
        try:
            next(a)
        except StopIteration:
            agents.remove(a)
    if not errors and (added != [1] * tiles or counter != [0] * tiles):
        errors.append(("adders, counters", added, counter))
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


def test_chunks_are_added_once_and_after_all_stores():
    for trial in range(300):
        rnd = random.Random(trial)
        assert chunks(rnd.randint(2, 16), rnd.randint(1, 6), trial) == []


def test_model_flags_a_count_in_front_of_the_store():
    assert any(chunks(4, 3, trial, "count first") for trial in range(40))


def group(KC, launches, tagged, seed, mistake=None):
    """KC CTAs of a group, launch after launch: sums stored, then all of them waited for and each CTA's share read (and cleared)."""
    rnd = random.Random(seed)
    slots = [[None] * KC for _ in range(KC)]       # [share][chunk]: launch whose sum it holds, None: empty
    counter, errors = 0, []

    def cta(chunk, launch):
        nonlocal counter
        if mistake == "count first":
            counter = (counter + 1) % KC
        for share in rnd.sample(range(KC), KC):
            yield
            if tagged and slots[share][chunk] is not None:
                errors.append("slot still full")
            slots[share][chunk] = launch
        if not tagged:
            yield
            if mistake != "count first":
                counter = (counter + 1) % KC
            while counter:
                yield
        else:
            while mistake != "no wait" and None in slots[chunk]:
                yield
        if slots[chunk] != [launch] * KC:
            errors.append("share read before all chunks are stored")
        if tagged:
            for c in range(KC):
                yield
                slots[chunk][c] = None
        yield

    for launch in range(launches):                 # (a launch begins when the one before has ended)
        agents = [cta(c, launch) for c in range(KC)]
        steps = 0
        while agents and not errors:
            steps += 1
            if steps > 100000:
                return errors + ["deadlock"]
            a = rnd.choice(agents)
            try:
                next(a)
            except StopIteration:
                agents.remove(a)
        if counter:
            errors.append("counter is not zero after a launch")
    return errors


@pytest.mark.parametrize("tagged", [False, True])
def test_chunks_of_a_group_meet(tagged):
    for trial in range(200):
        rnd = random.Random(trial)
        assert group(rnd.randint(2, 8), rnd.randint(1, 3), tagged, trial) == []


@pytest.mark.parametrize("tagged,mistake", [(False, "count first"), (True, "no wait")])
def test_group_model_flags_a_step_out_of_place(tagged, mistake):
    assert any(group(4, 2, tagged, trial, mistake) for trial in range(40))
