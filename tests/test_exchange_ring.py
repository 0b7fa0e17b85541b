"""A host model of the halo sweeps' exchange buffers under random schedules (no GPU).

A patch writes its words of sweep G (the sweep's number in each) into buffer G mod K from the start of
the sweep on (the rows that read no halo slot run first), while its fetch warps wait for the neighbours'
words of sweep G - 1 and for every patch's arrival at sweep G - 1 (the decision, one sweep late); then
it arrives at G, and the next sweep may start. The first sweep after a barrier of all patches (a linear
solve's first, or one after a refold) fetches no words and decides nothing. With three buffers no word
is overwritten before its readers have it; with two it happens."""
import random

import pytest


def simulate(buffers, seed, patches=9, sweeps=60):
    """True when every reader found its neighbours' words, False when one had been overwritten."""
    rng = random.Random(seed)
    near = [sorted(rng.sample([q for q in range(patches) if q != p], rng.randint(1, 3))) for p in range(patches)]
    near = [sorted(set(near[p]) | {q for q in range(patches) if p in near[q]}) for p in range(patches)]
    word = [[-1] * patches for _ in range(buffers)]
    arrived = [0] * sweeps
    # barriers follow these sweeps: linear solves and refolds of random length
    synced = {g for g in range(sweeps) if rng.random() < 0.1}
    weight = [rng.choice([1, 1, 5, 40]) for _ in range(patches)]   # some patches are much slower

    def run(p):
        for g in range(sweeps):
            todo = ["write"]
            if g > 0 and g - 1 not in synced:
                todo += ["decide"] + [("read", q) for q in near[p]]
            rng.shuffle(todo)   # the warps' order is free
            for what in todo:
                if what == "write":
                    word[g % buffers][p] = g
                elif what == "decide":
                    while arrived[g - 1] < patches:
                        yield
                else:
                    q = what[1]
                    while word[(g - 1) % buffers][q] < g - 1:
                        yield
                    if word[(g - 1) % buffers][q] != g - 1:
                        raise OverflowError
                yield
            arrived[g] += 1
            while g in synced and arrived[g] < patches:
                yield

    live = {p: run(p) for p in range(patches)}
    steps = 0
    try:
        while live:
            p = rng.choices(list(live), [1.0 / weight[q] for q in live])[0]
            for _ in range(rng.randint(1, 12)):
                steps += 1
                assert steps < 2_000_000, "stuck"
                try:
                    next(live[p])
                except StopIteration:
                    del live[p]
                    break
    except OverflowError:
        return False
    return True


@pytest.mark.parametrize("seed", range(60))
def test_three_buffers_keep_every_word_until_it_is_read(seed):
    assert simulate(3, seed)


def test_two_buffers_do_not():
    assert not all(simulate(2, seed) for seed in range(60))
