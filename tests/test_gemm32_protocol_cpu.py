"""The barriers of the roles of gemm32_long.cu and gemm32_long_outer.cu as coroutines under random schedules: nothing waits for good, and every
stage is converted, multiplied and drained once and in order."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "memorax_b200", "csrc")
SOURCE = {name: open(os.path.join(CSRC, name + ".cu")).read() for name in ("gemm32_long", "gemm32_long_outer")}
FIRST_RUN, LOW_RUN = (int(re.search(r"constexpr int %s = (\d+);" % name, SOURCE["gemm32_long"]).group(1)) for name in ("kFirstRun", "kLowRun"))


class Barrier:
    def __init__(self):
        self.phase = 0

    def arrive(self):
        self.phase += 1

    def done(self, parity):
        return (self.phase & 1) != parity


def bars(n):
    return [Barrier() for _ in range(n)]


def play(rng, actors, barriers):
    """Runs the coroutines in random order until all have ended."""
    idle, before = 0, None
    while actors:
        actor = rng.choice(actors)
        for _ in range(rng.randrange(1, 8)):
            if next(actor, "end") == "end":
                actors.remove(actor)
                break
        now = [b.phase for b in barriers]
        idle, before = idle + 1 if now == before else 0, now
        assert idle < 5000, "everyone waits"


# The copies of float32 tiles and the producers, which are the same in both kernels.
def fill(total, per_tile, raws, stages, raw_full, raw_empty, full, empty, planes):
    raw = [None] * raws

    def copies():
        for turn in range(total):
            while not raw_empty[turn % raws].done(1 ^ (turn // raws & 1)):
                yield
            raw[turn % raws] = divmod(turn, per_tile)
            yield
            raw_full[turn % raws].arrive()

    def producers():
        for turn in range(total):
            while not raw_full[turn % raws].done(turn // raws & 1):
                yield
            got = raw[turn % raws]
            yield
            raw_empty[turn % raws].arrive()
            while not empty[turn % stages].done(1 ^ (turn // stages & 1)):
                yield
            planes[turn % stages] = got
            yield
            full[turn % stages].arrive()

    return [copies(), producers()]


@pytest.mark.parametrize("sets,raws", [(1, 1), (2, 2)])
@pytest.mark.parametrize("run_length", [1, 2])
def test_products_with_a_weight(sets, raws, run_length, stages=2):
    for seed in range(300):
        rng = random.Random(seed)
        tiles, per_tile = rng.randrange(1, 6), rng.randrange(1, 7 if run_length == 1 else 40)
        total = tiles * per_tile
        groups = [bars(n) for n in (raws, raws, stages, stages, sets, sets, sets, sets)]
        raw_full, raw_empty, full, empty, main_full, main_empty, low_full, low_empty = groups
        planes, main, low, drained = [None] * stages, [[] for _ in range(sets)], [[] for _ in range(sets)], []

        def tensor_core():
            turn = main_turn = low_turn = 0
            for t in range(tiles):
                run = 0
                for s in range(per_tile):
                    while not full[turn % stages].done(turn // stages & 1):
                        yield
                    at, low_at, last = main_turn % sets, low_turn % sets, s + 1 == per_tile
                    if run == 0:
                        while not main_empty[at].done(1 ^ (main_turn // sets & 1)):
                            yield
                        main[at] = []
                    main[at].append(planes[turn % stages])
                    run += 1
                    if run == (FIRST_RUN if s < FIRST_RUN else run_length) or last:
                        main_full[at].arrive()
                        run, main_turn = 0, main_turn + 1
                    yield
                    if s % LOW_RUN == 0:
                        while not low_empty[low_at].done(1 ^ (low_turn // sets & 1)):
                            yield
                        low[low_at] = []
                    low[low_at].append(planes[turn % stages])
                    empty[turn % stages].arrive()
                    if (s + 1) % LOW_RUN == 0 or last:
                        low_full[low_at].arrive()
                        low_turn += 1
                    turn += 1
                    yield

        def epilogue():
            main_turn = low_turn = 0
            for t in range(tiles):
                s, is_low, mains, lows = 0, False, [], []
                while True:
                    turn = low_turn if is_low else main_turn
                    while not (low_full if is_low else main_full)[turn % sets].done(turn // sets & 1):
                        yield
                    (lows if is_low else mains).extend((low if is_low else main)[turn % sets])
                    for _ in range(rng.choice([1, 1, 40])):
                        yield
                    (low_empty if is_low else main_empty)[turn % sets].arrive()
                    if is_low:
                        low_turn, is_low = low_turn + 1, False
                        if s == per_tile:
                            break
                    else:
                        main_turn, s = main_turn + 1, min(s + (FIRST_RUN if s == 0 else run_length), per_tile)
                        is_low = s % LOW_RUN == 0 or s == per_tile
                assert mains == lows == [(t, i) for i in range(per_tile)]
                drained.append(t)

        play(rng, fill(total, per_tile, raws, stages, raw_full, raw_empty, full, empty, planes) + [tensor_core(), epilogue()], sum(groups, []))
        assert drained == list(range(tiles))


@pytest.mark.parametrize("run_length", [1, 2])
def test_products_of_two_activations(run_length, stages=2, sets=2, raws=1):
    for seed in range(300):
        rng = random.Random(seed)
        tiles, per_tile = rng.randrange(1, 6), rng.randrange(1, 20)
        groups = [bars(n) for n in (raws, raws, stages, stages, sets, sets)]
        raw_full, raw_empty, full, empty, acc_full, acc_empty = groups
        planes, acc, drained = [None] * stages, [[] for _ in range(sets)], []

        def tensor_core():
            turn = runs = 0
            for t in range(tiles):
                run = 0
                for s in range(per_tile):
                    while not full[turn % stages].done(turn // stages & 1):
                        yield
                    at = runs % sets
                    if run == 0:
                        while not acc_empty[at].done(1 ^ (runs // sets & 1)):
                            yield
                        acc[at] = []
                    acc[at].append(planes[turn % stages])
                    empty[turn % stages].arrive()
                    run += 1
                    if run == run_length or s + 1 == per_tile:
                        acc_full[at].arrive()
                        run, runs = 0, runs + 1
                    turn += 1
                    yield

        def epilogue():
            turn = 0
            for t in range(tiles):
                got = []
                for s in range(0, per_tile, run_length):
                    while not acc_full[turn % sets].done(turn // sets & 1):
                        yield
                    got += acc[turn % sets]
                    for _ in range(rng.choice([1, 1, 40])):
                        yield
                    acc_empty[turn % sets].arrive()
                    turn += 1
                assert got == [(t, i) for i in range(per_tile)]
                drained.append(t)

        play(rng, fill(tiles * per_tile, per_tile, raws, stages, raw_full, raw_empty, full, empty, planes) + [tensor_core(), epilogue()], sum(groups, []))
        assert drained == list(range(tiles))


# Of a pair, either CTA arrives on the other's barriers: a wait of CTA scope would not order what the other one did before.
@pytest.mark.parametrize("kernel", sorted(SOURCE))
def test_pairs_wait_at_cluster_scope(kernel):
    waits = re.findall(r".*mbar_wait\w*.*", SOURCE[kernel])
    assert waits and all("kPair ? mbar_wait_cluster_flag : mbar_wait_flag" in line for line in waits)
