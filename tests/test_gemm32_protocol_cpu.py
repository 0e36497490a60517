"""The barriers of the float16 products' roles (gemm32_f16.cu, gemm32_f16_outer.cu) as coroutines under random schedules: nothing waits for
good, every stage is drained once and in order, and a stage's units are read before the producers come round to their slot."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "memorax_b200", "csrc")
SLOTS = int(re.search(r"constexpr int kSlots = (\d+);", open(os.path.join(CSRC, "gemm32_common.cuh")).read()).group(1))


class Barrier:
    def __init__(self, count=1):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def done(self, parity):
        return (self.phase & 1) != parity


def play(rng, actors, progress):
    """Runs the coroutines in random order until all have ended."""
    idle, before = 0, None
    while actors:
        actor = rng.choice(actors)
        for _ in range(rng.randrange(1, 8)):
            if next(actor, "end") == "end":
                actors.remove(actor)
                break
        idle = idle + 1 if progress() == before else 0
        before = progress()
        assert idle < 5000, "everyone waits"


def bars(n):
    return [Barrier() for _ in range(n)]


# The product with a weight: hi*hi accumulators of runs of stages, one of the small products until an event or the tile's end.
@pytest.mark.parametrize("stages,sets", [(2, 1), (3, 2)])
@pytest.mark.parametrize("run_length", [1, 2])
def test_products_with_a_weight(stages, sets, run_length):
    for seed in range(300):
        rng = random.Random(seed)
        tiles, per_tile, p_event = rng.randrange(1, 6), rng.randrange(1, 17), rng.choice([0, .1, .5, 1])
        event = [[i > 0 and rng.random() < p_event for i in range(per_tile)] for _ in range(tiles)]
        full, empty, main_full, main_empty, low_full, low_empty = bars(stages), bars(stages), bars(sets), bars(sets), bars(sets), bars(sets)
        events, units, main, low, drained = [0] * SLOTS, [None] * SLOTS, [[] for _ in range(sets)], [[] for _ in range(sets)], []

        def producers():
            for turn in range(tiles * per_tile):
                t, s = divmod(turn, per_tile)
                while not empty[turn % stages].done(1 ^ (turn // stages & 1)):
                    yield
                units[turn % SLOTS] = (t, s)
                if event[t][s]:
                    events[turn % SLOTS] = turn + 1
                yield
                full[turn % stages].arrive()

        def tensor_core():
            turn = main_turn = low_turn = 0
            for t in range(tiles):
                low_open, run, most = False, 0, 0
                for s in range(per_tile):
                    while not full[turn % stages].done(turn // stages & 1):
                        yield
                    now = s > 0 and events[turn % SLOTS] == turn + 1
                    if now:
                        if run > 0:
                            main_full[main_turn % sets].arrive()
                            main_turn += 1
                        low_full[low_turn % sets].arrive()
                        run, low_turn, low_open = 0, low_turn + 1, False
                    at = main_turn % sets
                    if run == 0:
                        most = 2 if s == 0 else 1 if now else run_length
                        while not main_empty[at].done(1 ^ (main_turn // sets & 1)):
                            yield
                        main[at] = []
                    main[at].append((t, s))
                    run += 1
                    if run == most or s + 1 == per_tile:
                        main_full[at].arrive()
                        run, main_turn = 0, main_turn + 1
                    yield
                    if not low_open:
                        while not low_empty[low_turn % sets].done(1 ^ (low_turn // sets & 1)):
                            yield
                        low[low_turn % sets] = []
                    low[low_turn % sets].append((t, s))
                    low_open = True
                    empty[turn % stages].arrive()
                    turn += 1
                low_full[low_turn % sets].arrive()
                low_turn += 1
                yield

        def epilogue():
            turn = main_turn = low_turn = 0
            for t in range(tiles):
                s, was_drained, lows = 0, False, []
                while True:
                    is_low = s >= per_tile
                    if not is_low:
                        while not main_full[main_turn % sets].done(main_turn // sets & 1):
                            yield
                        is_low = s > 0 and not was_drained and events[turn % SLOTS] == turn + 1
                    if is_low:
                        while not low_full[low_turn % sets].done(low_turn // sets & 1):
                            yield
                        lows += low[low_turn % sets]
                        yield
                        low_empty[low_turn % sets].arrive()
                        low_turn += 1
                        yield
                        if s >= per_tile:
                            break
                        assert units[turn % SLOTS] == (t, s)
                        was_drained = True
                        continue
                    at = main_turn % sets
                    got = list(main[at])
                    yield
                    main_empty[at].arrive()
                    for _ in range(rng.choice([1, 1, 40])):   # (a warp that is held up behind its arrival)
                        yield
                    if s == 0:
                        assert units[turn % SLOTS] == (t, 0)
                    most, n, main_turn, was_drained = 2 if s == 0 else 1 if events[turn % SLOTS] == turn + 1 else run_length, 0, main_turn + 1, False
                    while True:
                        n, s, turn = n + 1, s + 1, turn + 1
                        if not (n < most and s < per_tile and events[turn % SLOTS] != turn + 1):
                            break
                    assert got == [(t, s - n + i) for i in range(n)]
                    drained.extend(got)
                assert lows == [(t, i) for i in range(per_tile)]

        play(rng, [producers(), tensor_core(), epilogue()],
             lambda: [b.phase for g in (full, empty, main_full, main_empty, low_full, low_empty) for b in g])
        assert drained == [(t, s) for t in range(tiles) for s in range(per_tile)]


# The product of two activations: one accumulator a run, units of the other CTA's columns that arrive when they please.
@pytest.mark.parametrize("run_length", [1, 2])
def test_products_of_two_activations(run_length, stages=2, sets=2):
    for seed in range(300):
        rng = random.Random(seed)
        tiles, per_tile, p_event = rng.randrange(1, 6), rng.randrange(1, 17), rng.choice([0, .1, .5, 1])
        event = [[i > 0 and rng.random() < p_event for i in range(per_tile)] for _ in range(tiles)]
        full, empty, acc_full, acc_empty, peer = bars(stages), bars(stages), bars(sets), bars(sets), bars(SLOTS)
        events, units, theirs, acc, sent = [0] * SLOTS, [None] * SLOTS, [None] * SLOTS, [[] for _ in range(sets)], []
        total = tiles * per_tile

        def producers():
            for turn in range(total):
                t, s = divmod(turn, per_tile)
                while not empty[turn % stages].done(1 ^ (turn // stages & 1)):
                    yield
                units[turn % SLOTS] = (t, s)
                sent.append(turn)
                if event[t][s]:
                    events[turn % SLOTS] = turn + 1
                yield
                full[turn % stages].arrive()

        def copies():   # of the other CTA's units
            for turn in range(total):
                while not sent:
                    yield
                for _ in range(rng.choice([0, 0, 30])):
                    yield
                theirs[sent.pop(0) % SLOTS] = divmod(turn, per_tile)
                peer[turn % SLOTS].arrive()

        def tensor_core():
            turn = runs = 0
            for t in range(tiles):
                run = 0
                for s in range(per_tile):
                    while not full[turn % stages].done(turn // stages & 1):
                        yield
                    if s > 0 and run > 0 and events[turn % SLOTS] == turn + 1:
                        acc_full[runs % sets].arrive()
                        run, runs = 0, runs + 1
                    at = runs % sets
                    if run == 0:
                        while not acc_empty[at].done(1 ^ (runs // sets & 1)):
                            yield
                        acc[at] = []
                    acc[at].append((t, s))
                    empty[turn % stages].arrive()
                    run += 1
                    if run == run_length or s + 1 == per_tile:
                        acc_full[at].arrive()
                        run, runs = 0, runs + 1
                    turn += 1
                    yield

        def epilogue():
            turn = run = 0
            for t in range(tiles):
                s = 0
                while s < per_tile:
                    while not acc_full[run % sets].done(run // sets & 1):
                        yield
                    slot, first = turn % SLOTS, s
                    got = list(acc[run % sets])
                    acc_empty[run % sets].arrive()
                    yield
                    n, run = 0, run + 1
                    while True:
                        while not peer[turn % SLOTS].done(turn // SLOTS & 1):
                            yield
                        n, s, turn = n + 1, s + 1, turn + 1
                        if not (n < run_length and s < per_tile and events[turn % SLOTS] != turn + 1):
                            break
                    assert got == [(t, first + i) for i in range(n)]
                for _ in range(rng.choice([1, 1, 60])):
                    yield
                assert units[slot] == theirs[slot] == (t, first)   # the sums are scaled at the tile's end

        play(rng, [producers(), copies(), tensor_core(), epilogue()], lambda: [b.phase for g in (full, empty, acc_full, acc_empty, peer) for b in g])
        assert not sent and [b.phase for b in peer] == [len(range(i, total, SLOTS)) for i in range(SLOTS)]


# Of a pair, either CTA arrives on the other's barriers: a wait of CTA scope would not order what the other one stored before.
@pytest.mark.parametrize("kernel", ["gemm32_f16.cu", "gemm32_f16_outer.cu"])
def test_pairs_wait_at_cluster_scope(kernel):
    source = open(os.path.join(CSRC, kernel)).read()
    waits = re.findall(r".*mbar_wait\w*.*", source)
    assert waits and all("kPair ? mbar_wait_cluster_flag : mbar_wait_flag" in line for line in waits)
