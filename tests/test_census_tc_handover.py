"""The hand-overs between the warps of a tensor-core census CTA
(csrc/census_tc.cuh: named barriers for staged rows and for accumulators read,
mbarriers for finished MMAs) as a model on the CPU, run under schedules that
hold back single warps for long. No GPU is needed, and none sees a schedule that
goes wrong."""
import random
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parents[1] / "module.clutec.cuda_b200" / "csrc" / "census_tc.cuh").read_text()
WIN, SLOTS = 5, 8
TILE_WARPS, ROW_WARPS = 3, 3  # (the kernel has 8 maxima warps a tile; the rule is the same for 3)


def _row_bars():
    """Barriers that staged rows take in turn."""
    m = re.search(r"constexpr int kRowBars = (\d+);", SRC)
    return int(m[1]) if m else int(re.search(r"row_arrive\(int r\) \{\s*switch \(r & (\d+)\)", SRC)[1]) + 1


def test_constants_of_the_model():
    assert re.search(rf"constexpr int kSlots = {SLOTS};", SRC)
    assert re.search(rf"kTileWarps = \d+, kRowWarps = {ROW_WARPS};", SRC)
    assert "constexpr int kR = 2;" in SRC


class Barrier:
    """A named barrier: a phase ends with the n-th arrival, whoever arrives."""

    def __init__(self, n):
        self.n, self.count, self.phase = n, 0, 0

    def arrive(self):
        self.count += 1
        if self.count == self.n:
            self.count, self.phase = 0, self.phase + 1


class Wrong(AssertionError):
    pass


class Model:
    """One strip of a tile pair. Actors are generators; what they yield is a
    condition to wait for, or with a second value True a wait that may give up
    (it then yields False). `give_up` is the chance of that for each time such a
    wait is looked at in vain; `stuck`: the tensor core completes nothing.
    `passed`: after it gave up a warp goes on when the MMA warp has begun the row
    (False: at once)."""

    def __init__(self, rng, rows, tiles, row_bars, give_up=0.0, stuck=False, passed=True):
        self.rng, self.rows, self.tiles = rng, rows, tiles
        self.give_up, self.stuck, self.passed = give_up, stuck, passed
        self.failed = False                # some wait gave up
        self.begun = [0] * tiles           # rows the MMA warp has begun
        self.row = [Barrier(ROW_WARPS + 1) for _ in range(row_bars)]
        self.read = [Barrier(TILE_WARPS + 1) for _ in range(tiles)]
        self.staged = [[-1] * ROW_WARPS for _ in range(SLOTS)]  # row held by a slot, each warp's part
        self.issued = []                   # MMAs (tile, row) in the tensor core, in order
        self.done = [0] * tiles            # rows whose MMAs are complete
        self.reads = [[0] * TILE_WARPS for _ in range(tiles)]   # rows each maxima warp has read

    def sync(self, bar):
        phase = bar.phase
        bar.arrive()
        return lambda: bar.phase != phase

    def mma_warp(self):
        for k in range(WIN - 1):
            yield self.sync(self.row[k % len(self.row)])
        for s in range(self.rows):
            k = s + WIN - 1
            yield self.sync(self.row[k % len(self.row)])
            for t in range(self.tiles):
                yield self.sync(self.read[t])
                self.begun[t] = s + 1
                if self.failed:
                    continue
                if any(r < s for r in self.reads[t]):
                    raise Wrong(f"tile {t} row {s}: accumulator not read")
                for r in (range(WIN) if s == 0 else (k, s - 1)):
                    if any(h != r for h in self.staged[r % SLOTS]):
                        raise Wrong(f"tile {t} row {s}: row {r} not staged")
                self.issued.append((t, s))

    def ready(self, t, s, ok):
        """wait_ready: row s of tile t complete; after a give-up, begun."""
        ok = ok and (yield lambda: self.done[t] > s, True)
        if not ok:
            self.failed = True
            if self.passed:
                yield lambda: self.begun[t] > s
        return ok

    def tensor_core(self):
        if self.stuck:
            return
        for _ in range(self.rows * self.tiles):
            yield lambda: self.issued
            t, s = self.issued.pop(0)
            yield lambda: True
            self.done[t] = s + 1

    def staging_warp(self, w):
        ok = True
        for k in range(self.rows + WIN - 1):
            if k >= SLOTS:
                ok = yield from self.ready(self.tiles - 1, k - SLOTS + 1, ok)
            yield lambda: True
            if ok:
                self.staged[k % SLOTS][w] = k
            self.row[k % len(self.row)].arrive()

    def maxima_warp(self, t, w):
        yield lambda: True
        self.read[t].arrive()
        ok = True
        for s in range(self.rows):
            ok = yield from self.ready(t, s, ok)
            if ok:
                self.reads[t][w] = s + 1
            self.read[t].arrive()

    def run(self):
        actors = [self.mma_warp(), self.tensor_core()] + [self.staging_warp(w) for w in range(ROW_WARPS)]
        actors += [self.maxima_warp(t, w) for t in range(self.tiles) for w in range(TILE_WARPS)]
        # an actor's share of the steps: some are held back for long
        share = [10.0 ** self.rng.uniform(-4, 0) for _ in actors]
        unpack = lambda y: y if isinstance(y, tuple) else (y, False)  # noqa: E731
        waits = [next(a, None) for a in actors]
        while True:
            live = [(i, *unpack(c)) for i, c in enumerate(waits) if c is not None]
            ready = [(i, c, b) for i, c, b in live if c() or (b and self.give_up)]
            if not ready:
                break
            i, c, b = self.rng.choices(ready, [share[i] for i, _, _ in ready])[0]
            ok = bool(c())
            if not ok and self.rng.random() >= self.give_up:
                continue
            try:
                waits[i] = actors[i].send(ok)
            except StopIteration:
                waits[i] = None
        left = [i for i, c in enumerate(waits) if c is not None and not (i == 1 and self.failed)]
        if left:
            raise Wrong(f"stalled: actors {left}")


def _schedules(n, **kw):
    for seed in range(n):
        rng = random.Random(seed)
        Model(rng, rng.choice([1, 3, 4, 9, 20]), rng.choice([1, 2]), **kw).run()


def test_rows_are_handed_over_under_every_schedule():
    _schedules(400, row_bars=_row_bars())


def test_the_model_finds_barriers_that_come_round_too_early():
    """Staging warps run up to SLOTS rows ahead of the MMA warp, so fewer
    barriers let a row's phase end without it."""
    with pytest.raises(Wrong):
        _schedules(400, row_bars=SLOTS // 2)


@pytest.mark.parametrize("stuck", [False, True])
def test_a_warp_that_gave_up_keeps_the_hand_overs_in_step(stuck):
    """Whichever waits give up, and if the tensor core never answers, every warp
    comes to its end (where the CTA reports the failure)."""
    assert re.search(r"if \(polls == 0\) passed\(t, s\);", SRC)  # the rule as modelled
    _schedules(400, row_bars=_row_bars(), give_up=0.05, stuck=stuck)


def test_the_model_finds_arrivals_that_run_ahead_after_a_give_up():
    """Arrivals that nothing holds back end phases without the MMA warp, which
    then waits for good."""
    with pytest.raises(Wrong):
        _schedules(400, row_bars=_row_bars(), give_up=0.05, stuck=True, passed=False)
