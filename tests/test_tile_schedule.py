"""The tiled step group's windows (k_tile), restated on the CPU: blocks of warps
in random interleavings, with the kernel's list buffers, mailboxes, step counters
and block barriers, and nothing else between them; a counter's additions are seen
by readers some time after they are made.  Every block must deliver each
window's spikes exactly once, and every spike must get a raster place of its own
in its own window.

The number of list buffers is the kernel's (kTileLists).  With two, a warp that
has no spike left to record starts the next window's update and overwrites
entries that a slower warp of the block has yet to read; the restatement shows
that."""
import os
import random
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "mgbrain_b200", "csrc", "tile.cuh")).read()

WARPS = 3      # warp 0 publishes, polls and sums the counters; warp 1 reserves the places
INLINE = 2     # spikes a mailbox place holds: one in its first chunk, one in its second
GATHERED = 12  # spikes of a window that fit in shared memory
SLOTS = 4      # counters


class Failure(Exception):
    pass


class Block:
    def __init__(self, tiles):
        self.count = self.total = 0
        self.mine = [None] * INLINE
        self.cnt = [0] * tiles
        self.spikes = []
        self.ctot = [0] * SLOTS
        self.sbase = [0, 0]
        self.stot = 0
        self.arrived = 0
        self.generation = 0
        self.delivered = []     # per window


def empty_mail(tiles):
    """[parity][reader][tile] places of two chunks {epoch, count, spike}, {epoch, spike}, all zero."""
    return [[[[(0, 0, None), (0, None)] for _ in range(tiles)] for _ in range(tiles)] for _ in range(2)]


class Group:
    """One launch of `windows` windows over `tiles` blocks; load[k][b][w]: spikes
    of warp w of block b in window k; counter: what the step counters hold at its
    start; add_up: readers wait until a window's counts add up to its spikes; mail,
    epoch: what earlier launches left, the first window's epoch."""

    def __init__(self, load, lists, seed, counter=0, add_up=True, mail=None, epoch=1, epochs=1 << 32):
        self.load, self.lists, self.add_up, self.epoch, self.epochs = load, lists, add_up, epoch, epochs
        self.windows, self.tiles = len(load), len(load[0])
        self.rng = random.Random(seed)
        self.list = [[[] for _ in range(self.tiles)] for _ in range(lists)]
        self.mail = mail or empty_mail(self.tiles)
        self.counter = [counter] * SLOTS
        self.seen = list(self.counter)      # what a reader gets: the counters of some time ago
        self.raster = [{} for _ in range(self.windows)]
        self.blocks = [Block(self.tiles) for _ in range(self.tiles)]

    def spike(self, k, b, w, i):
        return (k, b, w, i)

    def barrier(self, blk):
        blk.arrived += 1
        g = blk.generation
        if blk.arrived == WARPS:
            blk.arrived = 0
            blk.generation += 1
        while blk.generation == g:
            yield False            # waits: no progress

    def put(self, b, k, pos, e):
        row = self.list[k % self.lists][b]
        row.extend([None] * (pos + 1 - len(row)))
        row[pos] = e

    def record(self, k, b, w, c):
        blk = self.blocks[b]
        for q in range(w, c, WARPS):
            e = self.list[k % self.lists][b][q]
            yield True
            at = blk.sbase[k & 1]
            blk.sbase[k & 1] += 1
            if e is None or e[0] != k or e[1] != b:
                raise Failure(f"window {k}, tile {b}: entry {q} of its list is {e}")
            if at in self.raster[k] or not 0 <= at < blk.stot:
                raise Failure(f"window {k}: place {at} of {blk.stot}")
            self.raster[k][at] = e
            yield True

    def totals(self, k, blk, n):
        while self.add_up and self.seen[k % SLOTS] - blk.ctot[k % SLOTS] != n:
            yield False
        now = self.seen[k % SLOTS]
        blk.stot = now - blk.ctot[k % SLOTS]
        blk.ctot[k % SLOTS] = now

    def gather(self, k, b, w):
        """tile_gather: polled by warp 0; long lists copied by all warps."""
        blk = self.blocks[b]
        if w == 0:
            blk.spikes = [None] * GATHERED
            for l in range(self.tiles):
                place = self.mail[k & 1][b][l]
                epoch = (self.epoch + k) % self.epochs
                while place[0][0] != epoch:
                    yield False
                _, c, e = place[0]
                first = [e]
                if 1 < c <= INLINE:
                    while place[1][0] != epoch:
                        yield False
                    first.append(place[1][1])
                at = blk.total
                blk.total += c
                blk.cnt[l] = (c, at)
                if at + c <= GATHERED and c <= INLINE:
                    blk.spikes[at:at + c] = first[:c]
                yield True
        yield from self.barrier(blk)
        if blk.total <= GATHERED and any(c > INLINE for c, _ in blk.cnt):
            for l in range(w, self.tiles, WARPS):
                c, at = blk.cnt[l]
                if c > INLINE:
                    for q in range(c):
                        blk.spikes[at + q] = self.list[k % self.lists][l][q]
                        yield True
            yield from self.barrier(blk)

    def publish(self, k, b, c):
        blk = self.blocks[b]
        epoch = (self.epoch + k) % self.epochs
        for r in range(self.tiles):
            self.mail[k & 1][r][b][0] = (epoch, c, blk.mine[0])
            yield True
            if 1 < c <= INLINE:
                self.mail[k & 1][r][b][1] = (epoch, blk.mine[1])
                yield True

    def warp(self, b, w):
        blk = self.blocks[b]
        c_prev = n_prev = 0
        for k in range(self.windows):
            for i in range(self.load[k][b][w]):         # the update's spikes
                pos = blk.count
                blk.count += 1
                yield True
                e = self.spike(k, b, w, i)
                if pos < INLINE:
                    blk.mine[pos] = e
                self.put(b, k, pos, e)
                yield True
            yield from self.barrier(blk)
            c_now = blk.count
            yield True
            place = 0
            if w == 0:
                yield from self.publish(k, b, c_now)
            if w == 1:
                place = self.counter[k % SLOTS]
                self.counter[k % SLOTS] += c_now
                yield True
            yield from self.gather(k, b, w)
            if w == 1:
                blk.sbase[k & 1] = place - blk.ctot[k % SLOTS]
            if w == 0:
                blk.count = 0
                if k > 0:
                    yield from self.totals(k - 1, blk, n_prev)
            n_prev = blk.total
            yield True
            if blk.total <= GATHERED:                    # the delivery
                for q in range(w, blk.total, WARPS):
                    blk.delivered.append(blk.spikes[q])
                    yield True
            else:
                for l in range(self.tiles):
                    c, _ = blk.cnt[l]
                    for q in range(w, c, WARPS):
                        blk.delivered.append(self.list[k % self.lists][l][q] if c > INLINE
                                             else self.mail[k & 1][b][l][q][-1])
                        yield True
            yield from self.barrier(blk)
            if w == 0:
                blk.total = 0
            if k > 0:
                yield from self.record(k - 1, b, w, c_prev)
            c_prev = c_now
        k = self.windows
        if w == 0:
            yield from self.publish(k, b, 0)
        yield from self.gather(k, b, w)
        if w == 0:
            yield from self.totals(k - 1, blk, n_prev)
        yield from self.barrier(blk)
        yield from self.record(k - 1, b, w, c_prev)

    def run(self):
        live = [self.warp(b, w) for b in range(self.tiles) for w in range(WARPS)]
        weight = [1] * len(live)
        idle = 0
        while live:
            if self.rng.random() < 0.05:                 # some warps run ahead of the others for a while
                weight = [self.rng.choice((1, 1, 30)) for _ in live]
            if self.rng.random() < 0.02:
                self.seen = list(self.counter)
            i = self.rng.choices(range(len(live)), weight[:len(live)])[0]
            try:
                idle = 0 if next(live[i]) else idle + 1
            except StopIteration:
                live.pop(i)
            if idle > 100_000:
                raise Failure("every warp waits")
        for k in range(self.windows):
            want = {self.spike(k, b, w, i) for b in range(self.tiles) for w in range(WARPS)
                    for i in range(self.load[k][b][w])}
            if set(self.raster[k].values()) != want:
                raise Failure(f"window {k}: raster {sorted(self.raster[k].values())}")
            if sorted(self.raster[k]) != list(range(len(want))):
                raise Failure(f"window {k}: places {sorted(self.raster[k])}")
        want = sorted(self.spike(k, b, w, i) for k in range(self.windows) for b in range(self.tiles)
                      for w in range(WARPS) for i in range(self.load[k][b][w]))
        for b, blk in enumerate(self.blocks):
            if None in blk.delivered or sorted(blk.delivered) != want:
                raise Failure(f"tile {b} delivered other spikes")


def loads(seed):
    rng = random.Random(seed)
    tiles = rng.choice((1, 2, 3))
    most = rng.choice((1, 3, 6))
    return [[[rng.randint(0, most) for _ in range(WARPS)] for _ in range(tiles)] for _ in range(rng.randint(1, 6))]


def kernel_lists():
    m = re.search(r"constexpr int kTileLists = (\d+);", SOURCE)
    return int(m.group(1)) if m else 2      # (buffer k & 1 before there was a constant)


@pytest.mark.parametrize("chunk", range(8))
def test_windows_deliver_and_record_every_spike_once(chunk):
    for seed in range(60 * chunk, 60 * (chunk + 1)):
        Group(loads(seed), kernel_lists(), seed).run()


def test_two_list_buffers_would_not_do():
    failed = 0
    for seed in range(200):
        try:
            Group(loads(seed), 2, seed).run()
        except Failure:
            failed += 1
    assert failed > 0


def test_counters_must_be_zero_at_a_launch():
    """A launch whose waits ran out leaves counts behind: the next one's raster
    places would be off by them, and could lie past the history's end."""
    with pytest.raises(Failure, match="places"):
        Group([[[1, 1, 1]], [[1, 1, 1]]], kernel_lists(), 0, counter=5, add_up=False).run()
    with pytest.raises(Failure, match="waits"):
        Group([[[1, 1, 1]], [[1, 1, 1]]], kernel_lists(), 0, counter=5).run()


def test_counters_are_read_until_they_add_up():
    """The mailbox stores that tell of a window are not ordered after its counts."""
    failed = 0
    for seed in range(100):
        try:
            Group(loads(seed), kernel_lists(), seed, add_up=False).run()
        except Failure:
            failed += 1
    assert failed > 0
    for body in SOURCE.split("__global__")[1:]:      # both kernels read them so
        assert re.search(r"n_all \|\| !tile_again\(|!= n_all && tile_again\(", body)


def launches(seed, epochs, cleared):
    """Launches on one handle whose epochs wrap; cleared: the mailboxes are, and the
    epochs start again at 1, before a launch that would reach the wrap."""
    rng = random.Random(seed)
    tiles = rng.choice((2, 3))
    mail, epoch = empty_mail(tiles), 1
    for n in range(12):
        load = [[[rng.choice((0, 0, 1)) for _ in range(WARPS)] for _ in range(tiles)]
                for _ in range(rng.randint(1, 6))]
        windows = len(load) + 1           # the last one is empty
        if cleared and epoch + windows > epochs - 1:
            mail, epoch = empty_mail(tiles), 1
        Group(load, kernel_lists(), seed * 100 + n, mail=mail, epoch=epoch, epochs=epochs).run()
        epoch += windows


def test_epochs_that_wrap():
    for seed in range(40):
        launches(seed, 16, True)
    failed = 0
    for seed in range(40):
        try:
            launches(seed, 16, False)
        except Failure:
            failed += 1
    assert failed > 0
