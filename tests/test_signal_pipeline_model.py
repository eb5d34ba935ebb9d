"""The barrier protocol of the tensor-core Signal's warp roles (csrc/signal_tc.cu),
modelled on the CPU: waits and arrivals in any order the roles allow.  A run ends
without an arrival beyond a barrier's count and with every wait answered by the
phase it means; a run in which some wait runs out ends too, with every role out of
its loops soon after."""
import random

import pytest

BLOCK, OPERANDS, DRAINS, ARRIVALS = 8, 13, 8, 6


def drain_of(generic, narrow):
    """Stages of an accumulation group."""
    return 32 if generic or narrow else 12


class Bar:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self, n=1):
        assert n <= self.left, "more arrivals than the barrier counts"
        self.left -= n
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def done(self, parity):
        return (self.phase & 1) != parity


class Block:
    """One thread block: `units` = (stages, row groups, generic, narrow) each."""

    def __init__(self, units, bufs, ring, seed, fail_at=None, at_once=False):
        self.units, self.bufs, self.ring, self.rnd = units, bufs, ring, random.Random(seed)
        self.full, self.empty = [Bar(ARRIVALS) for _ in range(ring)], [Bar(1) for _ in range(ring)]
        self.accfull, self.accfree = Bar(1), Bar(DRAINS)
        self.nodefull, self.nodeempty = [Bar(1) for _ in range(bufs)], [Bar(OPERANDS) for _ in range(bufs)]
        self.unit_bar, self.unit_any = Bar(OPERANDS), []
        self.fail_at, self.at_once, self.abort = fail_at, at_once, False
        self.steps = self.steps_after = 0

    def wait(self, bar, parity, phase=None):
        """Yields until the phase is done; False when the wait failed."""
        ok = yield (bar, parity)
        assert not ok or phase is None or self.abort or bar.phase == phase, "answered by another phase"
        return ok

    def arrive(self, bar, n):
        """n single arrivals, or one of count n."""
        for k in [n] if self.at_once else [1] * n:
            bar.arrive(k)

    def mma(self):
        stage = group = 0
        for n, _, generic, narrow in self.units:
            drain = drain_of(generic, narrow)
            for st in range(n):
                if st % drain == 0 and not (yield from self.wait(self.accfree, (group & 1) ^ 1, group)):
                    return
                slot, turn = stage % self.ring, stage // self.ring
                if not (yield from self.wait(self.full[slot], turn & 1, turn + 1)):
                    return
                self.empty[slot].arrive()
                if st % drain == drain - 1 or st == n - 1:
                    self.accfull.arrive()
                    group += 1
                stage += 1

    def nodes(self, d):
        block0 = 0
        for n, *_ in self.units:
            blocks = -(-n // BLOCK)
            for blk in range((d + block0) & 1, blocks, 2):
                b, turn = (block0 + blk) % self.bufs, (block0 + blk) // self.bufs
                if not (yield from self.wait(self.nodeempty[b], (turn & 1) ^ 1, turn)):
                    return
                self.nodefull[b].arrive()
            block0 += blocks

    def operands(self, warp):
        # failed waits are not looked at: the warp walks on to the end of its unit
        stage0 = group0 = next_buf = 0
        drains = warp < DRAINS
        for unit, (n, groups, generic, narrow) in enumerate(self.units):
            drain = drain_of(generic, narrow)
            blocks, n_acc = -(-n // BLOCK), -(-n // drain)
            a_groups = 3 if generic else 2
            n_a = a_groups * groups
            is_a = warp < n_a
            per = 1 if narrow or OPERANDS - n_a < 4 else 2
            b_groups = 0 if generic else min((OPERANDS - n_a) // per, self.ring)
            step = a_groups if is_a else b_groups
            first = warp // groups if is_a else (warp - n_a) // per
            count = 1 if not is_a or warp % groups else ARRIVALS - (groups - 1) - (0 if generic else per)
            blk, folded, buf = -1, 0, 0

            def acquire(to):
                nonlocal blk, buf, next_buf
                while blk < to:
                    b, turn = next_buf % self.bufs, next_buf // self.bufs
                    yield from self.wait(self.nodefull[b], turn & 1, turn + 1)
                    buf, next_buf, blk = b, next_buf + 1, blk + 1
                    if blk < to:
                        self.nodeempty[buf].arrive()

            def fold_before(st):
                nonlocal folded
                while drains and folded < n_acc - 1 and st >= (folded + 1) * drain + self.ring - 1:
                    g = group0 + folded
                    yield from self.wait(self.accfull, g & 1, g + 1)
                    self.accfree.arrive()
                    folded += 1

            for st in range(first, n, step) if is_a or first < b_groups else ():
                slot, turn = (stage0 + st) % self.ring, (stage0 + st) // self.ring
                yield from fold_before(st)
                yield from acquire(st // BLOCK)
                yield from self.wait(self.empty[slot], (turn & 1) ^ 1, turn)
                yield None  # other warps run while the stage is written
                self.arrive(self.full[slot], count)
                if st + step >= n or (st + step) // BLOCK > blk:
                    self.nodeempty[buf].arrive()
            while blk < blocks - 1:
                yield from fold_before((blk + 1) * BLOCK)
                yield from acquire(blk + 1)
                self.nodeempty[buf].arrive()
            yield from fold_before(n + drain + self.ring)
            # the barrier that also tells whether any warp knows of a failed wait
            if len(self.unit_any) == unit:
                self.unit_any.append(False)
            self.unit_any[unit] |= self.abort
            turn = self.unit_bar.phase
            self.unit_bar.arrive()
            yield (self.unit_bar, turn & 1, True)
            if self.unit_any[unit]:
                return
            if drains and n > 0:
                g = group0 + folded
                yield from self.wait(self.accfull, g & 1, g + 1)
                self.accfree.arrive()
            stage0, group0 = stage0 + n, group0 + n_acc

    def run(self):
        roles = [self.mma(), self.nodes(0), self.nodes(1)] + [self.operands(w) for w in range(OPERANDS)]
        waits, slow = {}, [self.rnd.choice([0, 0.5, 0.95]) for _ in roles]
        answer = [None] * len(roles)
        alive = set(range(len(roles)))

        def ready(i):
            w = waits.get(i)
            return w is None or w[0].done(w[1])
        while alive:
            able = [i for i in alive if ready(i)]
            timed = [i for i in alive if not ready(i) and len(waits[i]) == 2]
            fails = timed and self.fail_at is not None and self.steps >= self.fail_at
            if fails and (not self.abort or not able or self.rnd.random() < 0.3):
                i = self.rnd.choice(timed)  # its wait runs out, or ends because another did
                self.abort, answer[i] = True, False
            else:
                assert able, f"roles {sorted(alive)} wait for ever"
                i = self.rnd.choice([i for i in able if self.rnd.random() >= slow[i]] or able)
                answer[i] = True
            self.steps += 1
            self.steps_after += self.abort
            try:
                w = roles[i].send(None if i not in waits else answer[i])
                if w is None:
                    waits[i] = (Bar(1), 1)  # ready at once
                else:
                    waits[i] = w
            except StopIteration:
                alive.discard(i)
                waits.pop(i, None)
        return self


UNITS = [
    [(75, 4, False, False)],
    [(75, 4, True, False), (75, 3, False, False), (75, 1, False, True)],
    [(n, 1 + n % 4, n % 3 == 0, n % 2 == 0) for n in (1, 2, 33, 34, 35, 64, 65, 8, 9, 1, 1, 1, 40)],
    [(7, 2, False, True), (0, 1, False, False), (5, 4, True, False), (32, 3, False, False), (96, 4, False, False)],
]
LAYOUTS = [(2, 8), (4, 3), (4, 8), (2, 3), (3, 5)]  # node buffers, ring slots


@pytest.mark.parametrize("bufs,ring", LAYOUTS)
@pytest.mark.parametrize("units", UNITS)
def test_every_wait_is_answered(units, bufs, ring):
    for seed in range(4):
        Block(units, bufs, ring, seed).run()


def _failures(units, bufs, ring, runs, **kw):
    """Runs in which a wait runs out, at places spread over the whole of a run."""
    total = Block(units, bufs, ring, 0).run().steps
    for seed in range(runs):
        yield Block(units, bufs, ring, seed, fail_at=random.Random(seed).randrange(total), **kw).run()


@pytest.mark.parametrize("bufs,ring", LAYOUTS)
@pytest.mark.parametrize("units", UNITS)
def test_a_block_ends_after_a_failed_wait(units, bufs, ring):
    longest = max(n for n, *_ in units)
    for block in _failures(units, bufs, ring, 12):
        # the MMA and node roles end with their next wait, the operand warps at the
        # end of the unit that they are in or, met at its barrier, of the next
        assert block.steps_after <= 16 * (2 * 4 * longest + 40)


def test_counted_arrivals_overflow_a_barrier():
    """Why arrivals are single ones: one of a count, made without the room that a
    wait stands for, exceeds what its phase has left."""
    with pytest.raises(AssertionError, match="more arrivals"):
        for _ in _failures(UNITS[1], 4, 4, 50, at_once=True):
            pass
