"""The barriers between the roles of the tile walk (``csrc/tile_walk.cu``, ``tile_walk_kernel``): the issuing thread, the state's warps and the
output warps as they wait and arrive there, run against one another in random orders. A wait asks for a phase's parity, as on the device: two phases ahead reads as
not there yet."""
import random

import pytest

WARPS = 2  # of the state, of the outputs (eight each on the device)


class Barrier:
    def __init__(self, count):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def there(self, use):
        return (self.phase & 1) != (use & 1)


class Walk:
    """``no_queries``, ``no_added``: the first chunks whose copies never come."""

    def __init__(self, steps, first, done=2, plain=(), no_queries=1 << 30, no_added=1 << 30):
        self.steps, self.first, self.plain, self.no_queries, self.no_added = steps, first, plain, no_queries, no_added
        self.q_full, self.added_full = [Barrier(1), Barrier(1)], [Barrier(1), Barrier(1)]
        self.added_read, self.outputs_read = [Barrier(WARPS), Barrier(WARPS)], [Barrier(WARPS), Barrier(WARPS)]
        self.state_in, self.done, self.state_read = Barrier(WARPS), [Barrier(1) for _ in range(done)], Barrier(WARPS)
        self.vote, self.last = Barrier(WARPS), Barrier(1 + 2 * WARPS)  # (no bound: everyone has to come)
        self.seen, self.raised, self.kept = [], 0, 0

    def done_of(self, k):
        n = len(self.done)
        return self.done[k % n], k // n

    # A role yields (barrier, use), which gives whether the wait ended well, or None for work that takes its time. `wait` does no more once one has run out.
    def wait(self, ok, bar, use):
        return ok and (yield bar, use)

    def meet(self, bar):
        use = bar.phase
        bar.arrive()
        yield bar, use, "unbounded"

    def copy(self, bars, at, chunk, none_from):
        if chunk < none_from:
            bars[at & 1].arrive()

    def issuer(self):
        ok = True
        for c in range(min(2, self.steps)):
            self.copy(self.added_full, c, c, self.no_added)
        for c in range(self.first, min(self.first + 2, self.steps)):
            self.copy(self.q_full, c - self.first, c, self.no_queries)
        for c in range(self.steps):
            k = c - self.first
            if k >= 0:
                ok = yield from self.wait(ok, self.state_in, k)
                ok = yield from self.wait(ok, self.q_full[k & 1], k >> 1)
                if k >= 2:
                    ok = yield from self.wait(ok, self.outputs_read[k & 1], (k >> 1) - 1)
                if not ok:
                    break
                yield None
                self.done_of(k)[0].arrive()
            ok = yield from self.wait(ok, self.added_read[c & 1], c >> 1)
            if ok and c + 2 < self.steps:
                self.copy(self.added_full, c, c + 2, self.no_added)
            if k >= 0:
                ok = yield from self.wait(ok, *self.done_of(k))
                if ok and c + 2 < self.steps:
                    self.copy(self.q_full, k, c + 2, self.no_queries)
            if not ok:
                break
        self.raised += not ok
        yield from self.meet(self.last)

    def state(self):
        ok, plain_chunks = True, 0
        for c in range(self.steps):
            k = c - self.first
            if k >= 0:
                yield from self.meet(self.vote)
                if k > 0:
                    ok = yield from self.wait(ok, *self.done_of(k - 1))
                if k - 1 in self.plain:
                    ok = yield from self.wait(ok, self.state_read, plain_chunks)
                    plain_chunks += 1
                yield None
                self.state_in.arrive()
            ok = yield from self.wait(ok, self.added_full[c & 1], c >> 1)
            yield None
            self.added_read[c & 1].arrive()
        self.raised += not ok
        yield from self.meet(self.vote)
        self.kept += ok
        yield from self.meet(self.last)

    def outputs(self):
        ok = True
        for k in range(self.steps - self.first):
            ok = yield from self.wait(ok, *self.done_of(k))
            if not ok:
                break
            yield None
            self.outputs_read[k & 1].arrive()
            yield None  # the adds, behind the arrival
            if k in self.plain:
                self.state_read.arrive()
            self.seen.append(k)
        self.raised += not ok
        yield from self.meet(self.last)


def _ends(walk, order):
    """Whether all roles come to their end, each as fast as its draw has it, where a wait that nothing can end runs out."""
    roles = [walk.issuer()] + [walk.state() for _ in range(WARPS)] + [walk.outputs() for _ in range(WARPS)]
    pace = [order.choice([1.0, 0.3, 0.03]) for _ in roles]
    waits = [None] * len(roles)
    while any(r is not None for r in roles):
        live = [i for i, r in enumerate(roles) if r is not None]
        ready, answer = [i for i in live if waits[i] is None or (waits[i][0].phase != waits[i][1] if len(waits[i]) == 3 else waits[i][0].there(waits[i][1]))], True
        if not ready:
            ready, answer = [i for i in live if len(waits[i]) == 2], False
            if not ready:
                return False
        i = order.choices(ready, [pace[j] for j in ready])[0]
        try:
            waits[i] = roles[i].send(None if waits[i] is None else answer)
        except StopIteration:
            roles[i] = None
    return True


@pytest.mark.parametrize("steps, first, plain", [(1, 0, ()), (2, 0, (0,)), (3, 2, ()), (9, 0, (2, 3, 7)), (12, 5, (6,)), (9, 0, tuple(range(9)))])
def test_every_order_comes_to_its_end(steps, first, plain):
    for seed in range(200):
        walk = Walk(steps, first, plain=plain)
        assert _ends(walk, random.Random(seed)) and walk.raised == 0 and walk.kept == WARPS, seed
        assert sorted(walk.seen) == sorted(list(range(steps - first)) * WARPS)


def test_one_barrier_for_products_would_not_do():
    """What the second one is there for: an output warp two products behind (its waits run out)."""
    def stuck(seed):
        walk = Walk(9, 0, done=1)
        return _ends(walk, random.Random(seed)) and walk.raised > 0
    assert any(stuck(seed) for seed in range(300))


@pytest.mark.parametrize("none", [dict(no_queries=0), dict(no_queries=3), dict(no_added=0), dict(no_added=4), dict(no_queries=2, no_added=2)])
@pytest.mark.parametrize("plain", [(), (0, 1, 4), tuple(range(9))])
def test_copies_that_do_not_come_end_the_walk(none, plain):
    """All roles come to their end and someone has raised the status word, plain chunks among them or not. A state that lacks what a chunk adds is not kept."""
    for seed in range(200):
        walk = Walk(9, 0, plain=plain, **none)
        assert _ends(walk, random.Random(seed)) and walk.raised > 0, seed
        assert "no_added" not in none or walk.kept == 0
