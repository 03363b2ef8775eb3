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
    def __init__(self, steps, first, done):
        self.steps, self.first = steps, first
        self.q_full, self.added_full = [Barrier(1), Barrier(1)], [Barrier(1), Barrier(1)]
        self.added_read, self.outputs_read = [Barrier(WARPS), Barrier(WARPS)], [Barrier(WARPS), Barrier(WARPS)]
        self.state_in, self.done = Barrier(WARPS), [Barrier(1) for _ in range(done)]
        self.seen = []

    def done_of(self, k):
        n = len(self.done)
        return self.done[k % n], k // n

    # a role yields what it waits for, (barrier, use), or None for work that takes its time
    def issuer(self):
        for c in range(min(2, self.steps)):
            self.added_full[c & 1].arrive()
        for c in range(self.first, min(self.first + 2, self.steps)):
            self.q_full[(c - self.first) & 1].arrive()
        for c in range(self.steps):
            k = c - self.first
            if k >= 0:
                yield self.state_in, k
                yield self.q_full[k & 1], k >> 1
                if k >= 2:
                    yield self.outputs_read[k & 1], (k >> 1) - 1
                yield None
                self.done_of(k)[0].arrive()
            yield self.added_read[c & 1], c >> 1
            if c + 2 < self.steps:
                self.added_full[c & 1].arrive()
            if k >= 0:
                yield self.done_of(k)
                if c + 2 < self.steps:
                    self.q_full[k & 1].arrive()

    def state(self):
        for c in range(self.steps):
            k = c - self.first
            if k >= 0:
                if k > 0:
                    yield self.done_of(k - 1)
                yield None
                self.state_in.arrive()
            yield self.added_full[c & 1], c >> 1
            yield None
            self.added_read[c & 1].arrive()

    def outputs(self):
        for k in range(self.steps - self.first):
            yield self.done_of(k)
            yield None
            self.outputs_read[k & 1].arrive()
            yield None  # the adds, behind the arrival
            self.seen.append(k)


def _ends(walk, order):
    """Whether all roles come to their end, each as fast as its draw has it."""
    roles = [walk.issuer()] + [walk.state() for _ in range(WARPS)] + [walk.outputs() for _ in range(WARPS)]
    pace = [order.choice([1.0, 0.3, 0.03]) for _ in roles]
    waits = [None] * len(roles)
    while any(r is not None for r in roles):
        ready = [i for i, r in enumerate(roles) if r is not None and (waits[i] is None or waits[i][0].there(waits[i][1]))]
        if not ready:
            return False
        i = order.choices(ready, [pace[j] for j in ready])[0]
        try:
            waits[i] = next(roles[i])
        except StopIteration:
            roles[i] = None
    return True


@pytest.mark.parametrize("steps, first", [(1, 0), (2, 0), (3, 2), (9, 0), (12, 5)])
def test_every_order_comes_to_its_end(steps, first):
    for seed in range(300):
        walk = Walk(steps, first, done=2)
        assert _ends(walk, random.Random(seed)), (seed, "stuck")
        assert sorted(walk.seen) == sorted(list(range(steps - first)) * WARPS)


def test_one_barrier_for_products_would_not_do():
    """What the second one is there for: an output warp two products behind."""
    assert not all(_ends(Walk(9, 0, done=1), random.Random(seed)) for seed in range(300))
