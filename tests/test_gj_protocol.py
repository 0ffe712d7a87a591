"""CPU model of the barrier protocol of the coarse inverse's tensor-core update (csrc/linalg.cu,
k_gjb_update_tc): a copy warp, an MMA warp and two epilogue groups, with copies and MMAs that complete
at random moments and waits that may give up.

The checks: every tile's sum is the product of its own row and column operands, the run never
deadlocks, and when the block ends no copy and no MMA is in flight -- also when one of the agents has
given up a wait while the others go on. With the last waits left to the agent that gave up, copies and
MMAs of the others can outlive the block; the model shows that, which is why they wait in any case."""
import random

import pytest
from test_ring_protocol import Bar, _schedule


def run(nrow, seed, giveup=None, always_wait=True):
    """giveup: (agent, number of the wait it gives up) or None. Returns (finished, log, left in flight)."""
    rnd = random.Random(seed)
    tiles = [(i, j) for i in range(nrow) for j in range(i + 1)][seed % 3:]
    a_full, drain = Bar(1), Bar(1)
    b_full, b_empty = [Bar(1), Bar(1)], [Bar(1), Bar(1)]
    acc_full, acc_empty = [Bar(1) for _ in range(4)], [Bar(1), Bar(1)]
    A, B, acc = [None], [None, None], [None] * 4
    inflight, pipe, log, done, left, waits = [], [], [], set(), [], {}

    def wait(agent, bar, parity, last=False):
        waits[agent] = waits.get(agent, -1) + (not last)
        if not last and giveup == (agent, waits[agent]):
            return False
        while not bar.test(parity):
            if left:                         # bounded: the model's run is over
                return False
            if giveup and rnd.random() < 2e-3:
                return False                 # a consequence of the first one
            yield 'w'
        return True

    def load(bar, store, k, value):
        bar.arrive(tx=1)
        inflight.append((bar, lambda: store.__setitem__(k, value)))

    def copies():
        row, na, nb, ok = None, 0, [0, 0], True
        for it, (i, j) in enumerate(tiles):
            for h in range(2):
                if it:
                    ok = yield from wait('copy', b_empty[h], (it - 1) & 1)
                if ok and h == 0 and i != row:
                    if it:
                        ok = yield from wait('copy', b_empty[1], (it - 1) & 1)
                    if ok:
                        load(a_full, A, 0, i)
                        na, row = na + 1, i
                if not ok:
                    break
                load(b_full[h], B, h, (j, h))
                nb[h] += 1
                yield
            if not ok:
                break
        if always_wait or not ok:
            if na:
                yield from wait('copy', a_full, (na - 1) & 1, last=True)
            for h in range(2):
                if nb[h]:
                    yield from wait('copy', b_full[h], (nb[h] - 1) & 1, last=True)
        done.add('copy')

    def mmas():
        row, na, ok = None, 0, True
        for it, (i, j) in enumerate(tiles):
            buf = it & 1
            if it >= 2:
                ok = yield from wait('mma', acc_empty[buf], ((it >> 1) - 1) & 1)
            if ok and i != row:
                ok = yield from wait('mma', a_full, na & 1)
                na, row = na + 1, i
            for h in range(2):
                if not ok:
                    break
                ok = yield from wait('mma', b_full[h], it & 1)
                if not ok:
                    break

                def product(k=2 * buf + h, h=h):
                    acc[k] = (A[0], B[h])
                pipe.append(product)
                pipe.append(b_empty[h].arrive)
                pipe.append(acc_full[2 * buf + h].arrive)
                yield
            if not ok:
                break
        if always_wait or not ok:
            pipe.append(drain.arrive)
            yield from wait('mma', drain, 0, last=True)
        done.add('mma')

    def tensor_pipe():                       # in order, each at a random moment
        while pipe or len(done) < 4:
            if pipe and rnd.random() < 0.3:
                pipe.pop(0)()
                yield
            else:
                yield 'w'

    def epilogue(g):
        for use, t in enumerate(range(g, len(tiles), 2)):
            ok = yield from wait(f'epi{g}', acc_full[2 * g], use & 1)
            if ok:
                ok = yield from wait(f'epi{g}', acc_full[2 * g + 1], use & 1)
            if not ok:
                break
            log.append((tiles[t], acc[2 * g], acc[2 * g + 1]))
            acc_empty[g].arrive()
            yield
        done.add(f'epi{g}')

    def block_end():
        while len(done) < 4:
            yield 'w'
        left.append(len(inflight) + len(pipe))

    tasks = dict(copy=copies(), mma=mmas(), pipe=tensor_pipe(), e0=epilogue(0), e1=epilogue(1), end=block_end())
    return _schedule(tasks, inflight, rnd), log, left, tiles


@pytest.mark.parametrize("nrow", [1, 2, 3, 5])
def test_every_tile_gets_its_operands(nrow):
    for seed in range(60):
        ok, log, left, tiles = run(nrow, seed)
        assert ok and left == [0]
        assert sorted(t for t, _, _ in log) == sorted(tiles)
        for (i, j), a, b in log:
            assert a == (i, (j, 0)) and b == (i, (j, 1))


def _leftovers(always_wait):
    n = 0
    for agent in ('copy', 'mma', 'epi0', 'epi1'):
        for k in range(10):
            for seed in range(12):
                ok, log, left, _ = run(4, seed, (agent, k), always_wait)
                assert ok
                n += left != [0]
                for (i, j), a, b in log:     # what was summed before stays right
                    assert a == (i, (j, 0)) and b == (i, (j, 1))
    return n


def test_nothing_in_flight_after_a_wait_gave_up():
    assert _leftovers(True) == 0


def test_last_waits_left_to_the_one_that_gave_up_are_not_enough():
    assert _leftovers(False) > 0
