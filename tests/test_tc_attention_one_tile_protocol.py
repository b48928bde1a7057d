"""The barrier protocol of the tcgen05 attention kernel with ONE query tile per CTA, replayed on the host under random schedules.

`csrc/attention_tcgen05.cu` (`attn_tc_pp_kernel`, NT = 1): four score buffers, the even steps' softmax in one warpgroup and the odd
steps' in another, the maximum in use handed from step to step through shared memory, sums kept per side.  As in the model of the two-tile form every access
is checked for the step that it is meant for; waits are by parity, so a waiter may be at most one phase away.  Nothing orders the copies' completion: they
may take any time, and value copies another than key copies (`delay`).
"""
import random

import pytest
from test_tc_attention_protocol import Barrier, Deadlock


def simulate(nsteps, seed, NS=4, KE=1, buffers=4, threads=2, chained=True, product_first=True, delay=None):
    """`delay(rnd, kind, j)`: how long the copy of a piece of tile j takes ("K" or "V").  `product_first`: the score thread waits for the product that
    used its buffer before it waits for the tile's keys, as the kernel does."""
    rnd = random.Random(seed)
    delay = delay or (lambda rnd, kind, j: rnd.randint(1, 6))
    W = threads
    bars = {("FULL", i): Barrier(1) for i in range(NS)}
    bars.update({("EMPTY", i): Barrier(1) for i in range(NS)})
    for b in range(buffers):
        bars.update({("SF", b): Barrier(1), ("PF", b): Barrier(W), ("SC", b): Barrier(W), ("OC", b): Barrier(W), ("OF", b): Barrier(1)})
    bars.update({("LF", side): Barrier(W) for side in range(2)})
    queues, copies, ring = [[], []], [], [None] * NS
    scores, probs, alpha, ref, done = {}, {}, {}, {}, {"issued": -1, "landed": -1}
    slot, phase = lambda j: j % buffers, lambda j: (j // buffers) & 1

    def wait(name, parity):
        while not bars[name].passed(parity):
            yield

    def k_index(j):
        return KE * j if j < 2 else 2 * KE + (KE + 1) * (j - 2) + 1

    def v_index(j):
        return (KE + 1) * nsteps - 1 if j == nsteps - 1 else 2 * KE + (KE + 1) * j

    def producer():
        order = [("K", 0)] * KE + ([("K", 1)] * KE if nsteps > 1 else [])
        for j in range(nsteps):
            order += [("V", j)] + ([("K", j + 2)] * KE if j + 2 < nsteps else [])
        for it, tile in enumerate(order):
            yield from wait(("EMPTY", it % NS), ((it // NS) & 1) ^ 1)
            copies.append([delay(rnd, *tile), it % NS, tile])

    def score_issuer():
        def buffer_free(j):
            if j >= buffers:
                yield from wait(("OF", slot(j)), phase(j - buffers))
                assert done["landed"] >= j - buffers, ("scores over probabilities still in use", j)

        for j in range(nsteps):
            if product_first:
                yield from buffer_free(j)
            entries = [k_index(j) + e for e in range(KE)]
            for idx in entries:
                yield from wait(("FULL", idx % NS), (idx // NS) & 1)
            sts = [idx % NS for idx in entries]
            assert all(ring[st] == ("K", j) for st in sts), ("scores from the wrong tile", j)
            if not product_first:
                yield from buffer_free(j)
            queues[1] += [("S", j, sts), ("commit", ("SF", slot(j)))] + [("commit", ("EMPTY", st)) for st in sts]

    def pv_issuer():
        for j in range(nsteps):
            st = v_index(j) % NS
            yield from wait(("PF", slot(j)), phase(j))
            yield from wait(("OC", slot(j)), phase(j))
            yield from wait(("FULL", st), (v_index(j) // NS) & 1)
            assert ring[st] == ("V", j) and all(probs.get((slot(j), w)) == j for w in range(W)), ("product of another step", j)
            done["issued"] = j
            queues[0] += [("PV", j, st), ("commit", ("OF", slot(j))), ("commit", ("EMPTY", st))]

    def softmax(side, w):
        for j in range(side, nsteps, 2):
            yield from wait(("SF", slot(j)), phase(j))
            assert scores.get(slot(j)) == j, ("scores of another step", j)
            yield
            if j > 0 and chained:
                yield from wait(("SC", slot(j - 1)), phase(j - 1))
            if j > 0:
                assert ref.get((slot(j - 1), w)) == j - 1, ("maximum of another step", j, ref.get((slot(j - 1), w)))
            alpha[slot(j), w] = ref[slot(j), w] = j
            bars["SC", slot(j)].arrive()
            for _ in range(rnd.randint(0, 3)):
                yield
            assert scores.get(slot(j)) == j
            probs[slot(j), w] = j
            bars["PF", slot(j)].arrive()
        bars["LF", side].arrive()

    def correction(c):
        for j in range(nsteps):
            yield from wait(("SC", slot(j)), phase(j))
            assert all(alpha[slot(j), w] == j for w in range(W)), ("scale factors of another step", j)
            if j > 0 and rnd.random() < 0.5:
                yield from wait(("OF", slot(j - 1)), phase(j - 1))
                assert done == {"issued": j - 1, "landed": j - 1}, ("output rescaled beside a product", j, done)
                for _ in range(rnd.randint(0, 3)):
                    yield
            bars["OC", slot(j)].arrive()
        for side in range(2):
            yield from wait(("LF", side), 0)
        yield from wait(("OF", slot(nsteps - 1)), phase(nsteps - 1))
        assert done["landed"] == nsteps - 1, "output stored before the last product"

    agents = [producer(), score_issuer(), pv_issuer()] + [softmax(side, w) for side in range(2) for w in range(W)] + [correction(c) for c in range(W)]
    idle = 0
    while agents:
        before = (sum(b.phase * 1000 + b.pending for b in bars.values()), sum(map(len, queues)), len(copies))
        queue = rnd.choice(queues)
        if queue and rnd.random() < 0.5:
            op = queue.pop(0)
            if op[0] == "commit":
                bars[op[1]].arrive()
            elif op[0] == "S":
                assert all(ring[st] == ("K", op[1]) for st in op[2]), ("scores read a stage that was refilled", op)
                scores[slot(op[1])] = op[1]
            else:
                assert ring[op[2]] == ("V", op[1]), ("product read a stage that was refilled", op)
                done["landed"] = op[1]
        for c in list(copies):
            c[0] -= 1
            if c[0] <= 0:
                ring[c[1]] = c[2]
                bars["FULL", c[1]].arrive()
                copies.remove(c)
        agent = rnd.choice(agents)
        try:
            next(agent)
            moved = before != (sum(b.phase * 1000 + b.pending for b in bars.values()), sum(map(len, queues)), len(copies))
        except StopIteration:
            agents.remove(agent)
            moved = True
        idle = 0 if moved else idle + 1
        if idle > 20000:
            raise Deadlock(f"nothing moves: {nsteps} steps, seed {seed}")


@pytest.mark.parametrize("stages,key_entries,buffers", [(4, 1, 4), (5, 4, 4), (11, 4, 4)])      # head size 256; joint rows of 512, and with few rows
@pytest.mark.parametrize("nsteps", [1, 2, 3, 4, 5, 6, 9, 23])
def test_one_tile_protocol_holds_under_random_schedules(nsteps, stages, key_entries, buffers):
    for seed in range(60):
        simulate(nsteps, seed, NS=stages, KE=key_entries, buffers=buffers)


DELAYS = {
    "any time": lambda rnd, kind, j: rnd.choice((1, 6, 60, 600)),
    "slow values": lambda rnd, kind, j: 400 if kind == "V" else rnd.randint(1, 6),
    "slow keys": lambda rnd, kind, j: 400 if kind == "K" else rnd.randint(1, 6),
    "a late value tile": lambda rnd, kind, j: 3000 if (kind, j) == ("V", 1) else rnd.randint(1, 6),
    "a late key tile": lambda rnd, kind, j: 3000 if (kind, j) == ("K", 2) else rnd.randint(1, 6),
    "values of the first tile late": lambda rnd, kind, j: 3000 if (kind, j) == ("V", 0) else rnd.randint(1, 6),
}


@pytest.mark.parametrize("delay", sorted(DELAYS))
@pytest.mark.parametrize("stages,key_entries", [(4, 1), (5, 4), (11, 4)])
@pytest.mark.parametrize("nsteps", [2, 4, 5, 6, 9, 14])
def test_one_tile_protocol_holds_whatever_the_copies_take(nsteps, stages, key_entries, delay):
    for seed in range(10):
        simulate(nsteps, seed, NS=stages, KE=key_entries, delay=DELAYS[delay])


def test_keys_must_not_be_waited_for_before_the_product():
    """Eleven entries: the first piece of K(j) takes the entry of V(j - 4).  Only product j - 4 tells that those values had come; polled before it, the
    entry's barrier may still be in their phase, and a wait for the other parity passes."""
    with pytest.raises(AssertionError, match="wrong tile"):
        for seed in range(60):
            simulate(9, seed, NS=11, KE=4, product_first=False, delay=DELAYS["slow values"])


def test_the_maximum_must_wait_for_the_step_before():
    """Without the wait for the other side's decision the model must see a maximum of another step."""
    with pytest.raises((AssertionError, Deadlock)):
        for seed in range(60):
            simulate(12, seed, chained=False)
