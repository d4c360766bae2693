"""Model check of the barrier protocol of the persistent attention forward kernel (``attn_fwd_kernel`` in
mist_b200/csrc/attn_fwd_tcgen05.cu).

Roles: K / V producer, Q producer, MMA issuer, per query tile ``i`` and half ``h`` of the keys a row of softmax warps
(warp ``w`` of the two halves shares the same query rows), the in-order tensor-core queue.

    full[s], empty[s]     ring of five slots in the order K0 V0 K1 V1 ..., across work items
    q_full[i], q_empty[i] Q tile of tile i: loaded / read by its last S product
    s_full[i]             S of the block is in tensor memory (and P V of the block before is done: the queue is in order)
    p_full[i][part]       first / second 32 keys of both halves of P lie over S, O is rescaled
    o_full[i]             the item's last P V is done
    pair barrier          the two warps that share rows: maxima of a block, sums at the end of an item

The simulation replays waits, arrivals and parities over lists of work items whose tiles have unequal and zero numbers
of blocks, and checks liveness and that no buffer is overwritten while in use or read before it is written."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

from protocol_sim import GroupBarrier, MBar, Resource, Sim, Task, TensorQueue  # noqa: E402

SLOTS = 5


def simulate(items, seed, rows=2, slow=None, drop=()):
    """``items``: blocks of tile 0 and of tile 1 of each work item; ``rows``: softmax warps per half; ``drop``: waits left
    out (mutation check)."""
    sim = Sim(seed)
    slow = slow or {}

    def lat(role, lo, hi):
        return sim.lat(lo, hi) * slow.get(role, 1.0)

    full = [MBar(sim, f"full{s}", 1) for s in range(SLOTS)]
    empty = [MBar(sim, f"empty{s}", 1) for s in range(SLOTS)]
    q_full, q_empty, s_full, o_full = ([MBar(sim, f"{n}{i}", 1) for i in range(2)]
                                       for n in ("q_full", "q_empty", "s_full", "o_full"))
    p_full = [[MBar(sim, f"p_full{i}{part}", 2 * rows) for part in range(2)] for i in range(2)]
    ring = [Resource(f"slot{s}") for s in range(SLOTS)]
    Q = [Resource(f"Q{i}") for i in range(2)]
    # S and, over it, the two parts of P: [tile][half][warp][part]
    SP = [[[[Resource(f"S{i}{h}{w}{part}") for part in range(2)] for w in range(rows)] for h in range(2)] for i in range(2)]
    O = [[[Resource(f"O{i}{h}{w}") for w in range(rows)] for h in range(2)] for i in range(2)]
    MAX = [[[Resource(f"max{i}{h}{w}") for w in range(rows)] for h in range(2)] for i in range(2)]
    pair = [[GroupBarrier(sim, 2) for _ in range(rows)] for _ in range(2)]
    tq = TensorQueue(sim)

    def load(res, bar, what):
        res.write_begin(what)

        def land():
            res.write_end(what)
            bar.arrive()
        sim.at(lat("tma", 0.5, 3.0), land)

    def kv_producer():
        n = 0
        for t, nb in enumerate(items):
            for j in range(max(nb)):
                for what in ("K", "V"):
                    s = n % SLOTS
                    if n >= SLOTS and "empty" not in drop:
                        yield ("wait", empty[s], (n // SLOTS - 1) & 1)
                    load(ring[s], full[s], (what, t, j))
                    n += 1
                    yield ("sleep", 0.01)

    def q_producer():
        cq = [0, 0]
        for t, nb in enumerate(items):
            for i in range(2):
                if nb[i] == 0:
                    continue
                if cq[i] > 0 and "q_empty" not in drop:
                    yield ("wait", q_empty[i], (cq[i] - 1) & 1)
                load(Q[i], q_full[i], t)
                cq[i] += 1
                yield ("sleep", 0.01)

    def mma():
        cq, cp, blocks = [0, 0], [0, 0], [0, 0]       # Q tiles, P tiles, S tiles so far
        state = dict(slot=0, lap=0)
        work = [(t, nb) for t, nb in enumerate(items) if max(nb) > 0]

        def take_slot():
            at = state["slot"]
            yield ("wait", full[at], state["lap"])
            state["slot"] += 1
            if state["slot"] == SLOTS:
                state["slot"], state["lap"] = 0, state["lap"] ^ 1
            return at

        def issue_s(i, at, active, last, t, j):
            if active:
                n = blocks[i]
                blocks[i] += 1

                def start():
                    ring[at].read_begin(("K", t, j))
                    Q[i].read_begin(t)
                    for h in range(2):
                        for w in range(rows):
                            for part in range(2):
                                SP[i][h][w][part].write_begin(("S", n))

                def end():
                    ring[at].read_end()
                    Q[i].read_end()
                    for h in range(2):
                        for w in range(rows):
                            for part in range(2):
                                SP[i][h][w][part].write_end(("S", n))
                tq.op(lat("mma", 0.2, 0.5), start, end)
                tq.commit(s_full[i])
                if last:
                    tq.commit(q_empty[i])
            if i == 1:
                tq.commit(empty[at])

        def first_s(t, nb, i, at):
            if nb[i] > 0:
                yield ("wait", q_full[i], cq[i] & 1)
                cq[i] += 1
            issue_s(i, at, nb[i] > 0, nb[i] == 1, t, 0)

        if not work:
            return
        at = yield from take_slot()
        for i in range(2):
            yield from first_s(*work[0], i, at)
        for k, (t, nb) in enumerate(work):
            nxt = work[k + 1] if k + 1 < len(work) else None
            for j in range(max(nb)):
                inside = j + 1 < max(nb)
                at_v = yield from take_slot()
                at_k = None
                if inside or nxt:
                    at_k = yield from take_slot()
                for i in range(2):
                    if j < nb[i]:
                        n = cp[i]
                        for part in range(2):
                            if "p_full" not in drop:
                                yield ("wait", p_full[i][part], n & 1)

                            def start(i=i, n=n, part=part, at_v=at_v, t=t, j=j):
                                ring[at_v].read_begin(("V", t, j))
                                for h in range(2):
                                    for w in range(rows):
                                        SP[i][h][w][part].read_begin(("P", n))
                                        O[i][h][w].write_begin((n, part))

                            def end(i=i, n=n, part=part, at_v=at_v):
                                ring[at_v].read_end()
                                for h in range(2):
                                    for w in range(rows):
                                        SP[i][h][w][part].read_end()
                                        O[i][h][w].write_end((n, part))
                            tq.op(lat("mma", 0.1, 0.3), start, end)
                            if part == 1 and j == nb[i] - 1:
                                tq.commit(o_full[i])
                        cp[i] += 1
                    if i == 1:
                        tq.commit(empty[at_v])
                    if inside:
                        issue_s(i, at_k, j + 1 < nb[i], j + 2 == nb[i], t, j + 1)
                    elif nxt:
                        yield from first_s(*nxt, i, at_k)

    def softmax(i, h, w):
        role = f"soft{i}"
        n, co = 0, 0
        for t, nb in enumerate(items):
            for j in range(nb[i]):
                yield ("wait", s_full[i], n & 1)
                for part in range(2):
                    SP[i][h][w][part].read_begin(("S", n))
                yield ("sleep", lat(role, 0.05, 0.3))
                for part in range(2):
                    SP[i][h][w][part].read_end()
                MAX[i][h][w].write_begin(n)
                MAX[i][h][w].write_end(n)
                if "pair" not in drop:
                    yield ("barrier", pair[i][w])
                MAX[i][h ^ 1][w].read_begin(n)
                yield ("sleep", lat(role, 0.01, 0.1))
                MAX[i][h ^ 1][w].read_end()
                if j > 0:                                   # O may be rescaled
                    O[i][h][w].read_begin((n - 1, 1))
                    yield ("sleep", lat(role, 0.05, 0.2))
                    O[i][h][w].read_end()
                for part in range(2):
                    yield ("sleep", lat(role, 0.3, 1.0))    # exponentials
                    SP[i][h][w][part].write_begin(("P", n))
                    SP[i][h][w][part].write_end(("P", n))
                    p_full[i][part].arrive()
                n += 1
            if nb[i] > 0:
                if "o_full" not in drop:
                    yield ("wait", o_full[i], co & 1)
                co += 1
            MAX[i][h][w].write_begin(("sum", t))
            MAX[i][h][w].write_end(("sum", t))
            yield ("barrier", pair[i][w])
            MAX[i][h ^ 1][w].read_begin(("sum", t))
            yield ("sleep", lat(role, 0.01, 0.1))
            MAX[i][h ^ 1][w].read_end()
            if "last_pair" not in drop:
                yield ("barrier", pair[i][w])
            if nb[i] > 0:
                O[i][h][w].read_begin((n - 1, 1))
                yield ("sleep", lat(role, 0.2, 0.8))
                O[i][h][w].read_end()
            yield ("sleep", 0.01)

    tasks = [Task(sim, kv_producer(), "kv"), Task(sim, q_producer(), "q"), Task(sim, mma(), "mma")]
    tasks += [Task(sim, softmax(i, h, w), f"soft{i}{h}{w}") for i in range(2) for h in range(2) for w in range(rows)]
    sim.run()
    stuck = [task.name for task in tasks if not task.done]
    assert not stuck, f"items={items} seed={seed}: stuck roles {stuck}"
    for i in range(2):
        assert s_full[i].completed == sum(nb[i] for nb in items)
        assert o_full[i].completed == sum(nb[i] > 0 for nb in items)


LISTS = [[(0, 0)], [(1, 1)], [(1, 0), (1, 1)], [(0, 1), (2, 2), (0, 0), (1, 2)], [(3, 4), (1, 2), (0, 0), (0, 0), (5, 6)],
         [(4, 0), (0, 3), (2, 0), (7, 7)], [(1, 1)] * 7, [(2, 3), (1, 2), (2, 3), (1, 2)], [(9, 10), (0, 0), (8, 1)]]


@pytest.mark.parametrize("items", LISTS)
def test_random_latencies(items):
    for seed in range(40):
        simulate(items, seed)


@pytest.mark.parametrize("role", ["tma", "mma", "soft0", "soft1"])
def test_one_slow_role(role):
    for items in LISTS[3:]:
        for seed in range(8):
            simulate(items, seed, slow={role: 20.0})
            simulate(items, 500 + seed, slow={role: 0.05})


@pytest.mark.parametrize("wait", ["empty", "q_empty", "p_full", "o_full", "pair", "last_pair"])
def test_a_wait_left_out_is_a_hazard(wait):
    """Mutation check of the model: without any one of these waits some schedule overwrites a buffer in use, or reads one
    that is not written."""
    failures = 0
    for seed in range(30):
        for slow in ({}, {"soft0": 8.0}, {"mma": 8.0}, {"tma": 0.05}, {"tma": 8.0}):
            for items in (LISTS[4], LISTS[6]):
                try:
                    simulate(items, seed, slow=slow, drop=(wait,))
                except AssertionError:
                    failures += 1
    assert failures > 0
