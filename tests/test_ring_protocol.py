"""A model of the barrier protocol of the tcgen05 prompt attention (csrc/attn_prompt_tc.cu),
run on the host with mbarrier semantics: a barrier completes a phase when its arrivals and
its bytes are in, and a wait names the PARITY of the phase it waits for, so a barrier that is
two phases on cannot be told from one that has not moved.  This is reasoning kept runnable, not
a test of the kernel: the kernel itself is held against the plain attention in
tests/test_gpu_kernels.py."""
import random

import pytest


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.tx, self.phase = count, count, 0, 0

    def arrive(self, tx=0):
        self.tx += tx
        self.pending -= 1
        assert self.pending >= 0, "more arrivals than the barrier expects"
        self._check()

    def complete_tx(self, n):
        self.tx -= n
        self._check()

    def _check(self):
        if self.pending == 0 and self.tx == 0:
            self.phase ^= 1
            self.pending = self.count

    def done(self, parity):                 # mbarrier.try_wait.parity
        return self.phase != parity


# ---------------------------------------------------------------------------
# The ring that the tcgen05 prompt attention had before its blocks took two streams (kept for what it shows
# about parities): a producer (keys and
# values of block j into one of six tiles), an issuing thread (scores of up to three blocks
# ahead, then P V block by block) and the softmax warps.  The producer may fetch the values of
# block j only when the product of block j - 3 has read its tile.  If it learns that from the
# barrier that alternate blocks share (pv_done[j & 1]), the barrier can be two phases on by
# the time a late producer looks, once the last scores are issued and nothing holds the last
# products back; with a barrier per tile (v_free[j % 3]) the next phase always needs the tile
# that the producer fetches after its wait.
def simulate_prompt_ring(n_blk, seed, per_tile, producer_lag):
    rnd = random.Random(seed)
    NBUF = 3
    full = [Barrier(1) for _ in range(6)]
    s_full, p_full = [Barrier(1) for _ in range(NBUF)], [Barrier(1) for _ in range(NBUF)]
    pv_done, v_free = [Barrier(1) for _ in range(2)], [Barrier(1) for _ in range(NBUF)]
    tiles = [None] * 6
    inflight = []                                             # tensor-core work and copies complete later, in order

    def producer():
        for i in range(2 * n_blk):
            slot, j, is_v = i % 6, i >> 1, i & 1
            for _ in range(producer_lag if i == 2 * n_blk - 1 else 0):
                yield                                         # the producer is late for the last tile
            if j >= NBUF:
                jp = j - NBUF
                if is_v:
                    bar, par = (v_free[jp % NBUF], (jp // NBUF) & 1) if per_tile else (pv_done[jp & 1], (jp >> 1) & 1)
                else:
                    bar, par = s_full[jp % NBUF], (jp // NBUF) & 1
                while not bar.done(par):
                    yield
            full[slot].arrive(tx=1)
            inflight.append(("copy", slot, (j, is_v)))
            yield

    def issuer():
        def issue_s(j):
            i = 2 * j
            while not full[i % 6].done((i // 6) & 1):
                yield
            assert tiles[i % 6] == (j, 0), f"scores of block {j} read tile {tiles[i % 6]}"
            inflight.append(("mma", [s_full[j % NBUF]], None))
        for j in range(min(NBUF, n_blk)):
            yield from issue_s(j)
        for j in range(n_blk):
            i = 2 * j + 1
            while not (p_full[j % NBUF].done((j // NBUF) & 1) and full[i % 6].done((i // 6) & 1)):
                yield
            assert tiles[i % 6] == (j, 1), f"product of block {j} read tile {tiles[i % 6]}"
            inflight.append(("mma", [pv_done[j & 1], v_free[j % NBUF]], None))
            if j + NBUF < n_blk:
                while not pv_done[j & 1].done((j >> 1) & 1):
                    yield
                yield from issue_s(j + NBUF)
            yield

    def softmax():
        for j in range(n_blk):
            while not s_full[j % NBUF].done((j // NBUF) & 1):
                yield
            yield
            p_full[j % NBUF].arrive()
        for j in (n_blk - 2, n_blk - 1):
            if j >= 0:
                while not pv_done[j & 1].done((j >> 1) & 1):
                    yield

    threads = [producer(), issuer(), softmax()]
    alive, idle = [0, 1, 2], 0
    while alive:
        if inflight and rnd.random() < 0.4:
            kind, a, b = inflight.pop(0)
            if kind == "copy":
                tiles[a] = b
                full[a].complete_tx(1)
            else:
                for bar in a:
                    bar.arrive()
            idle = 0
            continue
        t = rnd.choice(alive)
        try:
            next(threads[t])
        except StopIteration:
            alive.remove(t)
            idle = 0
            continue
        idle += 1
        assert idle < 20000 or inflight, "nothing moves"


@pytest.mark.parametrize("n_blk", [1, 2, 3, 4, 5, 6, 7, 16, 33])
def test_prompt_attention_ring_with_a_barrier_per_value_tile_always_finishes(n_blk):
    for seed in range(30):
        for lag in (0, 50, 3000):
            simulate_prompt_ring(n_blk, seed, per_tile=True, producer_lag=lag)


def test_prompt_attention_ring_on_the_shared_product_barrier_can_stall_a_late_producer():
    stalled = 0
    for seed in range(30):
        try:
            simulate_prompt_ring(9, seed, per_tile=False, producer_lag=3000)
        except AssertionError:
            stalled += 1
    assert stalled > 0


# ---------------------------------------------------------------------------
# The protocol of csrc/attn_prompt_tc.cu: a block works through its items one behind the other; five tiles, two streams of
# scores, and for each item either two tiles of rows over all key blocks or (split) one tile whose even and odd key blocks are
# a stream each, joined at the end.  Tensor-core instructions complete in order; copies complete in any order.
def simulate_two_streams(items, seed):
    """items: (key blocks, split) of each."""
    rnd = random.Random(seed)
    NSLOT, WARPS = 5, 2                                               # (two softmax warps a stream instead of four)
    full, empty = [Barrier(1) for _ in range(NSLOT)], [Barrier(1) for _ in range(NSLOT)]
    s_full, o_full = ([Barrier(1) for _ in range(2)] for _ in range(2))
    p_first, p_full, o_empty = ([Barrier(WARPS) for _ in range(2)] for _ in range(3))
    q_full, q_empty, join, joined = Barrier(1), Barrier(1), Barrier(2 * WARPS), Barrier(2 * WARPS)
    tiles, mma, copies = [None] * NSLOT, [], []
    state = dict(q=None)
    scores, result = [None, None], [None, None]                       # what S and O of each stream hold: (item, step)
    first, probs = [{}, {}], [{}, {}]                                 # (item, step) -> warps that have written P
    read = [dict(), dict()]                                           # item -> warps that have read O

    def place_k(n_blk, split, j):
        return max(2 * j - 1, 0) if split else 2 * j

    def place_v(n_blk, split, j):
        return min(2 * j + 2, 2 * n_blk - 1) if split else 2 * j + 1

    def block_of(split, s, t):
        return 2 * t + s if split else t

    def wait(bar, parity):
        while not bar.done(parity):
            yield

    def producer():
        base = 0
        for k, (n_blk, split) in enumerate(items):
            if k:
                yield from wait(q_empty, (k - 1) & 1)
            q_full.arrive(tx=1)
            copies.append(lambda k=k: (state.update(q=k), q_full.complete_tx(1)))
            for i in range(2 * n_blk):
                last = split and i == 2 * n_blk - 1
                is_v = (last or (i > 0 and not i & 1)) if split else bool(i & 1)
                j = n_blk - 1 if last else (((i - 2) >> 1 if is_v else (i + 1) >> 1) if split else i >> 1)
                assert i == (place_v if is_v else place_k)(n_blk, split, j)
                n = base + i
                if n >= NSLOT:
                    yield from wait(empty[n % NSLOT], (n // NSLOT - 1) & 1)
                full[n % NSLOT].arrive(tx=1)

                def land(n=n, what=(k, j, is_v)):
                    tiles[n % NSLOT] = what
                    full[n % NSLOT].complete_tx(1)
                copies.append(land)
                yield
            base += 2 * n_blk

    def issuer():
        base, steps, uses = 0, [0, 0], [0, 0]
        for k, (n_blk, split) in enumerate(items):
            def release(n, s):
                if split or s == 1:
                    mma.append(lambda: empty[n % NSLOT].arrive())

            def keys_here(s, t):
                j = block_of(split, s, t)
                if (split or s == 0) and j < n_blk:
                    n = base + place_k(n_blk, split, j)
                    yield from wait(full[n % NSLOT], (n // NSLOT) & 1)

            def issue_s(s, t):
                j = block_of(split, s, t)
                n = base + place_k(n_blk, split, j)
                yield from keys_here(s, t)

                def run():
                    assert tiles[n % NSLOT] == (k, j, False) and state["q"] == k
                    assert t == 0 or result[s] == (k, t - 1), "scores over probabilities that are not multiplied yet"
                    scores[s] = (k, t)
                    s_full[s].arrive()
                mma.append(run)
                release(n, s)
                if j == n_blk - 1 and (split or s == 1):
                    mma.append(lambda: q_empty.arrive())
            yield from wait(q_full, k & 1)
            for s in range(2):
                if block_of(split, s, 0) < n_blk:
                    yield from issue_s(s, 0)
            t = 0
            while block_of(split, 0, t) < n_blk:
                for s in range(2):
                    j = block_of(split, s, t)
                    if j >= n_blk:
                        break
                    n = base + place_v(n_blk, split, j)
                    if t == 0 and uses[s]:
                        yield from wait(o_empty[s], (uses[s] - 1) & 1)
                    if split or s == 0:
                        yield from wait(full[n % NSLOT], (n // NSLOT) & 1)
                    yield from wait(p_first[s], steps[s] & 1)

                    def begin(n=n, j=j, s=s, t=t, k=k, split=split):  # the product of the first keys
                        assert tiles[n % NSLOT] == (k, j, True) and first[s].get((k, t)) == WARPS
                        if t == 0 and result[s] is not None:          # the result before has been read by all who read it
                            kb = result[s][0]
                            nb, sb = items[kb]
                            assert read[s].get(kb) == (2 * WARPS if sb and nb > 1 else WARPS), "a result overwritten unread"
                    mma.append(begin)
                    yield from wait(p_full[s], steps[s] & 1)

                    def run(n=n, j=j, s=s, t=t, k=k):
                        assert tiles[n % NSLOT] == (k, j, True) and probs[s].get((k, t)) == WARPS
                        result[s] = (k, t)
                    mma.append(run)
                    release(n, s)
                    steps[s] += 1
                    if block_of(split, s, t + 1) < n_blk:
                        yield from issue_s(s, t + 1)
                    else:
                        mma.append(lambda s=s: o_full[s].arrive())
                        uses[s] += 1
                    yield
                t += 1
            base += 2 * n_blk

    def softmax(s):
        base, step, uses, joins = 0, 0, [0, 0], 0
        for k, (n_blk, split) in enumerate(items):
            ragged = k % 2 == 0
            t = 0
            while block_of(split, s, t) < n_blk:
                yield from wait(s_full[s], step & 1)
                step += 1
                assert scores[s] == (k, t) and (t == 0 or result[s] == (k, t - 1))   # (the result may be rescaled here)
                yield
                if ragged and block_of(split, s, t) == n_blk - 1 and (split or s == 0):
                    n = base + place_v(n_blk, split, n_blk - 1)       # the last values' rows beyond the end are zeroed
                    yield from wait(full[n % NSLOT], (n // NSLOT) & 1)
                    assert tiles[n % NSLOT] == (k, n_blk - 1, True)
                first[s][k, t] = first[s].get((k, t), 0) + 1
                p_first[s].arrive()
                yield
                probs[s][k, t] = probs[s].get((k, t), 0) + 1
                p_full[s].arrive()
                t += 1
            base += 2 * n_blk
            if not split or n_blk == 1:
                if not split or s == 0:
                    yield from wait(o_full[s], uses[s] & 1)
                    assert result[s] == (k, t - 1)
                    read[s][k] = read[s].get(k, 0) + 1
                    o_empty[s].arrive()
                uses[0] += 1
                uses[1] += 0 if split else 1
            else:
                yield from wait(o_full[0], uses[0] & 1)
                yield from wait(o_full[1], uses[1] & 1)
                uses = [u + 1 for u in uses]
                join.arrive()
                yield from wait(join, joins & 1)
                for i in range(2):
                    assert result[i] == (k, (n_blk + 1 - i) // 2 - 1)
                    read[i][k] = read[i].get(k, 0) + 1
                joined.arrive()
                yield from wait(joined, joins & 1)
                joins += 1
                o_empty[s].arrive()
            yield

    threads = [producer(), issuer()] + [softmax(w % 2) for w in range(2 * WARPS)]
    speed = [rnd.choice([1, 1, 5, 25]) for _ in threads]              # (some are late)
    alive, idle = list(range(len(threads))), 0
    while alive:
        if mma and rnd.random() < 0.4:
            mma.pop(0)()
            idle = 0
        elif copies and rnd.random() < 0.4:
            copies.pop(rnd.randrange(len(copies)))()
            idle = 0
        else:
            t = rnd.choices(alive, [1 / speed[i] for i in alive])[0]
            try:
                next(threads[t])
            except StopIteration:
                alive.remove(t)
                idle = 0
            idle += 1
            assert idle < 40000 or mma or copies, "nothing moves"


@pytest.mark.parametrize("n_blk", [1, 2, 3, 4, 5, 6, 7, 16, 33])
@pytest.mark.parametrize("split", [False, True])
def test_prompt_attention_of_two_streams_always_finishes(n_blk, split):
    for seed in range(10):
        simulate_two_streams([(n_blk, split)], seed)
        simulate_two_streams([(n_blk, split), (1, not split), (n_blk, not split)], seed)


def test_prompt_attention_of_two_streams_item_behind_item():
    for seed in range(60):
        rnd = random.Random(seed)
        simulate_two_streams([(rnd.choice([1, 1, 2, 3, 5, 8]), rnd.random() < 0.5) for _ in range(rnd.randint(2, 9))], seed)
