"""CPU model of the dense packed kernel's synchronisation (tk_pack.cu, k_ntt_packed):
a load thread, a store thread, two MMA issuers, four unpack warps and 16 epilogue
warps, exchanging through mbarriers with the kernel's counts and parities, under
random interleavings and random completion delays of the TMA loads, the stores'
reads and the MMAs, for both layouts (2 or 3 input slots, 3 or 2 output slots).
Every run completes, no wait's phase is lapped, and each shared resource is written
only after its readers are done: input slots, operand buffers, accumulators, output
slots."""
import random

import pytest

from test_tc5_protocol import Bar

UNPACK, EPI, ISSUERS = 4, 16, 2


class Sim:
    def __init__(self, ntiles, in_slots, out_slots, seed, skip=None):
        self.rng, self.n, self.S, self.NO, self.skip = (random.Random(seed), ntiles, in_slots,
                                                        out_slots, skip)
        # how fast threads, loads, store reads and MMAs go, another mix in every run
        self.speed = [self.rng.choice([1, 8, 64]) for _ in range(4)]
        self.in_full = [Bar(1) for _ in range(in_slots)]
        self.in_empty = [Bar(UNPACK) for _ in range(in_slots)]
        self.x_ready, self.op_free = [Bar(UNPACK) for _ in range(2)], [Bar(ISSUERS) for _ in range(2)]
        self.d_full, self.d_empty, self.drain = Bar(ISSUERS), Bar(EPI), Bar(ISSUERS)
        self.out_ready = [[Bar(4) for _ in range(4)] for _ in range(out_slots)]
        self.out_free = [Bar(1) for _ in range(out_slots)]
        self.loads, self.reads, self.mma = [], [], [[] for _ in range(ISSUERS)]
        self.slot = [None] * in_slots            # tile in it; None while being loaded
        self.in_reads = {}                       # tile -> unpack warps that read it
        self.op = [[None, 0], [None, 0]]         # operand buffer: tile, warps that wrote it
        self.op_reading = [0, 0]                 # MMAs in flight on it
        self.sums = {}                           # tile -> issuers whose MMAs completed
        self.sum_reads = {}                      # tile -> epilogue warps that read its sums
        self.out_writes = {}                     # (tile, quarter) -> warps that wrote it
        self.out_reading = {}                    # (tile, quarter) -> store still reading
        self.stored = []

    def wait(self, bar, phase, name):
        return (lambda: True) if name == self.skip else (lambda: bar.ready(phase & 1, phase))

    def loader(self):
        for k in range(self.n):
            s = k % self.S
            if k >= self.S:
                yield self.wait(self.in_empty[s], k // self.S - 1, "in_empty")
                assert self.in_reads.get(k - self.S, 0) == UNPACK, "input overwritten unread"
            self.slot[s] = None

            def land(s=s, k=k):
                self.slot[s] = k
                self.in_full[s].arrive()
            self.loads.append(land)
        for j in range(max(0, self.n - self.S), self.n):
            yield self.wait(self.in_full[j % self.S], j // self.S, "")

    def storer(self):
        order = []                               # store groups, oldest first
        for k in range(self.n):
            b = k % self.NO
            for g in range(4):
                yield self.wait(self.out_ready[b][g], k // self.NO, "out_ready")
                assert self.out_writes.get((k, g), 0) == 4, "stored before written"
                self.out_reading[k, g] = True
                order.append((k, g))
                self.reads.append(lambda key=(k, g): self.out_reading.update({key: False}))
            if k >= self.NO - 1:
                old = order[:len(order) - 4 * (self.NO - 1)]
                yield lambda old=old: not any(self.out_reading[o] for o in old)
                self.out_free[(k + 1) % self.NO].arrive()
            self.stored.append(k)

    def issuer(self, j):
        for k in range(self.n):
            b = k & 1
            yield self.wait(self.x_ready[b], k >> 1, "x_ready")
            if k >= 1:
                yield self.wait(self.d_empty, k - 1, "d_empty")
                assert self.sum_reads.get(k - 1, 0) == EPI, "sums overwritten unread"
            assert self.op[b] == [k, UNPACK], "multiplied before unpacked"
            self.op_reading[b] += 1
            self.mma[j] += [("mma", b, k), ("commit", self.d_full), ("commit", self.op_free[b])]
        self.mma[j].append(("commit", self.drain))
        yield self.wait(self.drain, 0, "")

    def unpack(self, w):
        for t in range(self.n):
            s, b = t % self.S, t & 1
            yield self.wait(self.in_full[s], t // self.S, "in_full")
            assert self.slot[s] == t, "unpacked before loaded"
            self.in_reads[t] = self.in_reads.get(t, 0) + 1
            self.in_empty[s].arrive()
            if t >= 2:
                yield self.wait(self.op_free[b], (t >> 1) - 1, "op_free")
            assert self.op_reading[b] == 0, "operand overwritten in use"
            if self.op[b][0] != t:
                assert t < 2 or self.op[b][0] == t - 2
                self.op[b] = [t, 0]
            self.op[b][1] += 1
            self.x_ready[b].arrive()

    def epilogue(self, w):
        g = w >> 2
        for k in range(self.n):
            b = k % self.NO
            if k >= self.NO:
                yield self.wait(self.out_free[b], k // self.NO - 1, "out_free")
            yield self.wait(self.d_full, k, "d_full")
            assert self.sums.get(k, 0) == ISSUERS, "sums read before complete"
            self.sum_reads[k] = self.sum_reads.get(k, 0) + 1
            self.d_empty.arrive()
            yield lambda: True
            assert not self.out_reading.get((k - self.NO, g), k >= self.NO), "output overwritten"
            self.out_writes[k, g] = self.out_writes.get((k, g), 0) + 1
            self.out_ready[b][g].arrive()

    def step_mma(self, queue):
        op = queue.pop(0)
        if op[0] == "commit":
            op[1].arrive()
        else:
            self.op_reading[op[1]] -= 1
            self.sums[op[2]] = self.sums.get(op[2], 0) + 1

    def run(self):
        agents = [self.loader(), self.storer()] + [self.issuer(j) for j in range(ISSUERS)] + \
            [self.unpack(w) for w in range(UNPACK)] + [self.epilogue(w) for w in range(EPI)]
        waiting = {i: next(a, None) for i, a in enumerate(agents)}
        waiting = {i: w for i, w in waiting.items() if w}
        while waiting or self.loads or self.reads or any(self.mma):
            ready = [i for i, w in waiting.items() if w()]
            work = [ready, self.loads, self.reads, [q for q in self.mma if q]]
            assert any(work), "deadlock"
            kind = self.rng.choices(range(4), [s if w else 0 for s, w in zip(self.speed, work)])[0]
            pick = self.rng.randrange(len(work[kind]))
            if kind == 0:
                i = ready[pick]
                waiting[i] = next(agents[i], None)
                if waiting[i] is None:
                    del waiting[i]
            elif kind < 3:
                work[kind].pop(pick)()
            else:
                self.step_mma(work[3][pick])
        assert self.stored == list(range(self.n))


@pytest.mark.parametrize("slots", [(2, 3), (3, 2)], ids=["2-bit", "3-bit"])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 5, 8, 15])
def test_protocol_random_interleavings(slots, ntiles):
    for seed in range(16):
        Sim(ntiles, *slots, 100 * ntiles + seed).run()


@pytest.mark.parametrize("skip", ["in_empty", "in_full", "x_ready", "op_free", "d_empty", "d_full",
                                  "out_ready", "out_free"])
def test_every_wait_is_needed(skip):
    """The checker itself: with any one wait left out some run breaks a rule."""
    with pytest.raises(AssertionError):
        for seed in range(50):
            Sim(15, 2, 3, seed, skip).run()
