"""The barriers of the tensor-core product on the wide form (mmq_wide_k, csrc/q4b_wide_tc.cu), as a model of its roles that runs
on the CPU under random schedules: which accumulator, stage and operand buffer a step of the first CTA's MMA warps takes, what
each role waits for, and by which parity.  Checked at every step: no MMA overwrites an accumulator that has not been read, or
reads a stage or an operand that is not the step's; no adding warp reads an accumulator of another part; none waits for good.

A barrier is waited for by the parity of a phase, so it must never be two phases away from the one that is waited for, to
either side.  Passes of more and of at most 64 rows in every order, tiles of 1, 2 and 4 super-blocks."""
import heapq
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "suzuku-engine-q4_b200", "csrc", "q4b_wide_tc.cu")
NACC, NSB = 4, 8


class Barrier:
    def __init__(self, pair, count):
        self.pair, self.count, self.left, self.phase, self.waiting = pair, count, count, 0, []

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1
            waiting, self.waiting = self.waiting, []
            for role, parity in waiting:
                self.wait(role, parity)

    def wait(self, role, parity):
        if (self.phase & 1) != parity:
            self.pair.after(role, 0)
        else:
            self.waiting.append((role, parity))


class Queue:
    def __init__(self, pair):
        self.pair, self.ops, self.waiting = pair, [], []

    def put(self, op):
        self.ops.append(op)
        while self.waiting:
            self.pair.after(self.waiting.pop(), 0)

    def wait(self, role, _):
        if self.ops:
            self.pair.after(role, 0)
        else:
            self.waiting.append(role)


class Pair:
    """One pair of CTAs: items (rows) of `mt` tiles of `n_it` steps.  A role is a generator that yields (barrier, parity)
    or (queue, None) to wait, or a time to let pass.  Of warps with the same task one stands for all."""

    def __init__(self, items, n_it, mt, rng):
        self.items, self.n_it, self.mt, self.rng = items, n_it, mt, rng
        bars = lambda n, count: [Barrier(self, count) for _ in range(n)]
        self.a_full = [bars(2, 2), bars(2, 1)]
        self.a_free, self.done, self.b_full = [[bars(n, 1) for _ in range(2)] for n in (4, NSB, NSB)]
        self.sums = [[bars(NACC, 1) for _ in range(2)] for _ in range(2)]
        self.acc_empty = bars(NACC, 2)
        self.stage = [[None] * NSB, [None] * NSB]            # part that has landed
        self.operand = [[None] * 4, [None] * 4]              # step that has been decoded
        self.d = [[None] * 8, [None] * 8]                    # super-block whose d is there
        self.acc = [None] * NACC                             # [part, its MMAs are complete]
        self.read = {}                                       # part: CTAs that have read it
        self.pipe = [Queue(self), Queue(self)]               # MMAs and commits on their way, by issuing warp
        self.loads = [Queue(self), Queue(self)]

    def tiles(self):
        for rows in self.items:
            for _ in range(self.mt):
                yield 2 if rows > 64 else 1

    # ---- the roles ----
    def tell(self):
        u = j = 0
        for parts in self.tiles():
            for _ in range(0, self.n_it, 2):
                for _ in range(2 * parts):
                    yield self.b_full[1][u % NSB], (u // NSB) & 1
                    u += 1
                yield self.a_full[1][(j >> 1) & 1], (j >> 2) & 1
                self.a_full[0][(j >> 1) & 1].arrive()
                j += 2

    def issue(self, w):
        u, v, j, tile = 0, 0, w, 0
        for parts in self.tiles():
            u += w * parts
            for k in range(w, self.n_it, 2):
                yield self.a_full[0][(j >> 1) & 1], (j >> 2) & 1
                for p in range(parts):
                    acc = 2 * w + (v & 1)
                    if v >= 2:
                        yield self.acc_empty[acc], (v // 2 - 1) & 1
                    yield self.b_full[0][u % NSB], (u // NSB) & 1
                    last = self.acc[acc]
                    assert last is None or self.read.get(last[0]) == 2, "an accumulator is overwritten before it is read"
                    self.acc[acc] = [u, False]
                    self.pipe[w].put((acc, u, j))
                    s = p if parts == 2 else tile & 1
                    self.pipe[w].put([self.done[r][u % NSB] for r in (0, 1)] + [self.sums[r][s][acc] for r in (0, 1)])
                    u, v = u + 1, v + 1
                self.pipe[w].put([self.a_free[r][j & 3] for r in (0, 1)])
                j += 2
                u += parts
            u -= w * parts
            tile += 1

    def tensor(self, w):
        """The MMAs of an issuing warp, in order, each after some time."""
        while True:
            yield self.pipe[w], None
            op = self.pipe[w].ops.pop(0)
            if isinstance(op, list):
                for b in op:
                    b.arrive()
                continue
            acc, u, j = op
            for _ in range(2):
                for r in (0, 1):
                    assert self.stage[r][u % NSB] == u, "activations of another part"
                    assert self.operand[r][j & 3] == j, "weights of another step"
                yield 1.0
            assert self.acc[acc][0] == u
            self.acc[acc][1] = True

    def copy(self, r):
        u = 0
        for parts in self.tiles():
            for _ in range(self.n_it * parts):
                if u >= NSB:
                    yield self.done[r][u % NSB], (u // NSB - 1) & 1
                self.stage[r][u % NSB] = None
                self.loads[r].put(u)
                u += 1

    def land(self, r):
        while True:
            yield self.loads[r], None
            u = self.loads[r].ops.pop(self.rng.randrange(len(self.loads[r].ops)))
            self.stage[r][u % NSB] = u
            self.b_full[r][u % NSB].arrive()

    def decode(self, r):
        g = 0
        for _ in self.tiles():
            for _ in range(0, self.n_it, 2):
                self.d[r][g & 7] = g
                for h in (0, 1):
                    if g >= 2:
                        yield self.a_free[r][2 * (g & 1) + h], (g // 2 - 1) & 1
                    self.operand[r][2 * (g & 1) + h] = 2 * g + h
                    yield 1.0
                self.a_full[r][g & 1].arrive()
                g += 1

    def add(self, r, s):
        v = j = tile = seen = first = 0                      # (first, u: which part it is, for the checks alone)
        for parts in self.tiles():
            v0, u = v + (s if parts == 2 else 0), first + (s if parts == 2 else 0)
            v, first = v + self.n_it // 2 * parts, first + self.n_it * parts
            if parts == 1 and (tile & 1) != s:
                j += self.n_it
            else:
                for k in range(self.n_it):
                    acc = 2 * (k & 1) + ((v0 + (k >> 1) * parts) & 1)
                    yield self.sums[r][s][acc], (seen >> acc) & 1
                    seen ^= 1 << acc
                    assert self.acc[acc] == [u, True], "an accumulator of another part is read"
                    assert self.d[r][(j >> 1) & 7] == j >> 1, "d of another super-block"
                    yield 1.0
                    assert self.acc[acc] == [u, True], "an accumulator is overwritten while it is read"
                    self.read[u] = self.read.get(u, 0) + 1
                    self.acc_empty[acc].arrive()
                    u, j = u + parts, j + 1
                    if self.rng.random() < 0.05:
                        yield 30.0
                yield 30.0                                   # a finished tile is stored
            tile += 1

    # ---- time ----
    def after(self, role, t):
        """A role goes on after about a time, longer for one that is slow in this run."""
        heapq.heappush(self.events, (self.now + (t + 0.2) * role[1] * 2.0 * self.rng.random(), next(self.order), role))

    def run(self):
        two, speeds = (0, 1), (0.3, 1.0, 1.0, 4.0)
        ends = [self.tell(), self.issue(0), self.issue(1)] + [self.add(r, s) for r in two for s in two]
        ends += [f(r) for f in (self.copy, self.decode) for r in two]
        self.now, self.events, self.order, left = 0.0, [], iter(range(1 << 30)), len(ends)
        for g in ends + [f(i) for f in (self.tensor, self.land) for i in two]:
            self.after((g, self.rng.choice(speeds)), 0)
        while self.events:
            self.now, _, role = heapq.heappop(self.events)
            try:
                to = next(role[0])
            except StopIteration:
                left -= 1
                continue
            if isinstance(to, float):
                self.after(role, to)
            else:
                to[0].wait(role, to[1])
        assert left == 0, "a role waits for good"


SHAPES = {"a super-block, one tile": (2, 1), "a super-block, three tiles": (2, 3), "two super-blocks": (4, 1), "two, two tiles": (4, 2),
          "four super-blocks": (8, 1)}


@pytest.mark.parametrize("shape", SHAPES)
def test_no_schedule_breaks_the_order_of_the_barriers(shape):
    n_it, mt = SHAPES[shape]
    for seed in range(200):
        rng = random.Random("%s %d" % (shape, seed))
        Pair([rng.choice((32, 128)) for _ in range(max(6, 32 // (n_it * mt)))], n_it, mt, rng).run()


def test_the_model_has_the_rules_of_the_kernel():
    """The lines that the model restates: a change to one of them is a change to the model too."""
    text = re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", open(SRC).read()))
    for line in ("wait(&s.b_full[u % W_NSB], (u / W_NSB) & 1u, 1u)",
                 "wait(&s.a_full[(j >> 1) & 1u], (j >> 2) & 1u, 1u)",
                 "wait(&s.b_full[sb], (u / W_NSB) & 1u, 1u)",
                 "const uint32_t acc = 2u * (warp & 1u) + (v & 1u); if (v >= 2u) wait(&s.acc_empty[acc], (v / 2u - 1u) & 1u, 4u);",
                 "const uint32_t v0 = v + (parts == 2u ? set : 0u); v += n_it / 2u * parts;",
                 "const uint32_t acc = 2u * (k & 1u) + ((v0 + (k >> 1) * parts) & 1u); wait(&s.sums[set][acc], (seen >> acc) & 1u, 32u);",
                 "mma_commit2(&s.done[sb]); mma_commit2(&s.sums[parts == 2u ? p : tile & 1u][acc]);",
                 "mma_commit2(&s.a_free[j & 3u])",
                 "if (u >= W_NSB) wait(&s.done[sb], (u / W_NSB - 1u) & 1u, 16u)",
                 "wait(&s.sums[set][acc], (seen >> acc) & 1u, 32u); seen ^= 1u << acc;",
                 "if (g >= 2u) wait(&s.a_free[2u * (g & 1u) + h], (g / 2u - 1u) & 1u, 2u)",
                 "W_NSB = %d;" % NSB, "W_HB = 64;", "W_A_COL = 256;", "W_NACC = W_A_COL / W_HB;"):
        assert line in text, line
