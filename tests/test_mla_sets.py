"""The waits of the sparse MLA kernel with its two softmax sets, which take chunks in turn, its two MMA issuers and the exchange of
partial scores between the two CTAs of a pair: in every order in which the roles of one CTA can run, and in random orders of a pair.
A wait names the parity of a barrier's phase, and must neither pass before what it waits for nor miss it."""
import itertools
import random

import pytest

from umdk_b200 import _native

S, P, O, END, READ, FREE, MAX = range(7)
XFULL, XFREE, PFULL, PFREE = range(7, 11)   # barriers of the exchange, each two in turn


def kernel_wait(step, c):
    """(barrier, parity) of a wait, as the kernel has it; the exchange's barriers stand behind the others."""
    if step >= XFULL:
        return 20 + 2 * (step - XFULL) + (c & 1), (c >> 1) & 1
    w = _native.cam().umdk_sparse_mla_wait(step, c)
    assert w >= 0
    return w >> 1, w & 1


BARS = 28


def programs(n, rescaled, groups, ctas):
    """Roles of a CTA: lists of ("wait", step, c), ("arrive", step, c, cta), ("mma", step, c). `groups`: warps of a set (and of those
    that take the partner's P in)."""
    out = []
    for cta in range(ctas):
        qk, pv, exchange = [], [], []
        for c in range(n):
            qk += ([("wait", READ, c - 1)] if c else []) + [("mma", S, c)]
            pv += ([("wait", O, c - 1), ("arrive", FREE, c - 1, cta)] if c else []) + [("wait", P, c), ("mma", O, c)]
            exchange += [("wait", S, c), ("arrive", READ, c, cta)]
            if ctas == 2:
                exchange += [("wait", XFREE, c - 2)] if c >= 2 else []
                exchange += [("arrive", XFULL, c, 1 - cta)]
        qk, pv = qk + [("mma", END, 0)], pv + [("mma", END, 0)]
        out += [(cta, 0, qk), (cta, 1, pv), (cta, None, exchange)]
        rescale = lambda c: [("wait", O, c - 1)] if c in rescaled else []
        free = lambda c: [("wait", FREE, c - 2)] if c >= 2 else []
        for g in range(groups):
            taken = []
            for c in range(n):
                taken += [("wait", PFULL, c)] if ctas == 2 else []
                taken += free(c) + rescale(c) if ctas == 1 else free(c) + rescale(c) + [("arrive", PFREE, c, 1 - cta)]
                taken += [("arrive", P, c, cta)]
            out.append((cta, None, taken))
        for s, g in itertools.product(range(2), range(groups)):
            soft = []
            for c in range(s, n, 2):
                soft += [("wait", S, c), ("arrive", READ, c, cta)]
                soft += [("wait", XFULL, c), ("arrive", XFREE, c, 1 - cta)] if ctas == 2 else []
                soft += ([("wait", MAX, c - 1, g)] if c else []) + [("arrive", MAX, c, cta, g)]
                if ctas == 2:
                    soft += ([("wait", PFREE, c - 2)] if c >= 2 else []) + [("arrive", PFULL, c, 1 - cta)]
                soft += free(c) + rescale(c) + [("arrive", P, c, cta)]
            out.append((cta, None, soft + [("wait", END, 0)]))
    return out


class Walk:
    def __init__(self, n, rescaled, groups=1, ctas=1, wait=kernel_wait):
        self.n, self.wait, self.groups = n, wait, groups
        self.roles = programs(n, rescaled, groups, ctas)
        self.progs = [p for _, _, p in self.roles]
        self.queues = sorted({(cta, q) for cta, q, _ in self.roles if q is not None})
        self.mmas = {(cta, q): [op for op in p if op[0] == "mma"] for cta, q, p in self.roles if q is not None}
        self.counts = {P: 2 * groups, READ: groups + 1, END: 2, XFREE: groups, PFULL: groups, PFREE: groups}
        z = len(self.progs)
        self.start = ((0,) * z, (0,) * len(self.queues), tuple((0, 0) for _ in range(ctas * BARS + ctas * 4)))
        # every arrival that a step of chunk c needs, to tell whether it has happened: (role, place) or (queue, place)
        self.needs = {}
        for r, (cta, q, p) in enumerate(self.roles):
            for i, op in enumerate(p):
                if op[0] == "arrive":
                    self.needs.setdefault((op[3], op[1], op[2], op[4:] or (0,)), []).append(("pc", r, i))
        for qi, key in enumerate(self.queues):
            for i, op in enumerate(self.mmas[key]):
                if op[1] == O and op[2] == n - 1:
                    continue   # no commit behind the last product but the final one
                self.needs.setdefault((key[0], op[1], op[2], (0,)), []).append(("done", qi, i))

    def slot(self, cta, step, c, g):
        bar, parity = self.wait(step, c)
        return (cta * BARS + bar + (g if step == MAX else 0)), parity

    def arrive(self, bars, cta, step, c, g=0):
        at, _ = self.slot(cta, step, c, g)
        phase, count = bars[at]
        count += 1
        if count == self.counts.get(step, 1):
            phase, count = phase + 1, 0
        return bars[:at] + ((phase, count),) + bars[at + 1:]

    def happened(self, state, cta, step, c, g):
        pcs, done, _ = state
        return all(pcs[a] > i if kind == "pc" else done[a] > i for kind, a, i in self.needs[cta, step, c, (g,)])

    def moves(self, state):
        """(next states, faults)"""
        pcs, done, bars = state
        nexts, faults = [], set()
        for qi, key in enumerate(self.queues):
            r = next(i for i, (cta, q, _) in enumerate(self.roles) if (cta, q) == key)
            queued = sum(op[0] == "mma" for op in self.progs[r][:pcs[r]])
            if done[qi] < queued:
                op = self.mmas[key][done[qi]]
                d = done[:qi] + (done[qi] + 1,) + done[qi + 1:]
                last = op[1] == O and op[2] == self.n - 1
                nexts.append((pcs, d, bars if last else self.arrive(bars, key[0], op[1], op[2])))
        for r, (cta, _, prog) in enumerate(self.roles):
            if pcs[r] == len(prog):
                continue
            op = prog[pcs[r]]
            on = pcs[:r] + (pcs[r] + 1,) + pcs[r + 1:]
            if op[0] == "mma":
                nexts.append((on, done, bars))
            elif op[0] == "arrive":
                nexts.append((on, done, self.arrive(bars, op[3], op[1], op[2], *op[4:])))
            else:
                g = op[3] if len(op) > 3 else 0
                at, parity = self.slot(cta, op[1], op[2], g)
                if bars[at][0] & 1 != parity:
                    if self.happened(state, cta, op[1], op[2], g):
                        nexts.append((on, done, bars))
                    else:
                        faults.add(("early", op[1]))
        if not nexts and not faults and any(pc < len(p) for pc, p in zip(pcs, self.progs)):
            faults.add(("stuck",))
        return nexts, faults

    def all_orders(self):
        found, seen, todo = set(), set(), [self.start]
        while todo:
            state = todo.pop()
            if state in seen:
                continue
            seen.add(state)
            nexts, faults = self.moves(state)
            found |= faults
            todo += nexts
        return found

    def random_order(self, rng):
        state = self.start
        while True:
            nexts, faults = self.moves(state)
            if faults or not nexts:
                return faults
            # now and then the first moves again and again: one role far ahead of the others
            state = nexts[0] if rng.random() < 0.3 else nexts[-1] if rng.random() < 0.3 else rng.choice(nexts)


def patterns(n):
    return [set(p) for k in range(n) for p in itertools.combinations(range(1, n), k)]


@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_every_order_of_one_cta(n):
    for rescaled in patterns(n):
        assert Walk(n, rescaled).all_orders() == set(), rescaled


def test_long_list_of_one_cta():
    for rescaled in ({1, 2, 3, 4, 5}, set(), {3}, {4, 5}):
        assert Walk(6, rescaled).all_orders() == set(), rescaled


def test_warps_of_a_set_need_not_keep_step():
    for rescaled in (set(), {2}):
        assert Walk(3, rescaled, groups=2).all_orders() == set(), rescaled


def test_random_orders_of_a_pair():
    rng = random.Random(1)
    for _ in range(400):
        n = rng.randint(1, 8)
        rescaled = {c for c in range(1, n) if rng.random() < 0.3}
        assert Walk(n, rescaled, groups=rng.randint(1, 2), ctas=2).random_order(rng) == set(), (n, rescaled)


@pytest.mark.parametrize("step,bar,kind", [
    (S, 0, ("early", S)),      # a set takes S(c-2) for S(c)
    (P, 2, ("stuck",)),        # both sets through before the issuer looks
    (FREE, 7, ("stuck",)),     # the other set's product through before this set looks
])
def test_the_walk_sees_one_barrier_where_two_are_needed(step, bar, kind):
    one = lambda st, c: (bar, c & 1) if st == step else kernel_wait(st, c)
    assert kind in Walk(4, set(), wait=one).all_orders()


def test_the_walk_sees_a_result_read_too_soon():
    end = lambda st, c: kernel_wait(O, 3) if st == END else kernel_wait(st, c)
    assert any(f[0] == "early" for f in Walk(4, set(), wait=end).all_orders())
