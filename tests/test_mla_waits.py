"""The waits between the softmax warps, the MMA issuer and the tensor core of the sparse MLA kernel, in every order in which the
roles can run: a wait names the parity of a barrier's phase, and must neither pass before what it waits for nor miss it."""
import itertools

import pytest

from umdk_b200 import _native

S, P, O, END = range(4)
WARPS = 2   # softmax warps that are modelled (they meet once a chunk)


def kernel_wait(step, c):
    w = _native.cam().umdk_sparse_mla_wait(step, c)
    assert w >= 0
    return w >> 1, w & 1


def faults(n, rescaled, wait=kernel_wait, last=END):
    """What can go wrong with n chunks of which those in ``rescaled`` rescale O: ("early", step) where a wait for the step can pass
    too soon, ("stuck",) where the roles can end up waiting for each other. All interleavings, barriers as the hardware has them:
    a phase ends with its last arrival, and a wait passes where the current phase has the other parity. ``last``: what the softmax
    warps wait for before they read O."""
    # the roles' programs: waits, arrivals, MMAs and commits into the tensor core's queue, the softmax warps' meeting
    def qk(c):
        return ([("wait", O, c - 2)] if c >= 2 else []) + [("mma", S, c)]
    issuer = qk(0)
    for c in range(n):
        issuer += (qk(c + 1) if c + 1 < n else []) + [("wait", P, c), ("mma", O if c + 1 < n else last, c)]
    softmax = []
    for c in range(n):
        softmax += [("wait", S, c), ("meet", c)] + ([("wait", O, c - 1)] if c in rescaled else []) + [("arrive", P, c)]
    softmax += [("wait", last, n - 1)]
    progs = [issuer] + [softmax] * WARPS

    found, seen = set(), set()
    start = ((0,) * len(progs), 0, 0, (0,) * 8, (0,) * 8)   # program counters, MMAs queued and done, phases, arrivals in them
    todo = [start]
    mmas = [op for op in issuer if op[0] == "mma"]

    def arrive(phase, count, step, c):
        bar = wait(step, c)[0]
        phase, count = list(phase), list(count)
        count[bar] += 1
        if count[bar] == (WARPS if step == P else 1):
            phase[bar], count[bar] = phase[bar] + 1, 0
        return tuple(phase), tuple(count)

    def happened(step, c, pcs, done):
        if step == P:
            return all(pc > softmax.index(("arrive", P, c)) for pc in pcs[1:])
        return ("mma", step, c) in mmas[:done]

    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        pcs, queued, done, phase, count = state
        nexts, passed = [], False
        if done < queued:   # the tensor core finishes the oldest MMA, its commit arrives
            nexts.append((pcs, queued, done + 1, *arrive(phase, count, *mmas[done][1:])))
        for r, prog in enumerate(progs):
            if pcs[r] == len(prog):
                continue
            op = prog[pcs[r]]
            step_on = tuple(pc + (i == r) for i, pc in enumerate(pcs))
            if op[0] == "mma":
                nexts.append((step_on, queued + 1, done, phase, count))
            elif op[0] == "arrive":
                nexts.append((step_on, queued, done, *arrive(phase, count, *op[1:])))
            elif op[0] == "meet":
                if all(pc >= prog.index(op) for pc in pcs[1:]):
                    nexts.append((step_on, queued, done, phase, count))
            else:
                bar, parity = wait(*op[1:])
                if phase[bar] & 1 != parity:
                    if not happened(*op[1:], pcs, done):
                        found.add(("early", op[1]))
                        passed = True
                        continue
                    nexts.append((step_on, queued, done, phase, count))
        if not nexts and not passed and any(pc < len(p) for pc, p in zip(pcs, progs)):
            found.add(("stuck",))
        todo += nexts
    return found


def patterns(n):
    return [set(p) for k in range(n) for p in itertools.combinations(range(1, n), k)]


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_the_result_is_read_behind_the_last_product(n):
    for rescaled in patterns(n):
        assert not any(f[0] == "early" for f in faults(n, rescaled)), rescaled


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_no_phase_is_missed(n):
    for rescaled in patterns(n):
        assert faults(n, rescaled) == set(), rescaled


@pytest.mark.parametrize("n", [2, 3, 4])
def test_the_walk_sees_a_missed_phase(n):
    """One barrier for every P: chunks that rescale nothing let the softmax warps get two phases ahead of the issuer."""
    one = lambda step, c: (2, c & 1) if step == P else kernel_wait(step, c)
    assert ("stuck",) in faults(n, set(), one)
    assert ("stuck",) not in faults(n, set(range(1, n)), one)


@pytest.mark.parametrize("n", [2, 3, 4])
def test_the_walk_sees_a_result_read_too_soon(n):
    """Behind chunks that rescale nothing the barrier of the single products may be two phases back: the same parity."""
    assert ("early", O) in faults(n, set(), last=O)
    assert ("early", O) not in faults(n, set(range(1, n)), last=O)
