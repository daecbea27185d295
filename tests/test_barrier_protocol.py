"""The mbarrier protocols of the tensor-core kernels, walked through every order in which their roles can run.

A role is a list of steps; ("wait", barrier, n) is the wait for phase n by its parity, which is all an mbarrier
offers: it passes when the phase the barrier is in has the other parity.  So a role that is two phases late waits
for good, and one that is two phases early passes at once.  The walk finds both.
"""
from __future__ import annotations

import pytest


def walk(roles, counts):
    """Explores all interleavings.  `roles`: {name: steps}; steps are ("wait", bar, n), ("arrive", bar), and the
    asynchronous ("commit", bar) (in order per role: products) and ("load", bar) (in any order).  `counts`: arrivals
    per phase (1 unless given).  Returns None, or what went wrong."""
    names = list(roles)
    bars = sorted({s[1] for steps in roles.values() for s in steps}, key=str)
    at = {b: i for i, b in enumerate(bars)}
    need = [counts.get(b, counts.get(b[0], 1) if isinstance(b, tuple) else 1) for b in bars]
    start = (tuple(0 for _ in names), tuple(() for _ in names), (), tuple((0, 0) for _ in bars))
    seen, todo = {start}, [start]

    def arrived(phases, b):
        phase, got = phases[at[b]]
        got += 1
        new = (phase + 1, 0) if got == need[at[b]] else (phase, got)
        return phases[:at[b]] + (new,) + phases[at[b] + 1:]

    while todo:
        pcs, queues, loads, phases = todo.pop()
        after = []
        for r, name in enumerate(names):
            if queues[r]:
                after.append((pcs, queues[:r] + (queues[r][1:],) + queues[r + 1:], loads, arrived(phases, queues[r][0])))
            if pcs[r] == len(roles[name]):
                continue
            step = roles[name][pcs[r]]
            moved = pcs[:r] + (pcs[r] + 1,) + pcs[r + 1:]
            if step[0] == "wait":
                phase = phases[at[step[1]]][0]
                if phase % 2 != step[2] % 2:
                    if phase != step[2] + 1:
                        return f"{name} passes {step} in phase {phase}"
                    after.append((moved, queues, loads, phases))
            elif step[0] == "arrive":
                after.append((moved, queues, loads, arrived(phases, step[1])))
            elif step[0] == "commit":
                after.append((moved, queues[:r] + (queues[r] + (step[1],),) + queues[r + 1:], loads, phases))
            else:
                after.append((moved, queues, tuple(sorted(loads + (step[1],), key=str)), phases))
        for b in set(loads):
            i = loads.index(b)
            after.append((pcs, queues, loads[:i] + loads[i + 1:], arrived(phases, b)))
        if not after and any(pc < len(roles[n]) for pc, n in zip(pcs, names)):
            return "stuck: " + ", ".join(f"{n} at {roles[n][pc]}" for pc, n in zip(pcs, names) if pc < len(roles[n]))
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def ring(prefix, t, slots):
    return (prefix, t % slots), t // slots


def producer(n, slots):
    steps = [("load", "stat")]
    for t in range(n):
        free, k = ring("free", t, slots)
        steps += ([("wait", free, k - 1)] if k else []) + [("load", ring("full", t, slots)[0])]
    return steps


def halves(n, slots, go, early, vectors):
    """Passes 3 and 4, one TMEM stage in two halves; `go` barriers on which chain 1 lets chain 2 follow."""
    full, free = (lambda t: ring("full", t, slots)), (lambda t: ring("free", t, slots)[0])
    c1, c2, ew = [("wait", "stat", 0)], [("wait", "stat", 0)], []

    def scores(c, t):
        c.append(("wait", *full(t)))
        if c is c1 and early:
            c.append(("commit", "s_ready"))
        c.append(("commit", "a" if c is c1 else "b"))

    scores(c1, 0)
    scores(c2, 0)
    for t in range(n):
        c1 += [("wait", "pa", t), ("commit", free(t))]
        c2 += [("wait", "pb", t), ("commit", free(t)), ("wait", *ring("go", t, go))]
        if t + 1 < n:
            scores(c1, t + 1)
            scores(c2, t + 1)
        c1.append(("arrive", ring("go", t, go)[0]))
        ew += [("wait", *full(t))] if vectors else []
        ew += [("wait", "s_ready", t)] if early else []
        ew += [("wait", "a", t), ("arrive", "pa"), ("wait", "b", t), ("arrive", "pb")]
    c1.append(("commit", "out"))
    c2.append(("commit", "out"))
    ew.append(("wait", "out", 0))
    return {"tma": producer(n, slots), "chain 1": c1, "chain 2": c2, "elementwise": ew}, {"free": 2, "out": 2}


def deep(n, slots, vectors):
    """Passes 3 and 4, head dims up to 64: group A two tiles ahead in two stages."""
    full, free = (lambda t: ring("full", t, slots)), (lambda t: ring("free", t, slots)[0])
    c1, c2, ew = [("wait", "stat", 0)], [("wait", "stat", 0)], []
    for t in range(min(2, n)):
        c1 += [("wait", *full(t)), ("commit", ("a", t))]
    for t in range(n):
        c1 += [("wait", ("p", t % 2), t // 2), ("wait", ("q", t % 2), t // 2), ("commit", free(t))]
        if t + 2 < n:
            c1 += [("wait", *full(t + 2)), ("commit", ("a", t % 2))]
        c2 += ([("wait", "b_free", t - 1)] if t else []) + [("wait", *full(t)), ("commit", "b"), ("commit", free(t))]
        ew += [("wait", *full(t))] if vectors else []
        ew += [("wait", ("a", t % 2), t // 2), ("arrive", ("p", t % 2)), ("wait", "b", t), ("arrive", "b_free"), ("arrive", ("q", t % 2))]
    c1.append(("commit", "out"))
    c2.append(("commit", "out"))
    ew.append(("wait", "out", 0))
    return {"tma": producer(n, slots), "chain 1": c1, "chain 2": c2, "elementwise": ew}, {"free": 2, "out": 2}


def sweep(n, slots):
    c, ew = [("wait", "stat", 0)], []
    for t in range(n):
        s, k = ring("s_free", t, 2)
        c += ([("wait", s, k - 1)] if k else []) + [("wait", *ring("full", t, slots)), ("commit", ring("s", t, 2)[0]), ("commit", ring("free", t, slots)[0])]
        ew += [("wait", *ring("s", t, 2)), ("arrive", s)]
    return {"tma": producer(n, slots), "chain 1": c, "chain 2": list(c), "elementwise": ew}, {"free": 2, "s": 2}


def first_backward(n, n0, n1, nd, keyside, p_over_s):
    """One issuing thread; dP nd tiles ahead, S one (or nd, if P goes over S)."""
    ns = nd if p_over_s else 1
    full0, full1 = (lambda t: ring("full0", t, n0)), (lambda t: ring("full1", t, n1))
    tma, mma, ew = [("load", "stat")], [("wait", "stat", 0)], []
    for t in range(n):
        for p, slots in (("1", n1), ("0", n0)):
            f, k = ring("free" + p, t, slots)
            tma += ([("wait", f, k - 1)] if k else []) + [("load", ring("full" + p, t, slots)[0])]

    def dp(t):
        mma.extend([("wait", *full1(t)), ("commit", ("dp", t % nd))] + ([] if keyside else [("commit", ring("free1", t, n1)[0])]))

    def s(t):
        mma.extend([("wait", *full0(t)), ("commit", ("s", t % ns))])

    for t in range(min(nd, n)):
        dp(t)
        if t < ns:
            s(t)
    for t in range(n):
        if not p_over_s and t + 1 < n:
            mma.append(("wait", "s_free", t))
            s(t + 1)
        mma += [("wait", ("p", t % nd), t // nd), ("commit", ring("free0", t, n0)[0])] + ([("commit", ring("free1", t, n1)[0])] if keyside else [])
        if t + nd < n:
            dp(t + nd)
            if p_over_s:
                s(t + nd)
        ew += [("wait", *full0(t))] if keyside else []
        ew += [("wait", ("s", t % ns), t // ns)] + ([] if p_over_s else [("arrive", "s_free")]) + [("wait", ("dp", t % nd), t // nd), ("arrive", ("p", t % nd))]
    mma.append(("commit", "out"))
    ew.append(("wait", "out", 0))
    return {"tma": tma, "mma": mma, "elementwise": ew}, {}


def forward(n, slots, stages, out):
    """One issuing thread, two query tiles with a softmax role each; P handed over in halves when there is one stage."""
    k_at = (lambda j: j) if not out else (lambda j: 2 * j) if stages == 1 else (lambda j: 0 if j == 0 else 2 * j - 1)
    v_at = lambda j: 2 * j + 1 if stages == 1 or j == n - 1 else 2 * j + 2
    tma, mma = [("load", ("q", 0)), ("load", ("q", 1))], []
    for i in range(n * (2 if out else 1)):
        f, k = ring("free", i, slots)
        tma += ([("wait", f, k - 1)] if k else []) + [("load", ring("full", i, slots)[0])]
    soft = {0: [], 1: []}

    def scores(x, t):
        mma.extend([("wait", ("q", x), 0)] if t == 0 else [])
        if not out and t >= stages:
            mma.append(("wait", ("s_free", x, t % stages), t // stages - 1))
        mma.extend([("wait", *ring("full", k_at(t), slots)), ("commit", ("s", x, t % stages))])
        if x == 1:
            mma.append(("commit", ring("free", k_at(t), slots)[0]))

    def output(x, t):
        if stages == 1:
            mma.append(("wait", ("half", x), t))
        else:
            mma.append(("wait", ("p", x, t % stages), t // stages))
        mma.append(("wait", *ring("full", v_at(t), slots)))
        if stages == 1:
            mma.append(("wait", ("p", x, 0), t))
        mma.append(("commit", ("o", x)))
        if t + 1 == n:
            mma.append(("commit", ("end", x)))
        if x == 1:
            mma.append(("commit", ring("free", v_at(t), slots)[0]))

    for t in range(min(stages, n) if out else n):
        for x in (0, 1):
            scores(x, t)
    for t in range(n if out else 0):
        for x in (0, 1):
            output(x, t)
            if t + stages < n:
                scores(x, t + stages)
    for x in (0, 1):
        for t in range(n):
            soft[x].append(("wait", ("s", x, t % stages), t // stages))
            if not out:
                soft[x].append(("arrive", ("s_free", x, t % stages)))
                continue
            if t:   # the rescaling, when the maximum grew (here: always; the other case waits for less)
                soft[x].append(("wait", ("o", x), t - 1))
            soft[x] += ([("arrive", ("half", x))] if stages == 1 else []) + [("arrive", ("p", x, t % stages))]
        if out:
            soft[x].append(("wait", ("end", x), 0))
    return {"tma": tma, "mma": mma, "softmax A": soft[0], "softmax B": soft[1]}, {}


@pytest.mark.parametrize("n", (1, 2, 3, 5))
@pytest.mark.parametrize("early,vectors", [(True, False), (False, True)])   # pass 3, pass 4
def test_passes_3_and_4_in_halves(n, early, vectors):
    assert walk(*halves(n, 2, 2, early, vectors)) is None


def test_one_go_barrier_would_not_do():
    """Chain 1 can signal twice before chain 2 looks (what chain 2 waits for next does not hold it back)."""
    assert "chain 2 at ('wait', ('go', 0)" in walk(*halves(2, 2, 1, False, True))


@pytest.mark.parametrize("n", (1, 2, 3, 5))
@pytest.mark.parametrize("vectors", (False, True))
def test_passes_3_and_4_deep(n, vectors):
    assert walk(*deep(n, 3, vectors)) is None


@pytest.mark.parametrize("n", (1, 2, 3, 5))
def test_sweep(n):
    assert walk(*sweep(n, 2)) is None


@pytest.mark.parametrize("n", (1, 3, 5))
@pytest.mark.parametrize("n0,n1,nd,keyside,p_over_s", [(2, 2, 2, False, False), (2, 3, 3, True, False), (2, 2, 2, True, True), (3, 3, 3, True, True)])
def test_first_backward(n, n0, n1, nd, keyside, p_over_s):
    assert walk(*first_backward(n, n0, n1, nd, keyside, p_over_s)) is None


@pytest.mark.parametrize("n", (1, 3, 4))
@pytest.mark.parametrize("stages,out", [(1, True), (2, True), (2, False)])
def test_forward(n, stages, out):
    assert walk(*forward(n, 4, stages, out)) is None
