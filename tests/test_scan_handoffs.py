"""The hand-offs between the warps of the tensor-core scan (``csrc/scan_tc.cu``), as a model that is searched exhaustively.

An mbarrier wait names a phase by its parity only: a warp that is held up until the barrier has completed TWO phases more than
it has seen waits for a phase that will not come. So no barrier may be able to run ahead of any of its waiters, however the
warps are scheduled. The model has one role per kind of warp, written in the order of the kernel's loop body, with asynchronous
copies and products completing at any time; every reachable state is visited, and every role has to reach its end."""

from __future__ import annotations

import pytest

NC = 5          # chunks: both slots of every double buffer are refilled at least once


class Op:
    WAIT, ARRIVE, COPY, MMA = range(4)


def wait(bar, use):
    """Wait for the completion of use number `use` of the barrier: the test is on that use's parity."""
    return (Op.WAIT, bar, use & 1)


def arrive(bar):
    return (Op.ARRIVE, bar)


def copy(bar):
    """A bulk copy whose bytes complete a phase of `bar`, at any later time."""
    return (Op.COPY, bar)


def mma(bar):
    """Products followed by a commit: complete a phase of `bar` later, in issue order."""
    return (Op.MMA, bar)


def scan_program(form="whole", producer_waits_for_un=False, kgt_before_un=True):
    """``form``: whole (outputs and states), transition (no U^T, no outputs), output (no state update)."""
    ut, state, out = form != "transition", form != "output", form != "transition"

    def load(n):
        b = n & 1
        return [copy(f"wq{b}")] + ([copy(f"ut{b}")] if ut else []) + ([copy(f"kgt{b}")] if state else [])

    producer = load(0) + [copy("aqk")] + load(1)
    issuer, output = [], [arrive("of")] if out else []
    compute = {0: [arrive("sb0")], 1: [arrive("sb1")]}
    for n in range(NC):
        b, use = n & 1, n >> 1
        more, refill = n + 1 < NC, n + 2 < NC
        producer += [wait("un", n)] if producer_waits_for_un else []
        producer += [wait("m2", n)] + ([copy("aqk")] if more else []) + (load(n + 2) if refill else [])
        issuer += [wait(f"wq{b}", use), wait("sb0", n), wait("sb1", n)] + ([mma("m1")] if state else [])
        issuer += [wait("of", n)] if out else []
        issuer += [wait(f"kgt{b}", use)] if state else [mma("m1")]
        issuer += [wait("un", n)] + ([mma("m30"), mma("m31")] if state else []) + [wait("aqk", n), mma("m2")]
        if out:
            output += [wait("m2", n)] + ([arrive("of")] if more else [])
        for part, role in compute.items():
            role += ([wait(f"ut{b}", use)] if ut else []) + [wait("m1", n)]
            role += [wait(f"kgt{b}", use)] if state and kgt_before_un else []
            role += [arrive("un")]
            role += [wait(f"kgt{b}", use)] if state and not kgt_before_un else []
            role += ([wait(f"m3{part}", n)] if state else []) + ([arrive(f"sb{part}")] if more else [])
    counts = {"un": 2}                                      # both halves of the compute warps arrive; one arrival elsewhere
    return [producer, issuer, compute[0], compute[1]] + ([output] if out else []), counts


def stuck_states(program, counts):
    """States of the whole block in which nothing can happen although a role has not ended."""
    names = sorted({op[1] for role in program for op in role})
    index = {n: i for i, n in enumerate(names)}
    need = [counts.get(n, 1) for n in names]
    # (position of every role, (completed phases' parity, pending arrivals) per barrier, copies in flight, products in flight)
    start = (tuple(0 for _ in program), tuple((0, need[i]) for i in range(len(names))), (), ())
    seen, todo, stuck = {start}, [start], []

    def complete(bars, bar):
        parity, pending = bars[bar]
        pending -= 1
        entry = (parity ^ 1, need[bar]) if pending == 0 else (parity, pending)
        return bars[:bar] + (entry,) + bars[bar + 1:]

    while todo:
        pos, bars, copies, products = todo.pop()
        after = []
        for r, role in enumerate(program):
            if pos[r] == len(role):
                continue
            op = role[pos[r]]
            nxt = pos[:r] + (pos[r] + 1,) + pos[r + 1:]
            bar = index[op[1]]
            if op[0] == Op.WAIT:
                if bars[bar][0] != op[2]:                   # the current phase is not the one waited for: it has completed
                    after.append((nxt, bars, copies, products))
            elif op[0] == Op.ARRIVE:
                after.append((nxt, complete(bars, bar), copies, products))
            elif op[0] == Op.COPY:
                after.append((nxt, bars, tuple(sorted(copies + (bar,))), products))
            else:
                after.append((nxt, bars, copies, products + (bar,)))
        for bar in set(copies):
            left = list(copies)
            left.remove(bar)
            after.append((pos, complete(bars, bar), tuple(left), products))
        if products:
            after.append((pos, complete(bars, products[0]), copies, products[1:]))
        if not after and any(p < len(role) for p, role in zip(pos, program)):
            stuck.append(pos)
        for state in after:
            if state not in seen:
                seen.add(state)
                todo.append(state)
    return stuck


@pytest.mark.parametrize("form", ["whole", "transition", "output"])
def test_no_schedule_of_the_scan_gets_stuck(form):
    assert not stuck_states(*scan_program(form))


@pytest.mark.parametrize("wrong", [{"producer_waits_for_un": True}, {"kgt_before_un": False}])
def test_the_search_finds_a_barrier_that_can_run_ahead(wrong):
    """The producer waiting for the Un hand-off, or the state pass waiting for KG^T after it: both barriers can run ahead."""
    assert stuck_states(*scan_program(**wrong))
