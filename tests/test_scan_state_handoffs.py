"""Chunk states leave the scan through tensor memory: the compute warps put the state there after its bf16 copy has been handed
on, the output warps store it and give the place back. The same exhaustive search as in test_scan_handoffs, with these two
barriers in the program."""

from __future__ import annotations

from tests.test_scan_handoffs import NC, arrive, scan_program, stuck_states, wait


def _with_states(give_back=True):
    program, counts = scan_program("whole")
    producer, issuer, half0, half1, output = program

    def compute(role, part):
        new, n = [], -1                                     # the state of chunk n goes out after the hand-off sb of chunk n + 1
        for op in role:
            new.append(op)
            if op == arrive(f"sb{part}"):
                n += 1
                if n > 0:
                    new += ([wait("he", n - 2)] if n > 1 and give_back else []) + [arrive("hf")]
        return new

    out, n = [], -1
    for op in output:                                       # [arrive of] then per chunk: wait m2, arrive of (but for the last)
        out.append(op)
        if op == arrive("of"):
            n += 1
            if n > 0:
                out += [wait("hf", n - 1), arrive("he")]
    return [producer, issuer, compute(half0, 0), compute(half1, 1), out], {**counts, "hf": 2}


def test_no_schedule_gets_stuck():
    program, counts = _with_states()
    assert sum(op == arrive("hf") for op in program[2]) == sum(op == wait("hf", 0) or op == wait("hf", 1) for op in program[4]) == NC - 1
    assert not stuck_states(program, counts)


def test_the_place_has_to_be_given_back():
    """Without the wait for it the compute warps run ahead of the output warps by two states."""
    assert stuck_states(*_with_states(give_back=False))

