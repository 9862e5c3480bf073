"""check.py's stage walks that leave the device's tape (cells -2^22 .. 2^22 - 1):
the verdict says "off tape" at the step that leaves it, and no other walk of the
batch notices.  The allowed cells fill a walk's tape exactly, so a head one cell
outside has no word there: the word before a walk's first is the last word of
the walk before it (of the first walk: outside the buffer)."""
import pytest

import oracle_lib as O
from gpu_common import ctx

pytestmark = pytest.mark.gpu

SIDE = 1 << 22


def line_of(codes):
    rows = ["---" if c < 0 else f"{c & 1}{'R' if c & 2 else 'L'}{c >> 2}" for c in codes]
    return "SURVIVOR table=" + "|".join(f"{rows[i]} {rows[i + 1]}" for i in range(0, len(rows), 2))


def runaway(write, right):
    """erdos_14 with N1 going to a fifteenth state that runs one way for ever:
    it reaches stages 1 to 8 before it first reads N1."""
    go = 14 << 2 | (2 if right else 0)
    codes = list(O.load_machine("erdos_14.txt")) + [go, go | 1]
    codes[27] = go | write
    return codes


def steps_on_tape(codes):
    """Steps until the head leaves the tape (the tables halt nowhere before)."""
    tape, head, st, t = bytearray(2 * SIDE), SIDE, 0, 0
    while 0 <= head < 2 * SIDE:
        c = codes[2 * st + tape[head]]
        tape[head] = c & 1
        head += 1 if c & 2 else -1
        st = c >> 2
        t += 1
    return t


def test_walks_off_either_end():
    tables = [runaway(w, r) for r in (0, 1) for w in (0, 1)]
    steps = [steps_on_tape(tables[0]), steps_on_tape(tables[2])]
    assert steps == [4271567, 4271572]
    off = [[line_of(t), f"   halt@None: FAIL stage 9: off tape at step {steps[i // 2]}"] for i, t in enumerate(tables)]
    for lines in off:  # the first and the last walk of its batch
        assert ctx().check_crafted(lines[:1]) == lines
    whole = line_of(O.load_machine("erdos_14.txt"))
    # left of a walk to the right's end, right of one to the left's, both beside whole walks
    batch = [off[0], off[2], off[1], O.check_line(whole), off[1], off[3], O.check_line(whole), off[3], off[0]]
    assert ctx().check_crafted([lines[0] for lines in batch]) == [v for lines in batch for v in lines]


def test_walks_of_mutants_equal_oracle():
    """Stage walks of erdos_14 with one or two cells changed: they fail at every
    stage, by limits, halts and runs far to either side."""
    import random
    rng = random.Random(12)
    base = O.load_machine("erdos_14.txt")
    lines = []
    for _ in range(120):
        t = list(base)
        for _ in range(rng.randint(1, 2)):
            t[rng.randrange(28)] = rng.randrange(-1, 56)
        if -1 in t:
            lines.append(line_of(t))
    got = ctx().check_crafted(lines)
    want = [v for line in lines for v in O.check_line(line)]
    assert len(got) == len(want)
    assert [g for g in got if ": off tape at" not in g] == [w for g, w in zip(got, want) if ": off tape at" not in g]
