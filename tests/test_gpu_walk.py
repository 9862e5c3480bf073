"""The checkers' word-at-a-time simulator (one warp per machine) against the
oracle's single-stepped restatement of recheck.c and deep.c, on random small
machines: loops inside a word and across words, zigzags, sweeps out of the
shared-memory window and off the tape, halts and cells never read, with the
counter's and the block's words partly filled."""
import random

import pytest

import e13b200 as E
import oracle_lib as O
from gpu_common import ctx

pytestmark = pytest.mark.gpu


def random_lines(n, nq, seed):
    rng = random.Random(seed)

    def cell():
        r = rng.random()
        return "---" if r < 0.04 else "?---" if r < 0.08 else f"{rng.randint(0, 1)}{rng.choice('LR')}{rng.randrange(nq)}"

    out = []
    for _ in range(n):
        table = "|".join(f"{cell()} {cell()}" for _ in range(nq))
        rel = rng.randint(0, 1)
        out.append(f"SURVIVOR X=-1 st0={rng.randrange(nq)} head0={rng.randint(-4, 3)} abs={1 - rel} rel={rel} "
                   f"steps=0 table={table}")
    return out


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nq,nmax", [(1, 1), (2, 3), (3, 9), (5, 10), (16, 4)])
def test_random_machines_equal_oracle(nq, nmax, mode):
    lines = random_lines(96, nq, 100 * nq + nmax)
    ins = [E.parse_survivor_line(l) for l in lines]
    outs = ctx().check(ins, nmax, mode)
    for line, ci, o in zip(lines, ins, outs):
        if mode == 0:
            ok, verdict, counters = O.recheck_line(line, nmax)
            got = E.format_recheck(o, nmax)
            if nmax < 9:  # recheck.c prints a counter it has not filled there, the library the empty set
                got, verdict = (v.split(" (c2 counter")[0] for v in (got, verdict))
            assert got == verdict, line
            for n in range(1, o.stages_done + 1):
                got = "".join(f"{o.ones_cells[n][j]}," for j in range(min(o.nones[n], 64)))
                assert got == counters[n - 1], (line, n)
        else:
            assert E.format_deep(ci, o, nmax) == O.deep_line(line, nmax), line


@pytest.mark.parametrize("nq,nmax", [(3, 1), (4, 2), (5, 3)])
def test_words_beyond_the_window_equal_oracle(nq, nmax):
    """Stage 1 may take 100,000 steps: many of these machines sweep, zigzag or
    shift past the window's ends (cells -4096 and 2^nmax + 4096)."""
    lines = random_lines(600, nq, 7 * nq)
    outs = ctx().check([E.parse_survivor_line(l) for l in lines], nmax, 0)
    assert sum(abs(o.fail_head) > 4096 + (1 << nmax) for o in outs) >= 30
    for line, o in zip(lines, outs):
        got, verdict = (v.split(" (c2 counter")[0] for v in (E.format_recheck(o, nmax), O.recheck_line(line, nmax)[1]))
        assert got == verdict, line


def test_runaway_survivor_equals_oracle():
    """A survivor that leaves the block at stage 12 and zigzags 16,000 cells
    beyond the window until its limit, 1.3e8 steps."""
    line = ("SURVIVOR X=9 st0=2 head0=-2 abs=1 rel=0 steps=271500 table=1L1 1R0|1L2 1L1|1R3 0R0|0L6 0R4|0L3 1R5|0R1 1R4|"
            "1R3 1L7|1L6 0L8|1L3 0L7|?0L10 ?1R9|?1R12 ?0L2|?0L12 ?---|?0R9 ?0L11")
    (o,) = ctx().check([E.parse_survivor_line(line)], 12, 0)
    ok, verdict, counters = O.recheck_line(line, 12)
    assert E.format_recheck(o, 12) == verdict
    for n in range(1, o.stages_done + 1):
        assert "".join(f"{o.ones_cells[n][j]}," for j in range(min(o.nones[n], 64))) == counters[n - 1]
