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
