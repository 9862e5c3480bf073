"""Whole tables and raw machines that outlive the first kernel's step limit
(1024 steps) run in a warp of their own: their results against the oracle on
limits around that step count, on tables that loop, sweep, halt and leave the
window late."""
import random

import pytest

import e13b200 as E
import oracle_lib as O
from gpu_common import ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,n,max_steps", [(2, 500, 1023), (2, 500, 1024), (3, 700, 1025), (4, 769, 5000),
                                            (13, 1500, 20000), (16, 33, 1 << 18), (1, 40, 4097)])
def test_raw_machines_equal_oracle(nq, n, max_steps):
    rng = random.Random(1000 * nq + n)
    # few halts, and mostly moves back and forth: more machines live long
    codes = bytes(rng.choice([rng.randrange(4 * nq)] * 30 + [255]) for _ in range(2 * nq * n))
    rows, total = ctx().raw_run(n, nq=nq, max_steps=max_steps, codes=codes)
    exp = O.raw_run(codes, n, nq, max_steps)
    assert rows == exp
    assert total == sum(r[0] for r in exp)


def test_long_tables_equal_oracle():
    base = O.load_machine("erdos_14.txt")
    rng = random.Random(5)
    tabs = [base]
    for _ in range(400):
        t = list(base)
        for _ in range(rng.randint(1, 2)):
            t[rng.randrange(28)] = rng.randrange(-1, 56)
        tabs.append(t)
    for nq, rows in ((2, 150), (3, 150)):
        tabs += [[rng.randrange(4 * nq) for _ in range(2 * nq)] + [-1] * (28 - 2 * nq) for _ in range(rows)]
    out = ctx().run_full(tabs, 14)
    assert out == [O.run_full(t, 14) for t in tabs]
