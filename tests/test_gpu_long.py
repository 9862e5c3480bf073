"""Long machines: the persistent kernel hands them to a kernel that runs one
machine per warp a tape word at a time.  Whole searches through it equal the
CPU oracle in every count and survivor line, at the settings where it can go
wrong: machines handed over almost at once, its time bound running out, its
queue and the frontier nearly full, and never handing over."""
import pytest

import e13b200 as E
import oracle_lib as O
from gpu_common import ctx, make_job

pytestmark = pytest.mark.gpu

# block 64 and warp stack 1: an epoch's outputs may need 2 * 296 * 33 + 65536 nodes of the frontier
TIGHT = dict(block=64, warp_stack=1, stack_nodes=2 * 296 * 33 + 65536)


@pytest.mark.parametrize("name,X,tune", [
    ("counters_f2_base_11", -1, dict(run_skip=1)),                 # in-place loops to the deadline
    ("counters_f2_base_17", -1, dict(run_skip=1, epoch_us=50)),    # the 1 ms bound: machines come back and go on
    ("counters_f2_base_27", -1, dict(run_skip=8192)),
    ("local_edits_f2", 8, dict(run_skip=1)),                       # forks of old machines, a survivor's read mask
    ("local_edits_f2", 8, dict(run_skip=1, **dict(TIGHT, stack_nodes=TIGHT["stack_nodes"] + 700))),
    ("local_edits_f2", 11, dict(run_skip=1, slice=1, **dict(TIGHT, stack_nodes=TIGHT["stack_nodes"] + 33))),
    ("local_edits_f2", 12, dict(run_skip=0)),
    ("doubling_X0", 0, dict(run_skip=1)),                          # free cells only, no budget
])
def test_long_machines_equal_oracle(searches, name, X, tune):
    e = searches[name]
    job = make_job(e, X)
    base = O.load_machine(e["machine"])
    free = e["free"] if e["mode"] != "delete" else None
    _, jo = O.setup(base, X, fmax=e["fmax"] or 0, free_cells=free)
    exp, recs = O.search(jo)
    c, surv = ctx().search(job, E.tuning(**tune))
    assert c.as_dict() == exp
    assert sorted(E.survivor_line(job, s) for s in surv) == sorted(O.survivor_line(X, r, jo.nq) for r in recs)


@pytest.mark.parametrize("block,slice_", [(768, 1), (768, 2), (768, 8), (64, 17), (32 * 21, 4096)])
@pytest.mark.parametrize("name,X", [("local_edits_f2", 11), ("counters_f2_base_11", -1)])
def test_slices_equal_oracle(searches, name, X, block, slice_):
    """Slices of one iteration of several steps, of the shortest one that
    starving warps shorten, and ones that end because lanes have stopped: every
    deadline and event falls on some step of an iteration."""
    e = searches[name]
    job = make_job(e, X)
    _, jo = O.setup(O.load_machine(e["machine"]), X, fmax=e["fmax"], free_cells=None)
    exp, recs = O.search(jo)
    c, surv = ctx().search(job, E.tuning(block=block, slice=slice_))
    assert c.as_dict() == exp
    assert sorted(E.survivor_line(job, s) for s in surv) == sorted(O.survivor_line(X, r, jo.nq) for r in recs)
