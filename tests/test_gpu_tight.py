"""Searches with little room: warp stacks of a node or two, and frontiers with
hardly more than an epoch's outputs.  They go through the outputs buffer for
most of their nodes, and still give the whole search."""
import pytest

import e13b200 as E
from gpu_common import check_entry, ctx, golden_lines, make_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,warp_stack", [(64, 1), (64, 2), (96, 1), (96, 2), (256, 1), (768, 1)])
@pytest.mark.parametrize("X", [1, 8, 11])
def test_small_warp_stacks(searches, X, block, warp_stack):
    """An epoch that ends because its outputs pass their soft limit has room for
    all that is then still written: what each warp's stack has no room for, the
    lanes and stacks, and the claimed input."""
    e = searches["local_edits_f3"]
    with E.Context(0) as c:  # with buffers of this size, not of an earlier search
        job = make_job(e, X)
        for slice_ in (24, 200):
            counts, surv = c.search(job, E.tuning(block=block, warp_stack=warp_stack, slice=slice_))
            check_entry(dict(e, expect=[x for x in e["expect"] if x["X"] == X]), [counts.as_dict()])
            assert sorted(E.survivor_line(job, s) for s in surv) == [l for l in golden_lines(e) if f" X={X} " in l]


@pytest.mark.parametrize("block,warp_stack", [(64, 1), (768, 256)])
def test_long_machines_leave_a_tight_frontier(searches, block, warp_stack):
    """A frontier with room for an epoch's outputs and 40 nodes more still hands
    its long machines over: the search of X = 8, whose longest machine takes
    208,000 steps, needs about the rounds that it needs with the default one."""
    e = searches["local_edits_f2"]
    job = make_job(e, 8)
    out_nodes = 2 * (148 * block // 32) * (32 + warp_stack) + 65536
    rounds = {}
    with E.Context(0) as c:
        for stack_nodes in (out_nodes + 40, 0):
            counts, _ = c.search(job, E.tuning(block=block, warp_stack=warp_stack, stack_nodes=stack_nodes))
            check_entry(dict(e, expect=[x for x in e["expect"] if x["X"] == 8]), [counts.as_dict()])
            rounds[stack_nodes] = c.stats().warp_rounds
    assert rounds[out_nodes + 40] < 2 * rounds[0], rounds
