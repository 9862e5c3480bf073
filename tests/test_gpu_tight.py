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
